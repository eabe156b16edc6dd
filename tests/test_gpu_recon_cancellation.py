"""The reconstruction turns every other row by half a turn with -|y|, so that what the SFU's sine
and cosine are off by on average cancels over the rows, for every pixel: integer uvw, where some
terms are polynomials, unmasked and with REF windows, rows far beyond one tile.

With |y| = 1 and phases spread evenly a systematic error of the terms is the mean error of a pixel's
sum divided by K.  What does not cancel is random: a term's 8e-7 (angle, roundings, SFU) over sqrt(K)
rows, 3.1e-9 for a pixel at K = 65,536 and less for a mean over 500; each of the four pixels of a
thread must be that close to no systematic error."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ref", [False, True])
@pytest.mark.parametrize("K", [65536, 65531])
def test_mean_error_of_each_pixel_of_four(oracle, ref, K):
    import viss_recon_shade_gb300 as V
    from viss_recon_shade_gb300.synth import fibonacci_sphere
    rng = np.random.default_rng(7)
    res = 45
    J = res * res
    l, m, n = fibonacci_sphere(J)
    u, v, w = (np.ceil(rng.normal(0, 300, K)).astype(np.float32) for _ in range(3))
    y = np.exp(2j * np.pi * rng.random(K)).astype(np.complex64)
    # ratios that can fire on no pixel: every tile runs unmasked
    shade = np.tile(np.array([0, 1, 0, 1], np.int32), (K, 1))
    cu = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    kw = dict(recon_mask=V.RECON_MASK_REF, res=res) if ref else {}
    F = V.recon(V.DftConfig(precision=V.PREC_FAST, norm=1.0 / K, **kw), *map(cu, (u, v, w, y, l, m, n)),
                shade=cu(shade) if ref else None).cpu().numpy()
    Fo = oracle.recon(oracle.make_cfg(norm=1.0 / K), u, v, w, None, y, l, m, n)
    err = F.astype(np.complex128) - Fo
    mean = [abs(err[i::4].mean()) for i in range(4)]
    rms = [np.sqrt((np.abs(err[i::4]) ** 2).mean()) for i in range(4)]
    print("mean", mean, "rms", rms)
    assert max(mean) <= 8e-7 / np.sqrt(K), (mean, rms)
