"""REF-mask reconstruction on a pass large enough for its four-CTA instance (64 items of 256 rows a
CTA), against the same rows on the first 20,000 pixels alone (three CTAs): a pixel's terms are the
same but for which of them are polynomials (integer uvw), each within 0.92e-6 |y|, fractional
2.36e-6, of the exact one on either side; 0.2e-6 for the sums.  Windows mask pixels of both."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frac", [False, True])
def test_instances_agree(frac):
    import viss_recon_shade_gb300 as V
    res, K, sub = 413, 62000, 20000
    J = res * res
    rng = np.random.default_rng(3 + frac)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    u, v, w = (rng.integers(-900, 901, K).astype(np.float32) for _ in range(3))
    if frac:
        u += rng.uniform(-0.5, 0.5, K).astype(np.float32)
    y = (rng.normal(size=K) + 1j * rng.normal(size=K)).astype(np.complex64)
    shade = np.stack([rng.integers(1, 60, K), rng.integers(1, 4, K), rng.integers(1, 60, K), rng.integers(1, 4, K)], 1)
    from viss_recon_shade_gb300.synth import fibonacci_sphere
    l, m, n = fibonacci_sphere(J)
    cfg = V.DftConfig.reference(res, precision=V.PREC_FAST).with_(norm=1.0)
    run = lambda c, k: V.recon(c, *map(cu, (u, v, w, y, l[:k], m[:k], n[:k])), shade=cu(shade.astype(np.int32)))  # noqa: E731
    big, small = run(cfg, J)[:sub].cpu().numpy(), run(cfg, sub).cpu().numpy()
    off = run(cfg.with_(recon_mask=V.RECON_MASK_NONE), sub).cpu().numpy()
    tol = 2 * (0.1e-6 + (2.36e-6 if frac else 0.92e-6)) * np.abs(y).sum()
    assert np.abs(big - small).max() <= tol
    assert np.abs(off - small).max() > 100 * tol  # the windows mask
