"""Single terms of the unmasked visibilities, where the packed and polynomial forms meet: integer
uvw (every other pixel's second row pair without the SFU, in groups of four pixels and a
remainder) and fractional ones, phases on the quadrant and half-turn boundaries and just off
them, FAST and compensated, at pixel counts around the groups, the chunks and the tile.

A visibility's error is bounded by that of its terms: 23 bits of a turn (3.7e-7 rad), the angle's
rounding (1.2e-7), the SFU (4.2e-7), and for each of fractional uvw and compensation three
roundings beside -3 pi (4.8e-7 each): 0.92e-6, 2.36e-6 and 3.8e-6; with 0.3e-6 for the sums."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("J", [1, 3, 4, 5, 31, 33, 511, 513, 1100])
@pytest.mark.parametrize("frac", [False, True])
@pytest.mark.parametrize("prec", ["fast", "comp"])
def test_terms(J, frac, prec):
    import viss_recon_shade_gb300 as V
    rng = np.random.default_rng(J + 10 * frac)
    K = 1500
    l = (rng.integers(-8, 9, J) / 8.0).astype(np.float32)  # with scale 1: multiples of 1/8 turn per unit of u
    m = np.where(rng.random(J) < 0.5, 0.0, rng.choice([2.0**-24, -(2.0**-24), 2.0**-12], J)).astype(np.float32)
    n = rng.uniform(-1, 1, J).astype(np.float32)
    b = rng.lognormal(0.0, 1.0, J).astype(np.float32)
    u, v, w = (rng.integers(-40, 41, K).astype(np.float32) for _ in range(3))
    w[: K // 2 + 1] = 0.0
    if frac:
        u += rng.choice([0.0, 0.25, 0.5, -0.125], K).astype(np.float32)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    cfg = V.DftConfig(mask=V.MASK_NONE, recon_mask=V.RECON_MASK_NONE, phase_scale=1.0, n_offset=-1.0,
                      precision=V.PREC_FAST if prec == "fast" else V.PREC_COMPENSATED)
    got = V.vis_dft(cfg, *map(cu, (u, v, w, l, m, n, b))).cpu().numpy()
    f8 = lambda x: x.astype(np.float64)  # noqa: E731
    t = np.outer(f8(u), f8(l)) + np.outer(f8(v), f8(m)) + np.outer(f8(w), f8(n) - 1.0)
    want = (f8(b) * np.exp(-2j * np.pi * t)).sum(1)
    tol = 0.3e-6 + 0.92e-6 + 1.44e-6 * (frac + (prec == "comp"))
    assert np.abs(got - want).max() <= tol * J * b.max()
