"""Single terms of the unmasked reconstruction where its packed and polynomial forms meet:
integer uvw (every other row's second pixel pair without the SFU, in groups of four rows and a
remainder) and fractional ones, phases on the quadrant and half-turn boundaries and just off
them, FAST and compensated, at row counts around the groups and the tile.

A pixel's error is bounded by that of its terms: the angle's 23 bits and roundings (3.7e-7 rad)
and the SFU's (4.2e-7), 8e-7 of |y| each; 1e-6 K max|y| leaves the sums' rounding room."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 3, 4, 5, 8, 511, 513])
@pytest.mark.parametrize("frac", [False, True])
@pytest.mark.parametrize("prec", ["fast", "comp"])
def test_terms(oracle, K, frac, prec):
    import viss_recon_shade_gb300 as V
    rng = np.random.default_rng(K + 10 * frac)
    J = 1500
    l = (rng.integers(-8, 9, J) / 8.0).astype(np.float32)  # with scale 1: multiples of 1/8 turn per unit of u
    m = np.where(rng.random(J) < 0.5, 0.0, rng.choice([2.0**-24, -(2.0**-24), 2.0**-12], J)).astype(np.float32)
    n = rng.uniform(-1, 1, J).astype(np.float32)
    u, v, w = (rng.integers(-40, 41, K).astype(np.float32) for _ in range(3))
    w[: K // 2 + 1] = 0.0
    if frac:
        u += rng.choice([0.0, 0.25, 0.5, -0.125], K).astype(np.float32)
    y = (rng.normal(size=K) + 1j * rng.normal(size=K)).astype(np.complex64)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    cfg = V.DftConfig(mask=V.MASK_NONE, recon_mask=V.RECON_MASK_NONE, phase_scale=1.0, n_offset=-1.0, norm=1.0,
                      precision=V.PREC_FAST if prec == "fast" else V.PREC_COMPENSATED)
    F = V.recon(cfg, *map(cu, (u, v, w, y, l, m, n))).cpu().numpy()
    Fo = oracle.recon(oracle.make_cfg(phase_scale=1.0, n_offset=-1.0, norm=1.0), u, v, w, None, y, l, m, n)
    assert np.abs(F - Fo).max() <= 1e-6 * K * np.abs(y).max()
