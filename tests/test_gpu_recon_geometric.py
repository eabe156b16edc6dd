"""The geometric reconstruction where its pieces meet: skies that end inside or on a warp's patch of
128 pixels, row counts around a load of 32 rows and a sum of 256, snapshots in order, several
to a load, and interleaved so that a load returns to a snapshot.  Some patches are hidden, some
seen and some open for every snapshot.  Pixels within 1e-9 of a limb are left out.

With integer uvw a pixel's error is bounded by that of its terms: the angle's 23 bits and
roundings (3.7e-7 rad) and the SFU's (4.2e-7), 8e-7 of |y| each; 1e-6 K max|y| leaves the sums'
rounding room.  The fractional and compensated instances weigh whole numbers with the phase 0
(a fractional row weighs nothing): sums below 5e5 are exact to the nearest integer."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


CASES = [(1, "sorted"), (31, "sorted"), (33, "mixed"), (255, "mixed"), (257, "sorted"), (900, "mixed")]


def setup(oracle, J, K, order, seed):
    from viss_recon_shade_gb300.synth import fibonacci_sphere
    rng = np.random.default_rng(seed)
    nsat, S = 5, (K + 6) // 7
    d = rng.normal(size=(S, 1, 3))
    d = d / np.linalg.norm(d, axis=2, keepdims=True) + 0.03 * rng.normal(size=(S, nsat, 3))
    pos = (2037.4 * d / np.linalg.norm(d, axis=2, keepdims=True)).astype(np.float32)
    a, b = np.triu_indices(nsat, 1)
    sel = np.arange(K) % a.size
    snap, pair = (np.arange(K) // 7).astype(np.int32), (a[sel] | (b[sel] << 16)).astype(np.int32)
    if order == "mixed":
        p = rng.permutation(K)
        snap, pair = snap[p], pair[p]
    lmn = fibonacci_sphere(J)
    mask, margin = oracle.geo_mask(oracle.make_geo(pos, snap, pair), 1737.4, *lmn, K, J)
    cu = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    geo = dict(snap=cu(snap), pair=cu(pair), sat_pos=cu(pos))
    return rng, lmn, mask, ~(margin < 1e-9).any(0), cu, geo


@pytest.mark.parametrize("J", [1, 127, 128, 129, 1025, 2000])
@pytest.mark.parametrize("K,order", CASES)
def test_patches(oracle, J, K, order):
    import viss_recon_shade_gb300 as V
    rng, (l, m, n), mask, pix, cu, geo = setup(oracle, J, K, order, J + 7 * K)
    u, v, w = (rng.integers(-40, 41, K).astype(np.float32) for _ in range(3))
    y = (rng.normal(size=K) + 1j * rng.normal(size=K)).astype(np.complex64)
    f8 = lambda x: x.astype(np.float64)  # noqa: E731
    t = np.outer(f8(u), f8(l)) + np.outer(f8(v), f8(m)) + np.outer(f8(w), f8(n) - 1.0)
    Fo = (np.where(mask, 0.0, y[:, None]) * np.exp(2j * np.pi * t)).sum(0)
    cfg = V.DftConfig.geometric(precision=V.PREC_FAST).with_(norm=1.0)
    F = V.recon(cfg, *map(cu, (u, v, w, y, l, m, n)), **geo).cpu().numpy()
    assert np.abs(F - Fo)[pix].max(initial=0.0) <= 1e-6 * K * np.abs(y).max()


@pytest.mark.parametrize("J", [1, 127, 128, 129, 1025, 2000])
@pytest.mark.parametrize("K,order", CASES)
@pytest.mark.parametrize("frac,prec", [(False, "fast"), (True, "fast"), (True, "comp")])
def test_weighted_counts(oracle, J, K, order, frac, prec):
    import viss_recon_shade_gb300 as V
    rng, lmn, mask, pix, cu, geo = setup(oracle, J, K, order, J + 7 * K + 1)
    y = rng.integers(1, 101, K).astype(np.float32)
    u = np.zeros(K, np.float32)
    if frac:
        u[K // 2], y[K // 2] = 0.5, 0.0
    z = np.zeros(K, np.float32)
    cfg = V.DftConfig.geometric(precision=V.PREC_FAST if prec == "fast" else V.PREC_COMPENSATED).with_(norm=1.0)
    F = V.recon(cfg, *map(cu, (u, z, z, y.astype(np.complex64), *lmn)), **geo).cpu().numpy()
    want = np.where(mask, 0.0, y[:, None].astype(np.float64)).sum(0)
    assert np.array_equal(np.round(F.real[pix]), want[pix])
