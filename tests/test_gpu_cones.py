"""The geometric mask where the cones and caps that shortcut it are degenerate or ragged: 2 to
32 satellites (lanes per snapshot rounded up to a power of two), skies that end inside a warp's
patch or a block, satellites far apart, on opposite sides of the Moon, on its surface, inside
it and at its centre, and rows in any order.  Zero phase, so that the visibilities count the
occluded pixels and the reconstruction the rows that see a pixel: exact integers, compared
with the FP64 oracle's mask (pixels within 1e-9 rad of a limb left out)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsat,S,J,kind", [(2, 37, 1, "near"), (3, 5, 1023, "near"), (5, 61, 2049, "wide"),
                                           (8, 130, 1111, "opposite"), (9, 33, 3001, "near"), (32, 7, 1500, "wide"),
                                           (4, 40, 900, "surface"), (3, 20, 700, "inside"), (2, 1, 65, "centre")])
def test_mask_counts(oracle, nsat, S, J, kind):
    import viss_recon_shade_gb300 as V
    from viss_recon_shade_gb300.synth import fibonacci_sphere
    rng = np.random.default_rng(nsat * 1000 + S)
    axis = rng.normal(size=(S, 1, 3))
    spread = {"near": 0.02, "wide": 3.0, "opposite": 0.01}.get(kind, 0.02)
    d = axis / np.linalg.norm(axis, axis=2, keepdims=True) + spread * rng.normal(size=(S, nsat, 3))
    if kind == "opposite":
        d[:, ::2] *= -1
    d /= np.linalg.norm(d, axis=2, keepdims=True)
    r = {"surface": 1737.4 + 1e-3, "inside": 1000.0}.get(kind, 2037.4)
    pos = (d * r).astype(np.float32)
    if kind == "centre":
        pos[:, 0] = 0.0
    m, n = np.triu_indices(nsat, 1)
    snap = np.repeat(np.arange(S), m.size).astype(np.int32)
    pair = np.tile(m | (n << 16), S).astype(np.int32)
    order = rng.permutation(snap.size) if S % 2 else np.arange(snap.size)
    snap, pair = snap[order], pair[order]
    K = snap.size
    l, mm, nn = fibonacci_sphere(J)
    mask, margin = oracle.geo_mask(oracle.make_geo(pos, snap, pair), 1737.4, l, mm, nn, K, J)
    limb = margin < 1e-9
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    z = torch.zeros(K, device="cuda")
    geo = dict(snap=cu(snap), pair=cu(pair), sat_pos=cu(pos))
    cfg = V.DftConfig.geometric(precision=V.PREC_FAST, occluded_value=1.0)
    Vg = V.vis_dft(cfg, z, z, z, *map(cu, (l, mm, nn)), torch.zeros(J, device="cuda"), **geo).cpu().numpy()
    Fg = V.recon(cfg.with_(norm=1.0), z, z, z, torch.ones(K, dtype=torch.complex64, device="cuda"), *map(cu, (l, mm, nn)),
                 **geo).cpu().numpy()
    rows, pix = ~limb.any(1), ~limb.any(0)
    assert np.array_equal(np.round(Vg.real[rows]).astype(np.int64), mask.sum(1)[rows])
    assert np.array_equal(np.round(Fg.real[pix]).astype(np.int64), (~mask).sum(0)[pix])
