"""Satellites from ten to ten thousand Moon radii away: the Moon is small in their sky, and the FP32
cosine of its angular radius a (3e-8 off) no longer gives a itself (3e-8 / sin a).  The cones that
show or hide a snapshot's pixels as a whole have to cover that.  Two satellites 60 degrees
apart, and pixels a few 1e-6 rad inside their shadows, on the side away from each other where
the cone that bounds both ends; zero phase, exact row counts against the FP64 oracle's mask."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radii", [10.0, 100.0, 300.0, 1000.0, 3000.0, 10000.0])
@pytest.mark.parametrize("inside", [1e-6, 5e-6])
def test_shadow_edges(oracle, radii, inside):
    import viss_recon_shade_gb300 as V
    rng = np.random.default_rng(int(radii))
    S = 600
    unit = lambda x: x / np.linalg.norm(x, axis=-1, keepdims=True)  # noqa: E731
    c = unit(rng.normal(size=(S, 3)))
    t = unit(np.cross(c, rng.normal(size=(S, 3))))
    r = 1737.4 * radii * rng.uniform(0.8, 1.25, (S, 1))
    pos = np.empty((S, 2, 3), np.float32)
    pix = []
    for i, sgn in enumerate((1.0, -1.0)):
        pos[:, i] = -r * (np.cos(np.pi / 6) * c + sgn * np.sin(np.pi / 6) * t)
        q = -pos[:, i].astype(np.float64)
        al = np.arcsin(1737.4 / np.linalg.norm(q, axis=1))[:, None] - inside
        q = unit(q)
        out = unit(sgn * (t - (t * q).sum(1, keepdims=True) * q))  # away from the other satellite
        pix.append(np.cos(al) * q + np.sin(al) * out)
    s = np.concatenate(pix)[rng.permutation(2 * S)].astype(np.float32)
    l, m, n = s.T.copy()
    J = l.size
    snap, pair = np.arange(S, dtype=np.int32), np.full(S, 1 << 16, np.int32)
    mask, margin = oracle.geo_mask(oracle.make_geo(pos, snap, pair), 1737.4, l, m, n, S, J)
    assert mask.any(0).mean() > 0.8  # the pixels are hidden where they were meant to be
    cu = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    z = torch.zeros(S, device="cuda")
    geo = dict(snap=cu(snap), pair=cu(pair), sat_pos=cu(pos))
    cfg = V.DftConfig.geometric(precision=V.PREC_FAST, occluded_value=1.0).with_(norm=1.0)
    F = V.recon(cfg, z, z, z, torch.ones(S, dtype=torch.complex64, device="cuda"), *map(cu, (l, m, n)), **geo).cpu().numpy()
    assert np.array_equal(np.round(F.real).astype(np.int64), (~mask).sum(0))
    # one snapshot a block: the vis kernel's cone is that snapshot's own
    rows = rng.permutation(S)[:6]
    for k in rows:
        g1 = dict(snap=cu(snap[k:k + 1]), pair=cu(pair[k:k + 1]), sat_pos=cu(pos))
        V1 = V.vis_dft(cfg, z[:1], z[:1], z[:1], *map(cu, (l, m, n)), torch.zeros(J, device="cuda"), **g1).cpu().numpy()
        assert round(float(V1.real[0])) == mask[k].sum()
