"""Pixels whose direction is (0, 0, 0) (the padding of a sky to a round size): no satellite hides
them, whatever the pixels around them, as the exact predicate (s . p < 0) has it.  Satellites
100 km above the ground (the Moon fills 71 degrees of their sky) and padding of one pixel,
of a few among real ones, of whole patches, and skies on both sides of the small order's
16,384 pixels.  Zero phase, so that the sums count rows and pixels: exact integers against the
FP64 oracle's mask."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("J,zeros", [(700, 1), (4096, 5), (4096, 600), (17000, 7)])
def test_zero_directions_are_never_hidden(oracle, J, zeros):
    import viss_recon_shade_gb300 as V
    from viss_recon_shade_gb300.synth import fibonacci_sphere
    rng = np.random.default_rng(J + zeros)
    l, m, n = (np.array(x, np.float32) for x in fibonacci_sphere(J))
    pad = rng.permutation(J)[:zeros]
    l[pad] = m[pad] = n[pad] = 0.0
    # shadows about +x, where the spatial order puts a direction of no axis, and about random axes
    S, nsat = 40, 4
    axis = rng.normal(size=(S, 1, 3))
    axis[::2] = np.array([-1.0, 0.0, 0.0]) + 0.1 * rng.normal(size=(S // 2, 1, 3))
    d = axis / np.linalg.norm(axis, axis=2, keepdims=True) + 0.02 * rng.normal(size=(S, nsat, 3))
    pos = (1837.4 * d / np.linalg.norm(d, axis=2, keepdims=True)).astype(np.float32)
    a, b = np.triu_indices(nsat, 1)
    snap = np.repeat(np.arange(S), a.size).astype(np.int32)
    pair = np.tile(a | (b << 16), S).astype(np.int32)
    K = snap.size
    mask, margin = oracle.geo_mask(oracle.make_geo(pos, snap, pair), 1737.4, l, m, n, K, J)
    assert not mask[:, pad].any()
    limb = margin < 1e-9
    limb[:, pad] = False  # no direction, no limb
    cu = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    z = torch.zeros(K, device="cuda")
    geo = dict(snap=cu(snap), pair=cu(pair), sat_pos=cu(pos))
    cfg = V.DftConfig.geometric(precision=V.PREC_FAST, occluded_value=1.0).with_(norm=1.0)
    F = V.recon(cfg, z, z, z, torch.ones(K, dtype=torch.complex64, device="cuda"), *map(cu, (l, m, n)), **geo).cpu().numpy()
    Vg = V.vis_dft(cfg, z, z, z, *map(cu, (l, m, n)), torch.zeros(J, device="cuda"), **geo).cpu().numpy()
    rows, pix = ~limb.any(1), ~limb.any(0)
    assert np.array_equal(np.round(F.real[pix]).astype(np.int64), (~mask).sum(0)[pix])
    assert np.array_equal(np.round(Vg.real[rows]).astype(np.int64), mask.sum(1)[rows])
