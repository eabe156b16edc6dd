"""The sky's spatial order in one block (up to 16,384 pixels) and by the device-wide sort above:
whole skies, a patch that falls into one cell of the counting sort, and repeated directions.
Whatever the order, every pixel has to come out in its place: zero-phase reconstructions count
the rows that see it, compared with the FP64 oracle's mask (limb pixels left out), and a second
pass gives the same bits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("J,kind", [(1, "sphere"), (1023, "sphere"), (1025, "patch"), (16384, "sphere"), (16384, "patch"),
                                    (16385, "sphere"), (5000, "same")])
def test_order_places_every_pixel(oracle, J, kind):
    import viss_recon_shade_gb300 as V
    from viss_recon_shade_gb300.synth import fibonacci_sphere
    rng = np.random.default_rng(J)
    l, m, n = fibonacci_sphere(J)
    if kind != "sphere":  # ~0.5 degrees about one direction, or that direction alone
        d = np.array([0.3, -0.9, 0.2]) + (0.005 if kind == "patch" else 0.0) * rng.normal(size=(J, 3))
        l, m, n = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32).T.copy()
    S, nsat = 24, 5
    # the limb crosses the patch: satellites around the direction's shadow edge
    p = rng.normal(size=(S, 1, 3)) + 0.02 * rng.normal(size=(S, nsat, 3))
    pos = (2037.4 * p / np.linalg.norm(p, axis=2, keepdims=True)).astype(np.float32)
    a, b = np.triu_indices(nsat, 1)
    snap = np.repeat(np.arange(S), a.size).astype(np.int32)
    pair = np.tile(a | (b << 16), S).astype(np.int32)
    K = snap.size
    mask, margin = oracle.geo_mask(oracle.make_geo(pos, snap, pair), 1737.4, l, m, n, K, J)
    cu = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    z = torch.zeros(K, device="cuda")
    cfg = V.DftConfig.geometric(precision=V.PREC_FAST).with_(norm=1.0)
    args = (cfg, z, z, z, torch.ones(K, dtype=torch.complex64, device="cuda"), *map(cu, (l, m, n)))
    geo = dict(snap=cu(snap), pair=cu(pair), sat_pos=cu(pos))
    F = V.recon(*args, **geo)
    pix = ~(margin < 1e-9).any(0)
    assert np.array_equal(np.round(F.real.cpu().numpy()[pix]).astype(np.int64), (~mask).sum(0)[pix])
    assert torch.equal(F, V.recon(*args, **geo))
