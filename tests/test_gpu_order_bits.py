"""The same call gives the same bits: geometric reconstructions of skies that crowd into one cell of
the spatial order (a field of a degree, one direction repeated, dense patches among a whole
sky), of rows in no order (snapshots interleaved, so that the order in which a pixel's rows are
added depends on the pixels that share its patch), with fractional uvw and complex
visibilities whose sums show any change of order.  And against the FP64 oracle at the usual
1e-5."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("J,kind", [(33, "field"), (1025, "field"), (4096, "mixed"), (5000, "same"), (16384, "field"),
                                    (16384, "mixed"), (16385, "field")])
def test_repeated_calls(oracle, J, kind):
    import viss_recon_shade_gb300 as V
    from viss_recon_shade_gb300.synth import fibonacci_sphere
    rng = np.random.default_rng(J)
    l, m, n = (np.array(x, np.float32) for x in fibonacci_sphere(J))
    c = np.array([0.3, -0.9, 0.2])
    if kind == "mixed":  # five dense patches in a whole sky
        for c5 in rng.normal(size=(5, 3)):
            at = rng.permutation(J)[: J // 12]
            d = c5 / np.linalg.norm(c5) + 0.005 * rng.normal(size=(at.size, 3))
            l[at], m[at], n[at] = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32).T
    else:
        d = c + (0.01 if kind == "field" else 0.0) * rng.normal(size=(J, 3))
        l, m, n = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32).T.copy()
    S, nsat = 24, 5
    # satellites over the shadow's edge: some of the field's pixels are hidden from some of them
    c = c / np.linalg.norm(c)
    e = np.cross(c, rng.normal(size=(S, 3)))
    e /= np.linalg.norm(e, axis=1, keepdims=True)
    t = np.pi - np.arcsin(1737.4 / 2037.4) + 0.01 * rng.normal(size=(S, nsat))
    p = np.cos(t)[..., None] * c + np.sin(t)[..., None] * e[:, None]
    pos = (2037.4 * p).astype(np.float32)
    a, b = np.triu_indices(nsat, 1)
    order = rng.permutation(S * a.size)
    snap = np.repeat(np.arange(S), a.size).astype(np.int32)[order]
    pair = np.tile(a | (b << 16), S).astype(np.int32)[order]
    K = snap.size
    u, v, w = (rng.normal(0, 300, K).astype(np.float32) for _ in range(3))
    y = (rng.normal(size=K) + 1j * rng.normal(size=K)).astype(np.complex64)
    cu = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    cfg = V.DftConfig.geometric(precision=V.PREC_FAST)
    args = (cfg, *map(cu, (u, v, w, y, l, m, n)))
    geo = dict(snap=cu(snap), pair=cu(pair), sat_pos=cu(pos))
    F = V.recon(*args, **geo)
    for _ in range(12):
        assert torch.equal(torch.view_as_real(V.recon(*args, **geo)), torch.view_as_real(F))
    Fo = oracle.recon(oracle.make_cfg(mask_mode=3, phase_scale=1.0, n_offset=-1.0, occluded_value=0.0, norm=1.0 / K), u, v, w,
                      None, y, l, m, n, geo=oracle.make_geo(pos, snap, pair))
    assert np.linalg.norm(F.cpu().numpy() - Fo) <= 1e-5 * np.linalg.norm(Fo)
