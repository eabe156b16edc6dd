"""Passes too small to fill the chip in full work items: the sky is cut into chunks of 32 to
256 pixels and the rows into segments of 32 to 128, and their partial sums are added 32
outputs to a block, eight partials side by side.  Sizes on both sides of those edges, against
the FP64 oracle at the usual bounds (normwise 1e-5, max 3e-5 of the largest value)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,J", [(1, 33), (31, 65), (33, 1023), (1025, 95), (3360, 2048), (5000, 4097), (28672, 6145)])
@pytest.mark.parametrize("ref", [False, True])
def test_small_passes(oracle, K, J, ref):
    import viss_recon_shade_gb300 as V
    from viss_recon_shade_gb300.synth import fibonacci_sphere, lognormal_sky
    rng = np.random.default_rng(K + J)
    u, v, w = (rng.normal(0, 400, K).astype(np.float32) for _ in range(3))
    l, m, n = fibonacci_sphere(J)
    b = lognormal_sky(J, seed=1, n_points=min(20, J))
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    res = max(8, int(np.sqrt(J)))
    M1 = rng.integers(0, res - 1, K)
    M2 = np.minimum(res - 1, M1 + rng.integers(0, res, K))
    M3 = np.where(rng.random(K) < 0.5, 0, rng.integers(0, 6, K))
    shade = np.stack([M1, M2, M3, M3 + rng.integers(0, res, K)], -1).astype(np.int32)
    kw = dict(mask=V.MASK_REF_QUIRK, recon_mask=V.RECON_MASK_REF, res=res) if ref else {}
    ok = dict(mask_mode=1, res=res, occluded_value=240.0) if ref else {}
    cfg = V.DftConfig(precision=V.PREC_FAST, **kw)
    Vg = V.vis_dft(cfg, *map(cu, (u, v, w, l, m, n, b)), shade=cu(shade) if ref else None).cpu().numpy()
    Fg = V.recon(cfg, *map(cu, (u, v, w)), cu(Vg), *map(cu, (l, m, n)), shade=cu(shade) if ref else None).cpu().numpy()
    Vo = oracle.vis_dft(oracle.make_cfg(**ok), u, v, w, l, m, n, b, shade=shade if ref else None)
    Fo = oracle.recon(oracle.make_cfg(norm=1.0 / K, **(dict(res=res, recon_ref_mask=True) if ref else {})), u, v, w, None, Vg,
                      l, m, n, shade=shade if ref else None)
    for g, o in ((Vg, Vo), (Fg, Fo)):
        d = g.astype(np.complex128) - o
        assert np.linalg.norm(d) <= 1e-5 * np.linalg.norm(o) and np.abs(d).max() <= 3e-5 * np.abs(o).max()
