"""The reconstruction's row segments hold every row once: channels of one row, of a few, and of
enough for segments of unequal lengths (four work items per CTA and more), unmasked and
geometric.  Zero phase and whole weights, sums below 5e5: exact to the nearest integer."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,J", [((4999,), 12289), ((7001, 1, 33, 4096), 12289), ((8191, 0, 513), 20001), ((9000,), 1500)])
@pytest.mark.parametrize("mask", ["none", "geo"])
def test_every_row_once(oracle, rows, J, mask):
    import viss_recon_shade_gb300 as V
    from viss_recon_shade_gb300.synth import fibonacci_sphere
    K = sum(rows)
    rng = np.random.default_rng(K)
    y = rng.integers(1, 51, K).astype(np.float32)
    off = np.concatenate([[0], np.cumsum(rows)])
    l, m, n = fibonacci_sphere(J)
    cu = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    z = torch.zeros(K, device="cuda")
    kw, hidden, pix = {}, None, np.ones(J, bool)
    cfg = V.DftConfig(mask=V.MASK_NONE, recon_mask=V.RECON_MASK_NONE, precision=V.PREC_FAST, phase_scale=1.0, n_offset=-1.0)
    if mask == "geo":
        S = 40
        d = rng.normal(size=(S, 1, 3)) + 0.02 * rng.normal(size=(S, 3, 3))
        pos = (2037.4 * d / np.linalg.norm(d, axis=2, keepdims=True)).astype(np.float32)
        snap = (np.arange(K) * S // K).astype(np.int32)
        pair = np.array([0 | 1 << 16, 0 | 2 << 16, 1 | 2 << 16], np.int32)[np.arange(K) % 3]
        # the oracle decides each (snapshot, pair) once
        us = np.repeat(np.arange(S), 3).astype(np.int32)
        up = np.tile(np.array([0 | 1 << 16, 0 | 2 << 16, 1 | 2 << 16], np.int32), S)
        hid, margin = oracle.geo_mask(oracle.make_geo(pos, us, up), 1737.4, l, m, n, us.size, J)
        hidden = np.asarray(hid, bool)
        which = snap * 3 + np.arange(K) % 3
        pix = ~(margin < 1e-9).any(0)
        kw = dict(snap=cu(snap), pair=cu(pair), sat_pos=cu(pos))
        cfg = V.DftConfig.geometric(precision=V.PREC_FAST)
    b = V.ChannelBatch(cfg.with_(norm=1.0), z, z, z, off, *map(cu, (l, m, n)), torch.zeros(len(rows), J, device="cuda"), **kw)
    F = b.recon(cu(y.astype(np.complex64)))
    F = F.cpu().numpy().reshape(len(rows), J)
    for c in range(len(rows)):
        k = np.arange(off[c], off[c + 1])
        if mask == "none":
            want = np.full(J, y[k].sum(dtype=np.float64))
        else:
            wsum = np.bincount(which[k], weights=y[k].astype(np.float64), minlength=hidden.shape[0])
            want = wsum @ (~hidden)
        assert np.array_equal(np.round(F[c].real)[pix], want[pix]), c
