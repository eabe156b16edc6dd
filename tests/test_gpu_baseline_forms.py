"""viss_baseline_uvw in its four forms (FP32 and FP64 positions, with and without the ceil), staged and a
thread a row: sizes around the blocks of 256 rows and beyond the 2,048-row ones, 1 to 992 pairs a
snapshot, against numpy's FP64 quotients; and a small call of any form takes one launch's
latency, not a chain of a thread's divisions (at most 2.5 times the shortest form's time,
the least of many: 6 against 5 us, a chain of eight rows took 23)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,nsat", [(1, 2), (255, 2), (257, 2), (5, 3), (120, 8), (9, 8), (10, 8), (3, 32), (4000, 8), (700, 16)])
@pytest.mark.parametrize("ordered", [True, False])
@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("rounding", [True, False])
def test_rows(S, nsat, ordered, fp64, rounding):
    import viss_recon_shade_gb300 as V
    rng = np.random.default_rng(S * nsat)
    p64 = rng.normal(0, 50.0, (S, nsat, 3))
    p64[S // 2:, 1] = p64[S // 2:, 0]  # equal positions
    p32 = p64.astype(np.float32)
    pos = torch.from_numpy(p32).cuda()
    got = V.baseline_uvw(pos, 29.97, ordered=ordered, rounding=rounding, pos64=torch.from_numpy(p64).cuda() if fp64 else None)
    m, n = np.array([(i, j) for i in range(nsat) for j in range(nsat) if (i != j if ordered else i < j)]).T
    d = p64[:, n] - p64[:, m] if fp64 else (p32[:, n] - p32[:, m]).astype(np.float64)
    x = (d * 1e3 / 29.97).reshape(-1, 3)
    for c in range(3):
        g = got[c].cpu().numpy()
        if rounding:
            assert np.array_equal(g, np.ceil(x[:, c]).astype(np.float32))
        else:
            assert np.all(np.abs(g - x[:, c]) <= np.spacing(np.abs(x[:, c]).astype(np.float32)))
    assert np.array_equal(got[3].cpu().numpy(), np.repeat(np.arange(S), m.size))
    assert np.array_equal(got[4].cpu().numpy(), np.tile(m | (n << 16), S))


def test_small_calls_are_short():
    import ctypes as C

    from viss_recon_shade_gb300 import _lib as L
    S, nsat = 120, 8
    p64 = torch.randn(S, nsat, 3, dtype=torch.float64, device="cuda")
    pos = p64.float()
    out = [torch.empty(S * nsat * (nsat - 1), device="cuda", dtype=t) for t in (torch.float32,) * 3 + (torch.int32,) * 2]
    ptr = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    us = {}
    for form in ((None, 1), (None, 0), (p64, 1), (p64, 0)):
        best = float("inf")
        for _ in range(20):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(50):
                assert L.lib.viss_baseline_uvw(ptr(pos), ptr(form[0]), S, nsat, 1, 30.0, form[1], *map(ptr, out), st) == L.VISS_OK
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) / 50 * 1e3)
        us[(form[0] is not None, form[1])] = best
    assert max(us.values()) <= 2.5 * min(us.values()), us
