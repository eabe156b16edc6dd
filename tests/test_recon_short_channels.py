"""Reconstructions of many channels with few rows each: where whole channels fill the chip their rows
are not cut into segments, whose partial sums would cost more than the shorter items gain.  The
workspace shows it (no partial sums in it), on any machine; on a GPU each channel equals its
own reconstruction."""
import ctypes as C

import numpy as np
import pytest


def _bytes(nch, rows, J, **kw):
    import viss_recon_shade_gb300 as V
    from viss_recon_shade_gb300 import _lib as L
    off = (C.c_int64 * (nch + 1))(*[rows * c for c in range(nch + 1)])
    b = L.Batch()
    b.nch, b.row_off = nch, C.cast(off, C.POINTER(C.c_int64))
    cfg = V.DftConfig(**kw).c(rows)
    return L.lib.viss_recon_batch_workspace(C.byref(cfg), C.byref(b), nch * rows, J, None, None)


@pytest.mark.parametrize("nch,rows,J,whole", [(64, 100, 20164, True), (64, 60, 5041, True), (16, 100, 20164, True),
                                              (4, 2000, 5041, False), (1, 400, 1024, False)])
def test_segments_by_workspace(nch, rows, J, whole):
    pad = -(-J // 1024) * 1024
    records = 32 * pad + 32 * nch * rows + 4096  # pixel and row records, flags
    assert (_bytes(nch, rows, J) <= records) == whole


@pytest.mark.gpu
@pytest.mark.parametrize("nch,rows,J", [(64, 100, 2048), (16, 130, 20000), (3, 513, 5000), (5, 1, 3000)])
@pytest.mark.parametrize("ints", [False, True])
def test_each_channel_is_its_own(nch, rows, J, ints):
    torch = pytest.importorskip("torch")
    import viss_recon_shade_gb300 as V
    from viss_recon_shade_gb300.synth import fibonacci_sphere
    rng = np.random.default_rng(nch + rows)
    cu = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    sizes = np.maximum(rows + rng.integers(-rows // 3, rows // 3 + 1, nch), 1)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    K = int(off[-1])
    u, v, w = (rng.normal(0, 200, K).astype(np.float32) for _ in range(3))
    if ints:
        u, v, w = np.ceil(u), np.ceil(v), np.ceil(w)
    y = cu((rng.normal(size=K) + 1j * rng.normal(size=K)).astype(np.complex64))
    u, v, w = map(cu, (u, v, w))
    lmn = list(map(cu, fibonacci_sphere(J)))
    b = V.ChannelBatch(V.DftConfig(), u, v, w, off, *lmn, torch.ones(nch, J, device="cuda"))
    F = b.recon(y)
    for c in range(nch):
        s = slice(int(off[c]), int(off[c + 1]))
        Fc = V.recon(V.DftConfig(), u[s].clone(), v[s].clone(), w[s].clone(), y[s].clone(), *lmn)
        assert torch.linalg.vector_norm(F[c] - Fc) <= 2e-6 * torch.linalg.vector_norm(Fc)
