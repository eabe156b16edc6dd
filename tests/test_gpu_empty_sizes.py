"""The reference-shaped calls on a workspace at empty sizes: no rows or no pixels do no work,
whatever the workspace held before (0xff bytes, as flag words: every error bit), and
viss_visscal_ws with a fine map gives the bits of the allocating call."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,J", [(0, 81), (77, 0), (0, 0), (77, 81)])
@pytest.mark.parametrize("fill", [0x00, 0xFF])
def test_imagerecon_ws_empty_sizes(K, J, fill):
    import viss_recon_shade_gb300 as V
    from viss_recon_shade_gb300 import _lib as L
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    f = torch.ones(256, device="cuda")
    vis = torch.ones(256, dtype=torch.complex64, device="cuda")
    F = torch.full((256,), 7.0, dtype=torch.complex64, device="cuda")
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    a = (K, J, 9, ptr(F), ptr(vis), *[ptr(f)] * 7, *[ptr(f)] * 4, 2.0, 2.0, 2.0, V.PREC_FAST)
    nb = C.c_size_t(0)
    assert L.lib.viss_imagerecon_ws(*a, None, C.byref(nb), st) == L.VISS_OK
    ws = torch.full((nb.value + 256,), fill, dtype=torch.uint8, device="cuda")
    assert L.lib.viss_imagerecon_ws(*a, ptr(ws), C.byref(nb), st) == L.VISS_OK, L.lib.viss_last_error()
    torch.cuda.synchronize()
    if K == 0:
        assert torch.count_nonzero(F[:J]) == 0
    assert torch.all(F[J:] == 7.0)


def test_visscal_ws_with_a_fine_map():
    import viss_recon_shade_gb300 as V
    from viss_recon_shade_gb300 import _lib as L
    from viss_recon_shade_gb300.synth import fibonacci_sphere, lognormal_sky
    K, res, J = 300, 21, 50
    rng = np.random.default_rng(3)
    cu = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    count, nxq = V.nxq(cu(rng.integers(1, J + 1, res * res).astype(np.float32)), J)
    nxq = nxq.float()
    uvw = [cu(np.ceil(rng.normal(0, 50, K)).astype(np.float32)) for _ in range(3)]
    lmn = list(map(cu, fibonacci_sphere(J)))
    FF = cu(lognormal_sky(res * res, seed=4))
    M = [cu(rng.integers(lo, hi, K).astype(np.int32)) for lo, hi in ((0, 9), (12, 21), (0, 2), (2, 21))]
    vis = torch.zeros(K, dtype=torch.complex64, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    a = (K, J, res, ptr(FF), ptr(vis), *map(ptr, uvw), *map(ptr, lmn), *map(ptr, M), ptr(nxq), ptr(count), 2.0, 2.0,
         2.0, V.VARIANT_OPTIM, V.MASK_REF_QUIRK, V.PREC_FAST)
    assert L.lib.viss_visscal(*a, st) == L.VISS_OK
    want = vis.clone()
    vis.zero_()
    nb = C.c_size_t(0)
    assert L.lib.viss_visscal_ws(*a, None, C.byref(nb), st) == L.VISS_OK and nb.value > 0
    ws = torch.full((nb.value,), 0xFF, dtype=torch.uint8, device="cuda")
    assert L.lib.viss_visscal_ws(*a, ptr(ws), C.byref(nb), st) == L.VISS_OK
    torch.cuda.synchronize()
    assert torch.equal(torch.view_as_real(vis), torch.view_as_real(want))
