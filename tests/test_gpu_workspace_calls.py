"""viss_visscal_ws / viss_imagerecon_ws: the reference-shaped calls on a caller workspace give the
bits of the allocating ones (FAST reads the window columns, PLAIN packs them), report the
size they need, and refuse a short or misaligned workspace."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fast", "plain"])
@pytest.mark.parametrize("masked", [True, False])
def test_same_bits(precision, masked):
    import viss_recon_shade_gb300 as V
    from viss_recon_shade_gb300 import _lib as L
    from viss_recon_shade_gb300.synth import fibonacci_sphere, lognormal_sky
    K, res = 777, 33
    J = res * res
    rng = np.random.default_rng(5)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    uvw = [cu(np.ceil(rng.normal(0, 200, K)).astype(np.float32)) for _ in range(3)]
    lmn = list(map(cu, fibonacci_sphere(J)))
    b = cu(lognormal_sky(J, seed=2))
    M = [cu(rng.integers(lo, hi, K).astype(np.int32)) for lo, hi in ((0, 9), (12, 33), (0, 2), (2, 33))]
    wgt = cu(rng.uniform(0.2, 1, K).astype(np.float32))
    r1, r2 = V.recon_ratios(torch.stack(M, -1))
    p = V.PREC_FAST if precision == "fast" else V.PREC_PLAIN
    out = []
    ptr = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    vis, F = torch.empty(K, dtype=torch.complex64, device="cuda"), torch.empty(J, dtype=torch.complex64, device="cuda")
    mask = V.MASK_REF_QUIRK if masked else V.MASK_NONE
    a1 = (K, J, res, ptr(b), ptr(vis), *map(ptr, uvw), *map(ptr, lmn), *(map(ptr, M) if masked else [None] * 4), None, None,
          2.0, 2.0, 2.0, V.VARIANT_OPTIM, mask, p)
    a2 = (K, J, res, ptr(F), ptr(vis), *map(ptr, uvw), *map(ptr, lmn), ptr(wgt),
          *(map(ptr, (r1, r2, r1, r2)) if masked else [None] * 4), 2.0, 2.0, 2.0, p)
    L.check(L.lib.viss_visscal(*a1, st), "viss_visscal")
    L.check(L.lib.viss_imagerecon(*a2, st), "viss_imagerecon")
    out = vis.clone(), F.clone()
    for fn, a, o, want in ((L.lib.viss_visscal_ws, a1, vis, out[0]), (L.lib.viss_imagerecon_ws, a2, F, out[1])):
        nb = C.c_size_t(0)
        assert fn(*a, None, C.byref(nb), st) == L.VISS_OK and nb.value > 0
        ws = torch.empty(nb.value + 256, dtype=torch.uint8, device="cuda")
        short = C.c_size_t(nb.value - 1)
        assert fn(*a, C.c_void_p(ws.data_ptr()), C.byref(short), st) == L.VISS_ERR_WORKSPACE
        assert fn(*a, C.c_void_p(ws.data_ptr() + 16), C.byref(nb), st) == L.VISS_ERR_WORKSPACE
        assert fn(*a, None, None, st) == L.VISS_ERR_INVALID
        o.zero_()
        if o is F:
            vis.copy_(out[0])
        assert fn(*a, C.c_void_p(ws.data_ptr()), C.byref(nb), st) == L.VISS_OK
        torch.cuda.synchronize()
        assert torch.equal(o, want)
