"""Sums of partial results beyond FP32's range: a pass split into several work items adds their
partial sums, which may be infinite one by one, overflow on the way to a finite sum, or be scaled
back into range by the norm.  The result is that of the sum in 64 bits: infinities stay
infinities, finite values are within the usual 1e-5."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

K, J = 5000, 4097  # eight and more items in each direction


def _pass():
    from viss_recon_shade_gb300.synth import fibonacci_sphere
    cu = lambda x: torch.from_numpy(np.ascontiguousarray(x, dtype=np.float32)).cuda()  # noqa: E731
    return [torch.zeros(K, device="cuda")] * 3, list(map(cu, fibonacci_sphere(J))), cu


@pytest.mark.parametrize("at", [0, 1500, J - 1])
@pytest.mark.parametrize("value", [np.inf, -np.inf])
def test_vis_one_infinite_pixel(at, value):
    import viss_recon_shade_gb300 as V
    uvw, lmn, cu = _pass()
    b = np.ones(J, np.float32)
    b[at] = value
    Vg = V.vis_dft(V.DftConfig(precision=V.PREC_FAST, n_offset=0.0), *uvw, *lmn, cu(b)).cpu().numpy()
    assert np.all(Vg.real == value)


def test_vis_partials_overflow_on_the_way():
    import viss_recon_shade_gb300 as V
    uvw, lmn, cu = _pass()
    b = np.zeros(J, np.float32)
    b[[10, 1000, 2000, 3000, 4000]] = 3e38, 2e38, 1e38, -3e38, -2e38  # partials of 32 to 512 pixels apart
    Vg = V.vis_dft(V.DftConfig(precision=V.PREC_FAST, n_offset=0.0), *uvw, *lmn, cu(b)).cpu().numpy()
    assert np.all(np.abs(Vg.real - 1e38) <= 1e-5 * 3e38)


def test_recon_sum_scaled_back_by_the_norm():
    import viss_recon_shade_gb300 as V
    uvw, lmn, cu = _pass()
    y = torch.full((K,), 2e36, dtype=torch.complex64, device="cuda")  # 1e40 in all, 2e38 in 100 rows
    cfg = V.DftConfig(precision=V.PREC_FAST, n_offset=0.0, norm=1.0 / K)
    F = V.recon(cfg, *uvw, y, *lmn).cpu().numpy()
    assert np.all(np.abs(F.real - 2e36) <= 1e-5 * 2e36)


def test_recon_one_infinite_row_and_norm_out_of_range():
    import viss_recon_shade_gb300 as V
    uvw, lmn, cu = _pass()
    y = torch.ones(K, dtype=torch.complex64, device="cuda")
    F = V.recon(V.DftConfig(precision=V.PREC_FAST, n_offset=0.0, norm=3e38), *uvw, y, *lmn).cpu().numpy()
    assert np.all(F.real == np.inf)
