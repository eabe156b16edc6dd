"""FP64 orbits and their baselines (viss_orbit_positions with fp64, viss_baseline_uvw with
pos64) against the oracle's FP64 restatement, where the block and table edges lie: 2 to 32
satellites (one pair a snapshot up to 992), windows that end in a block, more orbits than
one block's RAAN table, separations beyond the series of sqrt(1 - x^2), zero-filled samples
and an eccentric orbit (the general kernel).

Tolerance: a position carries the rounding of an angle of at most 2 pi + the RAAN (a few
2^-53 of it) and a dozen FP64 products, below 1e-14 of the semi-major axis; 1e-13 leaves the
libraries' sin and cos room.  Baselines are one FP64 difference and product rounded to
float: within one float ulp of the oracle's quotient."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsat,res,counts,e,scale", [(2, 360, 7, 0.0, 1.0), (3, 363, 30, 0.0, 1.0), (5, 1440, 1, 0.0, 5.0),
                                                     (8, 777, 16, 0.0, 1.0), (32, 360, 2, 0.0, 20.0), (8, 360, 3, 0.01, 1.0)])
@pytest.mark.parametrize("ordered", [True, False])
def test_f64_positions_and_baselines(oracle, nsat, res, counts, e, scale, ordered):
    import viss_recon_shade_gb300 as V
    r1 = tuple(scale * 100e3 * i / (nsat - 1) for i in range(nsat))  # up to 2,000 km: x = d / 2a = 0.49
    r2 = tuple(x / 10 for x in r1)
    kw = dict(incl_deg=30.0, argp_deg=17.0, raan_step_deg=0.08)
    cfg = V.OrbitConfig(nsat=nsat, orbit_res=res, orbit_counts=counts, index=3, e=e, r1_m=r1, r2_m=r2, fp64=True, **kw)
    pos, pos64 = V.orbit_positions(cfg, want_f64=True)
    ref = oracle.orbit_positions_f64(oracle.make_orbit_cfg(nsat, res, counts, index=3, a_km=cfg.a_km, e=e, r1_m=r1, r2_m=r2,
                                                           **kw))
    p = pos64.cpu().numpy()
    assert p.shape == ref.shape
    assert np.abs(p - ref).max() <= 1e-13 * cfg.a_km
    assert np.array_equal(pos.cpu().numpy(), p.astype(np.float32))
    u, v, w, snap, pair = V.baseline_uvw(pos, 29.97, ordered=ordered, rounding=False, pos64=pos64)
    ru, rv, rw, rs, rp = oracle.uvw(np.zeros((2, nsat, 3), np.float32), 29.97, ordered=ordered, rounding=False)
    P = rs.size // 2
    assert np.array_equal(snap.cpu().numpy(), np.repeat(np.arange(p.shape[0]), P))
    assert np.array_equal(pair.cpu().numpy(), np.tile(rp[:P], p.shape[0]))
    m, n = rp[:P] & 0xFFFF, rp[:P] >> 16
    d = ((p[:, n] - p[:, m]) * 1e3 / 29.97).reshape(-1, 3)
    for c, x in enumerate((u, v, w)):
        assert np.all(np.abs(x.cpu().numpy() - d[:, c]) <= np.spacing(np.abs(d[:, c]).astype(np.float32)))
    # with the ceil: the oracle's integers
    for got, c in zip(V.baseline_uvw(pos, 29.97, ordered=ordered, rounding=True, pos64=pos64)[:3], range(3)):
        assert np.array_equal(got.cpu().numpy(), np.ceil(d[:, c]).astype(np.float32))
