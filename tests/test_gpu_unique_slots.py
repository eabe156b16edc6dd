"""The first table of viss_unique_uvw holds the rows of an orbit campaign at any frequency: one table
pass, by the launches counted, from 1 to 30 MHz and for positions that share no row.
The rows themselves against the baselines' own unique rows."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _unique(V, pos, lam):
    u, v, w, _, _ = V.baseline_uvw(pos, lam, ordered=True, rounding=True)
    q = torch.stack([u, v, w], -1).long() + (1 << 20)
    key = torch.unique((q[:, 0] << 42) | (q[:, 1] << 21) | q[:, 2])
    return torch.stack([key >> 42, (key >> 21) & 0x1FFFFF, key & 0x1FFFFF]).sub_(1 << 20).float()


@pytest.mark.parametrize("mhz", [1.0, 10.0, 20.0, 30.0, "random"])
def test_one_table_pass(mhz):
    import viss_recon_shade_gb300 as V
    from viss_recon_shade_gb300 import _lib as L
    if mhz == "random":  # 56 new rows a snapshot: as many unique rows as rows
        g = torch.Generator(device="cuda").manual_seed(1)
        pos, lam = 1500.0 * torch.randn(100003, 8, 3, device="cuda", generator=g).clamp_(-2, 2), 10.0
    else:
        r1 = (0.0, 1e3, 4.45e3, 6e3, 9.1e3, 16.2e3, 35.3e3, 100e3)
        cfg = V.OrbitConfig(nsat=8, orbit_res=86400, orbit_counts=14, r1_m=r1, r2_m=tuple(x / 10 for x in r1))
        pos, lam = V.orbit_positions(cfg), 300.0 / mhz
    n0 = L.lib.viss_launch_count()
    few = V.unique_uvw(pos, 1e5 * lam, capacity=1 << 23)  # a handful of rows: no table could fill
    n1 = L.lib.viss_launch_count()
    got = V.unique_uvw(pos, lam, capacity=1 << 23)
    assert 0 < few[0].numel() < 1 << 16 and L.lib.viss_launch_count() - n1 == n1 - n0
    assert torch.equal(torch.stack(list(got)), _unique(V, pos, lam))
