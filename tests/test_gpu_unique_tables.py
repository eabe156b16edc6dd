"""viss_unique_uvw where its table, run length and sort keys change: more unique rows than the
first table's 2^22 slots (a larger one follows), coordinates that use 1 to 21 bits of a key
field, one snapshot, and run lengths that do not divide S.  The rows must equal numpy's
sorted unique rows of the oracle's baselines exactly."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,nsat,spread_km,lam", [(90001, 8, 50.0, 10.0), (1, 3, 50.0, 10.0), (17, 5, 0.0, 30.0),
                                                  (4099, 6, 1e-3, 10.0), (3001, 4, 2000.0, 10.0)])
def test_unique_rows(oracle, S, nsat, spread_km, lam):
    import viss_recon_shade_gb300 as V
    rng = np.random.default_rng(S)
    pos = rng.normal(0, spread_km, (S, nsat, 3)).clip(-2.6 * spread_km, 2.6 * spread_km).astype(np.float32)
    u, v, w, _, _ = oracle.uvw(pos, lam, ordered=True, rounding=True)
    q = np.stack([u, v, w], -1).astype(np.int64) + (1 << 20)
    key = np.unique((q[:, 0] << 42) | (q[:, 1] << 21) | q[:, 2])
    if S == 90001:
        assert key.size > 1 << 22  # more than the first table holds
    got = V.unique_uvw(torch.from_numpy(pos).cuda(), lam)
    ref = [(key >> 42), (key >> 21) & 0x1FFFFF, key & 0x1FFFFF]
    for g, r in zip(got, ref):
        assert np.array_equal(g.cpu().numpy(), (r - (1 << 20)).astype(np.float32))
