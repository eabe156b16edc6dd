"""The work that users of this framework have it do, as cases to be timed and compared.

A case is a dict of plain values; `kind` says which chain of public entry points it runs:

  imaging      vis_dft + recon of one channel with the geometric Moon mask (continuous uvw of an orbit):
               the simulator's main pass, from a quick look to the 10 MHz and 30 MHz configurations
  fit_step     vis_dft_autograd forward and backward: one gradient of a sky fit
  channels     ChannelBatch.step(): many frequency channels of uneven length through one batched pass
  unmasked     vis_dft + recon of arbitrary continuous uvw, no mask, weights in the reconstruction
  reference    visscal + imagerecon with the reference programs' conventions: integer uvw, REF windows
  fine_map     nxq + vis_dft_map: a fine sky grid averaged onto coarse pixels under REF windows
  tables       orbit_positions + unique_uvw + shade_windows + normalise_shade: what the uvw and shade
               programs compute before any visibility
  continuous   orbit_positions (FP64) + baseline_uvw: the rows of the continuous-uvw configurations

Orbits, uvw, windows and skies are made here with plain torch, so that exact() needs none of the
package's code.
"""
from __future__ import annotations

import math

import torch

import viss_recon_shade_gb300 as V
from viss_recon_shade_gb300.autograd import vis_dft_autograd

MOON_KM = 1737.4
A_KM = MOON_KM + 300.0
DEV = "cuda"


def listed():
    return [
        # a quick look: one orbit window of 120 snapshots on a 2,048-pixel sky, where launches and latency count
        dict(name="imaging_quick", kind="imaging", nsat=8, snaps=120, pixels=2048, mhz=10.0, sky="lognormal"),
        # the small 1 MHz configuration (28,672 visibilities x 12,288 pixels)
        dict(name="imaging_1MHz", kind="imaging", nsat=8, snaps=1024, pixels=12288, mhz=1.0, sky="lognormal"),
        # the 10 MHz configuration (1,835,008 visibilities x 196,608 pixels)
        dict(name="imaging_10MHz", kind="imaging", nsat=8, snaps=65536, pixels=196608, mhz=10.0, sky="powerlaw"),
        # 30 MHz, 16 satellites (120 baselines), an eighth of the largest configuration's snapshots, ragged sizes
        dict(name="imaging_30MHz", kind="imaging", nsat=16, snaps=8191, pixels=196613, mhz=30.0, sky="powerlaw"),
        # one gradient of the differentiable 10 MHz configuration (458,752 visibilities x 49,152 pixels)
        dict(name="fit_step_10MHz", kind="fit_step", nsat=8, snaps=16384, pixels=49152, mhz=10.0, sky="lognormal"),
        # batched channels over 1-30 MHz with uneven snapshot counts
        dict(name="channels_24", kind="channels", nsat=8, nch=24, snaps_lo=512, snaps_hi=4096, pixels=49152),
        # baselines beyond the FAST path's reach: compensated phase, no geometry, odd sizes
        dict(name="unmasked_comp", kind="unmasked", rows=200003, pixels=65537, sigma=9000.0, precision="compensated"),
        # the reference's 1 MHz programs: 28,672 integer uvw on a RES = 111 grid
        dict(name="reference_1M", kind="reference", rows=28672, res=111, mhz=1.0),
        # the reference's 10 MHz programs: sorted integer uvw on a RES = 443 grid
        dict(name="reference_10M", kind="reference", rows=262144, res=443, mhz=10.0),
        # a fine 362 x 362 sky averaged onto 12,288 pixels
        dict(name="fine_map_362", kind="fine_map", rows=28672, res=362, pixels=12288, mhz=1.0),
        # the uvw and shade programs over 403,200 snapshots of 8 satellites at 10 MHz
        dict(name="tables_403200", kind="tables", nsat=8, orbit_res=86400, orbits=14, mhz=10.0, res=20940),
        # the rows of the 10 MHz configuration: 65,536 snapshots, 28 baselines, FP64 positions
        dict(name="continuous_65536", kind="continuous", nsat=8, orbit_res=12288, orbits=16, mhz=10.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["imaging", "imaging", "imaging", "fit_step", "channels", "unmasked", "reference", "fine_map",
                       "tables", "continuous"])
    if kind in ("imaging", "fit_step"):
        nsat = rng.choice([6, 7, 8, 8, 9, 12, 16])
        pairs = nsat * (nsat - 1) // 2
        pixels = _log(rng, 2048, 196608)
        most = min(65536, int(1.8e11 / (pairs * pixels)))
        return dict(kind=kind, nsat=nsat, snaps=_log(rng, 120, max(121, most)), pixels=pixels,
                    mhz=round(math.exp(rng.uniform(0.0, math.log(30.0))), 2), sky=rng.choice(["lognormal", "powerlaw"]))
    if kind == "channels":
        lo = _log(rng, 128, 1024)
        return dict(kind=kind, nsat=8, nch=rng.randint(2, 24), snaps_lo=lo, snaps_hi=lo * rng.randint(2, 4),
                    pixels=_log(rng, 4096, 49152))
    if kind == "unmasked":
        precision = rng.choice(["fast", "compensated"])
        return dict(kind=kind, rows=_log(rng, 2048, 262144), pixels=_log(rng, 2048, 131072),
                    sigma=round(rng.uniform(100.0, 3000.0 if precision == "fast" else 9000.0), 1), precision=precision)
    if kind == "reference":
        return dict(kind=kind, rows=_log(rng, 4096, 262144), res=_log(rng, 48, 443), mhz=rng.choice([1.0, 3.0, 10.0]))
    if kind == "fine_map":
        res = _log(rng, 96, 362)
        return dict(kind=kind, rows=_log(rng, 2048, 28672), res=res, pixels=res * res // rng.randint(3, 12),
                    mhz=rng.choice([1.0, 3.0]))
    if kind == "tables":
        return dict(kind=kind, nsat=rng.choice([4, 6, 8]), orbit_res=360 * rng.randint(4, 240), orbits=rng.randint(2, 14),
                    mhz=rng.choice([1.0, 3.0, 10.0]), res=rng.choice([2094, 6282, 20940]))
    return dict(kind=kind, nsat=rng.choice([4, 8, 16]), orbit_res=3 * _log(rng, 120, 4096), orbits=rng.randint(1, 16),
                mhz=round(rng.uniform(1.0, 30.0), 1))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _separations(nsat):
    """Along-track separations in metres at the two ends of the ramp: the reference's eight, else log-spaced."""
    if nsat == 8:
        r1 = [0.0, 1e3, 4.45e3, 6e3, 9.1e3, 16.2e3, 35.3e3, 100e3]
    else:
        r1 = [0.0] + [1e3 * 100.0 ** (i / (nsat - 2)) for i in range(nsat - 1)]
    return r1, [x / 10.0 for x in r1]


def _orbit(S, nsat, phase0, raan0):
    """S windowed snapshots of nsat satellites on inclined circular orbits: FP64 positions [S, nsat, 3] in km."""
    orbits = 16 if S >= 2048 else 1
    span = -(-S // orbits)
    g = torch.arange(S, device=DEV)
    k = (g // span).double()
    theta = 2 * math.pi / 3 * (g % span).double() / span + k * math.radians(10.0) + phase0
    raan = k * math.radians(0.08) + raan0
    r1, r2 = (torch.tensor(r, dtype=torch.float64, device=DEV) for r in _separations(nsat))
    ramp = 1.0 - (2.0 * g.double() / S - 1.0).abs()  # 0 .. 1 .. 0: r1 -> r2 -> r1
    sep = r1 + (r2 - r1) * ramp[:, None]
    w = theta[:, None] + 2.0 * torch.asin(sep / (2.0 * A_KM * 1e3))
    cr, sr, ci, si = torch.cos(raan)[:, None], torch.sin(raan)[:, None], math.cos(math.pi / 6), math.sin(math.pi / 6)
    cw, sw = torch.cos(w), torch.sin(w)
    return A_KM * torch.stack([cw * cr - sw * ci * sr, cw * sr + sw * ci * cr, sw * si], -1)


def _rows(pos, mhz, ordered=False):
    """Baseline rows, snapshot-major: uvw in wavelengths as FP64 [S * pairs, 3], snapshot and packed pair."""
    S, nsat = pos.shape[:2]
    pairs = [(m, n) for m in range(nsat) for n in range(nsat) if (m != n if ordered else m < n)]
    m = torch.tensor([p[0] for p in pairs], device=DEV)
    n = torch.tensor([p[1] for p in pairs], device=DEV)
    uvw = ((pos[:, n] - pos[:, m]) * (1e3 * mhz / 300.0)).reshape(-1, 3)
    snap = torch.arange(S, device=DEV, dtype=torch.int32).repeat_interleave(len(pairs))
    pair = (m | (n << 16)).to(torch.int32).repeat(S)
    return uvw, snap, pair


def _columns(uvw):
    return tuple(uvw[:, c].float().contiguous() for c in range(3))


def _sphere(J):
    i = torch.arange(J, device=DEV, dtype=torch.float64) + 0.5
    z = 1.0 - 2.0 * i / J
    r = torch.sqrt((1.0 - z * z).clamp_min(0.0))
    phi = math.pi * (3.0 - math.sqrt(5.0)) * i
    return (r * torch.cos(phi)).float(), (r * torch.sin(phi)).float(), z.float()


def _sky(n, kind, gen, mhz=10.0):
    J = n.numel()
    if kind == "lognormal":
        b = torch.exp(torch.randn(J, generator=gen, device=DEV, dtype=torch.float64))
    else:
        b = (1.0 + n.double()) ** 2 * 100.0 * mhz ** -2.5
    points = torch.randperm(J, generator=gen, device=DEV)[:max(1, J // 400)]
    b[points] += b.mean() * (5.0 + 45.0 * torch.rand(points.numel(), generator=gen, device=DEV, dtype=torch.float64))
    return b.float()


def _phases(gen):
    a = torch.rand(2, generator=gen, device=DEV, dtype=torch.float64).tolist()
    return 2 * math.pi * a[0], 2 * math.pi * a[1]


def _integer_uvw(rows, mhz, gen):
    """`rows` sorted unique integer uvw (ceil of an orbit's ordered baselines), spread over the whole set."""
    phase, raan = _phases(gen)
    S = max(256, rows // 40)
    while True:
        uvw, _, _ = _rows(_orbit(S, 8, phase, raan), mhz, ordered=True)
        q = torch.ceil(uvw).long() + (1 << 20)
        key = torch.unique((q[:, 0] << 42) | (q[:, 1] << 21) | q[:, 2])
        if key.numel() >= rows:
            break
        S *= 2
    key = key[torch.arange(rows, device=DEV) * key.numel() // rows]
    q = torch.stack([key >> 42, (key >> 21) & 0x1FFFFF, key & 0x1FFFFF], -1) - (1 << 20)
    return q.double()


def _windows(uvw, res):
    """Moon shade windows of the rows on a res x res grid, normalised (M1 <= M2, M3 <= M4, 0-based)."""
    r = uvw.norm(dim=1).clamp_min(1e-9)
    theta = math.pi - torch.atan2(uvw[:, 1], uvw[:, 0])
    phi = math.pi / 2 - torch.asin((uvw[:, 2] / r).clamp(-1.0, 1.0))
    half = math.atan(MOON_KM / (float(r.mean()) + MOON_KM))
    ti, pi_ = torch.round(theta / (2 * math.pi / res)), torch.round(phi / (math.pi / res))
    tr = round(half / (2 * math.pi / res))
    pr = tr // 2
    cols = []
    for c, d in ((ti, tr), (pi_, pr)):
        a, b = c - d, c + d
        a = torch.where(a <= 0, a + res, a)
        b = torch.where(b > res, b - res, b)
        cols += [torch.minimum(a, b) - 1, torch.maximum(a, b) - 1]
    return torch.stack(cols, -1).to(torch.int32)


def prepare(case, seed):
    gen = _gen(seed)
    kind = case["kind"]
    s = dict(kind=kind)
    if kind in ("imaging", "fit_step"):
        pos = _orbit(case["snaps"], case["nsat"], *_phases(gen))
        uvw, snap, pair = _rows(pos, case["mhz"])
        l, m, n = _sphere(case["pixels"])
        s.update(uvw=_columns(uvw), lmn=(l, m, n), bright=_sky(n, case["sky"], gen, case["mhz"]),
                 geo=dict(snap=snap, pair=pair, sat_pos=pos.float().contiguous()),
                 cfg=V.DftConfig.geometric(precision=V.PREC_FAST, occluded_value=0.0))
        if kind == "fit_step":
            K = uvw.shape[0]
            s["g"] = torch.randn(K, 2, generator=gen, device=DEV)
    elif kind == "channels":
        r = torch.randint(case["snaps_lo"], case["snaps_hi"] + 1, (case["nch"],), generator=torch.Generator().manual_seed(5)).tolist()
        l, m, n = _sphere(case["pixels"])
        uvws, snaps, pairs, poss, brights, off, s_off = [], [], [], [], [], [0], 0
        for c, S in enumerate(r):
            mhz = 30.0 ** (c / max(1, case["nch"] - 1))
            pos = _orbit(S, case["nsat"], *_phases(gen))
            uvw, snap, pair = _rows(pos, mhz)
            uvws.append(uvw); snaps.append(snap + s_off); pairs.append(pair); poss.append(pos.float())
            brights.append(_sky(n, "powerlaw", gen, mhz))
            off.append(off[-1] + uvw.shape[0])
            s_off += S
        u, v, w = _columns(torch.cat(uvws))
        s.update(uvw=(u, v, w), lmn=(l, m, n), bright=torch.stack(brights), off=off,
                 geo=dict(snap=torch.cat(snaps), pair=torch.cat(pairs), sat_pos=torch.cat(poss)))
        s["batch"] = V.ChannelBatch(V.DftConfig.geometric(precision=V.PREC_FAST, occluded_value=0.0), u, v, w, off, l, m, n,
                                    s["bright"], **s["geo"])
    elif kind == "unmasked":
        K = case["rows"]
        uvw = torch.randn(K, 3, generator=gen, device=DEV, dtype=torch.float64) * case["sigma"]
        l, m, n = _sphere(case["pixels"])
        p = V.PREC_COMPENSATED if case["precision"] == "compensated" else V.PREC_FAST
        s.update(uvw=_columns(uvw), lmn=(l, m, n), bright=_sky(n, "lognormal", gen),
                 wgt=0.2 + 0.8 * torch.rand(K, generator=gen, device=DEV),
                 cfg=V.DftConfig(mask=V.MASK_NONE, recon_mask=V.RECON_MASK_NONE, precision=p, phase_scale=1.0, n_offset=-1.0))
    elif kind == "reference":
        J = case["res"] ** 2
        uvw = _integer_uvw(case["rows"], case["mhz"], gen)
        shade = _windows(uvw, case["res"])
        l, m, n = _sphere(J)
        K = case["rows"]
        r1, r2 = shade[:, 0].float() / shade[:, 1].float(), shade[:, 2].float() / shade[:, 3].float()
        s.update(uvw=_columns(uvw), lmn=(l, m, n), bright=_sky(n, "lognormal", gen), res=case["res"], shade=shade,
                 M=[shade[:, c].contiguous() for c in range(4)], ratios=(r1, r2),
                 wgt=1.0 / torch.randint(1, 9, (K,), generator=gen, device=DEV).float(),
                 V=torch.zeros(K, dtype=torch.complex64, device=DEV), F=torch.zeros(J, dtype=torch.complex64, device=DEV))
    elif kind == "fine_map":
        res, J = case["res"], case["pixels"]
        X = res * res
        uvw = _integer_uvw(case["rows"], case["mhz"], gen)
        l, m, n = _sphere(J)
        # runs of consecutive fine pixels share a coarse pixel, a few of them moved elsewhere
        coarse = torch.arange(X, device=DEV) * J // X
        moved = torch.randperm(X, generator=gen, device=DEV)[:X // 50]
        keep = torch.ones(X, dtype=torch.bool, device=DEV)
        keep[torch.arange(J, device=DEV) * X // J] = False  # these would empty a coarse pixel
        keep[(torch.arange(J, device=DEV) * X + J - 1) // J] = False
        moved = moved[keep[moved]]
        coarse[moved] = torch.randint(0, J, (moved.numel(),), generator=gen, device=DEV)
        s.update(uvw=_columns(uvw), lmn=(l, m, n), FF=_sky(torch.zeros(X, device=DEV), "lognormal", gen),
                 NX=(coarse + 1).float(), coarse=coarse, J=J, res=res, shade=_windows(uvw, res),
                 cfg=V.DftConfig.reference(res))
    elif kind == "tables":
        r1, r2 = _separations(case["nsat"])
        s.update(orbit=V.OrbitConfig(nsat=case["nsat"], orbit_res=case["orbit_res"], orbit_counts=case["orbits"],
                                     index=1 + seed % 1000, r1_m=tuple(r1), r2_m=tuple(r2)),
                 lam=300.0 / case["mhz"], res=case["res"])
        # the number of unique rows depends on the orbit: they go to the front of a program's own arrays
        snaps = case["orbits"] * (case["orbit_res"] // 3)
        rows = min(case["nsat"] * (case["nsat"] - 1) * snaps, case["orbits"] << 18)
        s.update(table=torch.zeros(3, rows, device=DEV), shade=torch.zeros(rows, 4, dtype=torch.int32, device=DEV))
    else:
        r1, r2 = _separations(case["nsat"])
        s.update(orbit=V.OrbitConfig(nsat=case["nsat"], orbit_res=case["orbit_res"], orbit_counts=case["orbits"],
                                     index=1 + seed % 1000, a_km=A_KM, r1_m=tuple(r1), r2_m=tuple(r2), fp64=True),
                 lam=300.0 / case["mhz"])
    return s


# ------------------------------------------------------------------ the pass
def run(s):
    kind = s["kind"]
    if kind == "imaging":
        vis = V.vis_dft(s["cfg"], *s["uvw"], *s["lmn"], s["bright"], **s["geo"])
        return vis, V.recon(s["cfg"], *s["uvw"], vis, *s["lmn"], **s["geo"])
    if kind == "fit_step":
        x = s["bright"].detach().requires_grad_(True)
        vis = vis_dft_autograd(x, s["cfg"], *s["uvw"], *s["lmn"], **s["geo"])
        (torch.view_as_real(vis) * s["g"]).sum().backward()
        return vis.detach(), x.grad
    if kind == "channels":
        b = s["batch"]
        b.step()
        return b.V, b.F
    if kind == "unmasked":
        vis = V.vis_dft(s["cfg"], *s["uvw"], *s["lmn"], s["bright"])
        return vis, V.recon(s["cfg"], *s["uvw"], vis, *s["lmn"], wgt=s["wgt"])
    if kind == "reference":
        K, J, res = s["V"].numel(), s["F"].numel(), s["res"]
        V.visscal(K, J, res, s["bright"], s["V"], *s["uvw"], *s["lmn"], *s["M"])
        r1, r2 = s["ratios"]
        V.imagerecon(K, J, res, s["F"], s["V"], *s["uvw"], *s["lmn"], s["wgt"], r1, r2, r1, r2)
        return s["V"], s["F"]
    if kind == "fine_map":
        count, nxq = V.nxq(s["NX"], s["J"])
        return count, nxq, V.vis_dft_map(s["cfg"], *s["uvw"], *s["lmn"], s["FF"], nxq, count, shade=s["shade"])
    if kind == "tables":
        u, v, w = V.unique_uvw(V.orbit_positions(s["orbit"]), s["lam"])
        raw, mean_r = V.shade_windows(u, v, w, s["res"])
        K = u.numel()
        for c, x in enumerate((u, v, w)):
            s["table"][c, :K] = x
        s["shade"][:K] = V.normalise_shade(raw)
        return s["table"], s["shade"], K, mean_r
    pos, pos64 = V.orbit_positions(s["orbit"], want_f64=True)
    return (pos, pos64) + V.baseline_uvw(pos, s["lam"], ordered=False, rounding=False, pos64=pos64)


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Bytes: inputs read once and outputs written once.  Flops: the transforms' multiply-adds; per term of a
    pass a phase of three products, a sine, a cosine and a complex multiply-add by a real (12 operations)."""
    kind = case["kind"]
    if kind in ("imaging", "fit_step"):
        K, J = case["snaps"] * case["nsat"] * (case["nsat"] - 1) // 2, case["pixels"]
        geo = 8 * K + 12 * case["snaps"] * case["nsat"]
        return {"bytes": 2 * (12 * K + geo + 12 * J) + 4 * J + 8 * K + 8 * K + 8 * J, "flops": 2 * 12 * K * J}
    if kind == "channels":
        pairs = case["nsat"] * (case["nsat"] - 1) // 2
        K, J = case["nch"] * (case["snaps_lo"] + case["snaps_hi"]) // 2 * pairs, case["pixels"]
        return {"bytes": 2 * (20 * K + 12 * J) + 16 * K + 12 * case["nch"] * J, "flops": 2 * 12 * K * J}
    if kind == "unmasked":
        K, J = case["rows"], case["pixels"]
        return {"bytes": 44 * K + 36 * J, "flops": 2 * 12 * K * J}
    if kind == "reference":
        K, J = case["rows"], case["res"] ** 2
        return {"bytes": 76 * K + 36 * J, "flops": 2 * 12 * K * J}
    if kind == "fine_map":
        K, J, X = case["rows"], case["pixels"], case["res"] ** 2
        return {"bytes": 36 * K + 20 * J + 16 * X, "flops": 12 * K * J}
    S = case["orbits"] * (case["orbit_res"] // 3)
    if kind == "tables":
        # positions written and read once, the unique rows and their windows written (about 100,000 an orbit at 10 MHz)
        rows = min(case["nsat"] * (case["nsat"] - 1) * S, int(10000 * case["mhz"] * case["orbits"]))
        return {"bytes": 24 * S * case["nsat"] + 28 * rows, "flops": S * case["nsat"] * (case["nsat"] - 1) * 9}
    return {"bytes": S * (60 * case["nsat"] + 20 * case["nsat"] * (case["nsat"] - 1) // 2),
            "flops": S * (60 * case["nsat"] + 9 * case["nsat"] * (case["nsat"] - 1) // 2)}


# ------------------------------------------------------------------ 64-bit results
MOST_TERMS = 2.5e10  # some ten seconds of FP64 work


def _turns(uvw, lmn, scale, offset):
    u = torch.stack([c.double() for c in uvw], -1) * scale
    p = torch.stack([lmn[0].double(), lmn[1].double(), lmn[2].double() + offset], 0)
    return u, p


def _visible(geo, lmn, k0, k1):
    """[k1 - k0, J] in FP64: neither satellite of the row has the Moon between itself and the pixel."""
    s = torch.stack([c.double() for c in lmn], 0)
    a = (s * s).sum(0)
    snap, pair = geo["snap"][k0:k1].long(), geo["pair"][k0:k1].long()
    ok = None
    for sat in (pair & 0xFFFF, pair >> 16):
        p = geo["sat_pos"][snap, sat].double()
        b = p @ s
        c = ((p * p).sum(1) - MOON_KM ** 2)[:, None]
        see = ~((b < 0) & (b * b - a * c > 0))
        ok = see if ok is None else ok & see
    return ok


def _both_ways(s, bright, weight, scale, offset, norm, visible=None, value=None, seen=None, y=None):
    """The visibilities of `bright`, and the reconstruction of `y` (default: those visibilities rounded to
    complex64, as a pass hands them on) times `weight`, in FP64, rows in chunks.  visible(k0, k1): mask of both;
    value(k0, k1): the brightness of every (row, pixel); seen(k0, k1): mask of the reconstruction alone."""
    u, p = _turns(s["uvw"], s["lmn"], scale, offset)
    K, J = u.shape[0], p.shape[1]
    vis = torch.empty(K, dtype=torch.complex128, device=DEV)
    F = torch.zeros(J, dtype=torch.complex128, device=DEV)
    b = None if bright is None else bright.double()
    step = max(1, int(2.5e8) // J)
    for k0 in range(0, K, step):
        k1 = min(K, k0 + step)
        t = u[k0:k1] @ p
        t = (t - torch.round(t)) * (2 * math.pi)
        c, d = torch.cos(t), torch.sin(t)
        del t
        ok = visible(k0, k1) if visible else None
        if ok is not None:
            c *= ok
            d *= ok
        if value is None:
            vis[k0:k1] = torch.complex(c @ b, -(d @ b))
        else:
            x = value(k0, k1)
            vis[k0:k1] = torch.complex((c * x).sum(1), -(d * x).sum(1))
        if norm is None:
            continue
        if seen:
            ok = seen(k0, k1)
            c *= ok
            d *= ok
        g = (vis[k0:k1].to(torch.complex64).to(torch.complex128) if y is None else y[k0:k1]) * (1.0 if weight is None else weight[k0:k1].double())
        F += torch.complex(g.real @ c - g.imag @ d, g.real @ d + g.imag @ c) * norm
    return vis, F


def exact(case, seed):
    kind = case["kind"]
    if kind in ("tables",):
        return None  # the reference's float arithmetic: whole rows, compared as they are
    w = work(case)
    if kind != "continuous" and w["flops"] > 24 * MOST_TERMS:
        return None
    s = prepare(case, seed)
    if kind == "imaging":
        K = s["uvw"][0].numel()
        return _both_ways(s, s["bright"], None, 1.0, -1.0, 1.0 / K, visible=lambda a, b: _visible(s["geo"], s["lmn"], a, b))
    if kind == "fit_step":
        vis, F = _both_ways(s, s["bright"], None, 1.0, -1.0, 1.0, visible=lambda a, b: _visible(s["geo"], s["lmn"], a, b),
                            y=torch.view_as_complex(s["g"]).to(torch.complex128))
        return vis, F.real
    if kind == "channels":
        out, F = [], []
        for c in range(len(s["off"]) - 1):
            a, b = s["off"][c], s["off"][c + 1]
            ch = dict(uvw=tuple(x[a:b] for x in s["uvw"]), lmn=s["lmn"])
            geo = dict(snap=s["geo"]["snap"][a:b], pair=s["geo"]["pair"][a:b], sat_pos=s["geo"]["sat_pos"])
            vis, f = _both_ways(ch, s["bright"][c], None, 1.0, -1.0, 1.0 / (b - a), visible=lambda i, j: _visible(geo, s["lmn"], i, j))
            out.append(vis)
            F.append(f)
        return torch.cat(out), torch.stack(F)
    if kind == "unmasked":
        return _both_ways(s, s["bright"], s["wgt"], 1.0, -1.0, 1.0 / case["rows"])
    if kind == "reference":
        K, res = case["rows"], s["res"]
        J = res * res
        q, r = torch.arange(J, device=DEV) // res, torch.arange(J, device=DEV) % res
        b = s["bright"].double()

        def value(a, e):
            M = s["shade"][a:e]
            hit = (M[:, 2:3] <= 0) & (q <= M[:, 3:4]) & (r > M[:, 0:1]) & (r < M[:, 1:2])
            return torch.where(hit, 240.0, b)

        def seen(a, e):
            r1, r2 = s["ratios"][0][a:e, None], s["ratios"][1][a:e, None]
            return ~(((r1 - r.float()).abs() < r1) & ((r2 - q.float()).abs() < r2))

        return _both_ways(s, None, s["wgt"], 0.5, 0.0, 1.0 / K, value=value, seen=seen)
    if kind == "fine_map":
        res, J = s["res"], s["J"]
        X = res * res
        q, r = torch.arange(X, device=DEV) // res, torch.arange(X, device=DEV) % res
        count = torch.bincount(s["coarse"], minlength=J)
        order = torch.sort(s["coarse"], stable=True).indices
        ff = s["FF"].double()
        base = torch.zeros(J, dtype=torch.float64, device=DEV).index_add_(0, s["coarse"], ff)

        def value(a, e):
            M = s["shade"][a:e]
            out = base.repeat(e - a, 1)
            for i in range(0, e - a, 512):
                m = M[i:i + 512]
                hit = (m[:, 2:3] <= 0) & (q <= m[:, 3:4]) & (r > m[:, 0:1]) & (r < m[:, 1:2])
                k, x = torch.nonzero(hit, as_tuple=True)
                out.view(-1).index_add_(0, (k + i) * J + s["coarse"][x], 240.0 - ff[x])
            return out / count

        vis, _ = _both_ways(s, None, None, 0.5, 0.0, None, value=value)
        return count.int(), order.int(), vis
    return _continuous(case, s)


def _continuous(case, s):
    """FP64 orbits as the continuous configurations define them (windows of a third of an orbit, each 10 degrees later)."""
    o = s["orbit"]
    res, total, span = o.orbit_res, o.orbit_res * o.orbit_counts, o.orbit_res // 3
    interval = res // 360 * 10
    S = o.orbit_counts * span
    g = torch.arange(S, device=DEV)
    k0 = g // span
    start = k0 * res + k0 * interval
    wrap = k0 * (res + interval) > total
    start = torch.where(wrap, start - (total // (res + interval) + 1) * res, start)
    i = start + g % span
    zero = (start + span > total) & (i >= total)
    half = total // 2
    r1 = torch.tensor(o.r1_m, dtype=torch.float32, device=DEV).double()
    r2 = torch.tensor(o.r2_m, dtype=torch.float32, device=DEV).double()
    x = i.double()[:, None]
    d = torch.where(x < half, r1 + (r2 - r1) / (half - 1) * x, r2 + (r1 - r2) / (half - 1) * (x - half))
    k, po = i // res, (i % res).double()[:, None]
    step = math.radians(o.raan_step_deg)
    raan = (k.double() * step + (o.index - 1) * o.orbit_counts * step)[:, None]
    w = 2 * math.pi / (res - 1) * po + 2.0 * torch.asin(d / (2.0 * o.a_km * 1e3))
    w = w + math.radians(o.argp_deg)
    ci, si = math.cos(math.radians(o.incl_deg)), math.sin(math.radians(o.incl_deg))
    cw, sw, cr, sr = torch.cos(w), torch.sin(w), torch.cos(raan), torch.sin(raan)
    pos = o.a_km * torch.stack([cw * cr - sw * ci * sr, cw * sr + sw * ci * cr, sw * si], -1)
    pos[zero] = 0.0
    uvw, snap, pair = _rows(pos, 300.0 / s["lam"])
    return (pos, pos) + tuple(uvw[:, c] for c in range(3)) + (snap, pair)
