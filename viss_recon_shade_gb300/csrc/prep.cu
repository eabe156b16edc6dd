// prep.cu -- per-pass preparation kernels: fixed-point pixel and visibility
// records, satellite directions and occlusion cones.  All O(J + K + S*nsat);
// the O(K*J) work is in vis_dft.cu and recon.cu.
#include <cfloat>

#include "viss_internal.cuh"

namespace viss {

// ------------------------------------------------------------- pixels
// Pixel j: phase coordinates x = s*l, y = s*m, z = s*(n + n_offset) in turns per
// wavelength, evaluated in double from the float inputs.
// Records are written at position `pos`; with a permutation the pixel at pos
// is perm[pos] (records keep the original index in rec1.w / geo.w).
__device__ __forceinline__ float4 prep_pixel(const PixPrepArgs& a, int64_t pos) {
  if (pos >= a.J) {
    a.rec0[pos] = make_int4(0, 0, 0, 0);
    if (a.rec1) a.rec1[pos] = make_int4(0, 0, 0, (int)pos);
    if (a.lo) a.lo[pos] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.geo) a.geo[pos] = make_float4(0.f, 0.f, 0.f, __int_as_float((int)pos));
    if (a.qr) a.qr[pos] = make_int2(-1, -1);
    return make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const int64_t j = a.perm ? (int64_t)a.perm[pos] : pos;
  float b = 0.f;
  if (a.bright) {
    b = a.bright[j];
    if (a.trunc) b = (float)(int)b;  // int addFF = FF[..] (vissGen10M_shade.cu:128)
  }
  const float lj = a.l[j], mj = a.m[j], nj = a.n[j];
  uint32_t A, B, C;
  float4 rec1, lo = make_float4(0.f, 0.f, 0.f, 0.f);
  if (a.pow2) {
    // s is a power of two and s * n_offset * 2^32 an integer (s = 1 or 1/2, n_offset = -1 or 0):
    // the products are exact in FP32 and the offset adds whole units after the rounding, so these are
    // the double path's records without its ~15 FP64 operations a pixel
    const float s32 = (float)(a.sl * 4294967296.0), s1 = (float)a.sl;
    const float xa = lj * s32, ya = mj * s32, za = nj * s32;
    A = (uint32_t)(unsigned long long)__float2ll_rn(xa);
    B = (uint32_t)(unsigned long long)__float2ll_rn(ya);
    C = (uint32_t)(unsigned long long)__float2ll_rn(za) + (uint32_t)(unsigned long long)a.off32;
    rec1 = make_float4(lj * s1, mj * s1, nj * s1, __int_as_float((int)j));
    if (a.lo)
      lo = make_float4((xa - rintf(xa)) * 0x1p-32f, (ya - rintf(ya)) * 0x1p-32f, (za - rintf(za)) * 0x1p-32f, 0.f);
  } else {
    const double x = a.sl * (double)lj;
    const double y = a.sm * (double)mj;
    const double z = a.sn * ((double)nj + a.n_offset);
    A = fix32(x);
    B = fix32(y);
    C = fix32(z);
    // coordinates for the fractional part of uvw; z without the n_offset shift (|s*n| <= 1)
    rec1 = make_float4((float)x, (float)y, (float)(a.sn * (double)nj), __int_as_float((int)j));
    if (a.lo) {
      const double sc = 4294967296.0;
      const double xa = x * sc, ya = y * sc, za = z * sc;
      lo = make_float4((float)((xa - rint(xa)) / sc), (float)((ya - rint(ya)) / sc), (float)((za - rint(za)) / sc), 0.f);
    }
  }
  a.rec0[pos] = make_int4((int)A, (int)B, (int)C, __float_as_int(b));
  if (a.rec1) reinterpret_cast<float4*>(a.rec1)[pos] = rec1;
  if (a.lo) a.lo[pos] = lo;
  float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
  if (a.geo) {
    // unit direction, scaled by the largest coordinate first (good to 2e-7, against the 2e-6 of
    // the limb within which the test is re-decided from the inputs)
    const float big = fmaxf(fabsf(lj), fmaxf(fabsf(mj), fabsf(nj)));
    const float gx = lj / big, gy = mj / big, gz = nj / big;
    const float inv = big > 0.f ? 1.0f / sqrtf(fmaf(gx, gx, fmaf(gy, gy, gz * gz))) : 0.f;
    g = big > 0.f ? make_float4(gx * inv, gy * inv, gz * inv, 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
    g.w = __int_as_float((int)j);
    a.geo[pos] = g;
  }
  if (a.qr) {
    const int res = a.res > 0 ? a.res : 1;
    const int64_t i = a.widx ? (int64_t)a.widx[j] : j;
    int64_t q = i / res, r = i - q * res;
    if (r < 0) { r += res; --q; }  // floor division for negative indices
    a.qr[pos] = make_int2((int)q, (int)r);
  }
  return g;
}

constexpr int PREP_THREADS = 256;  // every part of prep_kernel
static_assert(PREP_THREADS == REC_THREADS, "the caps' blocks are the recon's");

__device__ __forceinline__ float warp_sum(float x) {
  for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
__device__ __forceinline__ float warp_max(float x) {
  for (int o = 16; o; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
__device__ __forceinline__ float warp_min(float x) {
  for (int o = 16; o; o >>= 1) x = fminf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
__device__ __forceinline__ float chord2(const float4& a, const float4& g) {  // |a - g|^2
  const float dx = g.x - a.x, dy = g.y - a.y, dz = g.z - a.z;
  return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

// Bounding cap of unit vectors: their normalised sum as axis, and the angle r of their largest
// distance c from it, c = 2 sin(r / 2) (a chord keeps its relative accuracy in FP32 where a
// cosine near 1 does not), widened by 2e-6 against the rounding of both.  {axis, cos r},
// {sin r}; cos r = -2 without an axis.
__device__ __forceinline__ float4 cap_axis(float sx, float sy, float sz) {
  const float nn = sqrtf(fmaf(sx, sx, fmaf(sy, sy, sz * sz)));
  return nn > 1e-3f ? make_float4(sx / nn, sy / nn, sz / nn, 1.f) : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ void cap_write(const float4& axis, float c2, float4* out) {
  float cr = -2.f, sr = 1.f;
  if (axis.w != 0.f && c2 < 3.999f) {
    const float r = 2.f * asinf(0.5f * sqrtf(c2)) + 2e-6f;
    cr = cosf(r);
    sr = sinf(r);
  }
  out[0] = make_float4(axis.x, axis.y, axis.z, cr);
  out[1] = make_float4(sr, 0.f, 0.f, 0.f);
}

// The records and, on the way, the cap of each warp's patch of 32 * REC_TJ positions: one launch and
// no second read of the directions (cap kernels with FP64 cosines and arc cosines took 22 us
// beside 5 us of records on 2,048-12,288 pixels).
__device__ void prep_pixels_caps(const PixPrepArgs& a, int block, float4* wcaps) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t p0 = (int64_t)block * REC_PIX + warp * 32 * REC_TJ + lane;
  float4 g[REC_TJ];
  float sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll
  for (int i = 0; i < REC_TJ; ++i) {
    g[i] = prep_pixel(a, p0 + 32 * i);  // zero past the last pixel
    sx += g[i].x; sy += g[i].y; sz += g[i].z;
  }
  sx = warp_sum(sx); sy = warp_sum(sy); sz = warp_sum(sz);
  const float4 wa = cap_axis(sx, sy, sz);
  float c2 = 0.f;
#pragma unroll
  for (int i = 0; i < REC_TJ; ++i) {
    // no direction (0, 0, 0), which no satellite hides: a cap of 90 degrees, which no snapshot hides
    // as a whole (half angles of shadows are below that).  Its chord, 1, would pass for 60 degrees.
    const bool none = g[i].x == 0.f && g[i].y == 0.f && g[i].z == 0.f;
    if (p0 + 32 * i < a.J) c2 = fmaxf(c2, none ? 2.f : chord2(wa, g[i]));
  }
  c2 = warp_max(c2);
  if (lane == 0) cap_write(wa, c2, wcaps + 2 * ((int64_t)block * (REC_THREADS / 32) + warp));
}

// {min, max} of widx over each run of VIS_P positions (the fine indices a vis
// tile's REF windows test), {1, 0} for a run past J
__global__ void ref_ranges_kernel(const int32_t* widx, int64_t J, int64_t ntiles, int2* rng) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntiles) return;
  int lo = 0x7fffffff, hi = -0x7fffffff - 1;
  for (int64_t j = t * VIS_P; j < (t + 1) * VIS_P && j < J; ++j) {
    lo = min(lo, widx[j]);
    hi = max(hi, widx[j]);
  }
  rng[t] = lo <= hi ? make_int2(lo, hi) : make_int2(1, 0);
}

int launch_prep_ref_ranges(const int32_t* widx, int64_t J, int64_t ntiles, int2* rng, cudaStream_t st) {
  if (ntiles <= 0) return VISS_OK;
  ref_ranges_kernel<<<(unsigned)((ntiles + 127) / 128), 128, 0, st>>>(widx, J, ntiles, rng);
  VISS_LAUNCH_CHECK("ref_ranges_kernel");
  return VISS_OK;
}

// ------------------------------------------------------------- rows
// Reference recon mask (vissGen10M_shade.cu:166): skip iff
//   fabsf(r1 - thetaP) < r1 && fabsf(r2 - phiP) < r2,  r = (float)Ma / (float)Mb
// with thetaP, phiP non-negative integers.  The set of integers t passing the
// first test is {1..tmax} (empty when r1 <= 0 or NaN); tmax is found from the
// exact float predicate.
__device__ int recon_ratio_tmax(float r) {
  if (!(r > 0.f) || isinf(r)) return 0;
  // candidates t < 2r; find the largest t >= 1 with fabsf(r - t) < r
  double lim = 2.0 * (double)r;
  long long t = (long long)ceil(lim) - 1;
  if (t > 2147483000LL) t = 2147483000LL;
  for (long long c = t + 1; c >= t - 1 && c >= 1; --c) {
    if (fabsf(r - (float)c) < r) return (int)c;
  }
  return 0;
}

// Input row of padded row pr, or -1 for a padding row.
__device__ __forceinline__ int64_t padded_row_source(const ChannelRows& ch, int64_t pr) {
  const int64_t b = pr / VIS_ROWS;
  int lo = 0, hi = ch.nch - 1;  // channel c with rb_off[c] <= b < rb_off[c+1]
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (ch.rb_off[mid] <= b) lo = mid;
    else hi = mid - 1;
  }
  const int64_t k = ch.row_off[lo] + (pr - ch.rb_off[lo] * VIS_ROWS);
  return k < ch.row_off[lo + 1] ? k : -1;
}

__device__ __forceinline__ void prep_row(const RowPrepArgs& a, bool recon, int64_t pr) {
  const int64_t k = a.padded ? padded_row_source(a.ch, pr) : (pr < a.K ? pr : -1);
  if (k < 0) {
    a.rows0[pr] = make_int4(0, 0, 0, PHASE_BIAS);
    a.rows1[pr] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.rowsat) a.rowsat[pr] = PAD_PACKED;
    if (a.rowpm) a.rowpm[pr] = make_int2(0, 1);
    if (a.uf) a.uf[pr] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.win) a.win[pr] = recon ? make_int4(0, 0, 0, 0) : make_int4(1, 0, 0, 0);
    return;
  }
  // u = U + f, U the nearest integer, |f| <= 1/2: exact in FP32 (f has no bit below u's last)
  const float u3[3] = {a.u[k], a.v[k], a.w[k]};
  float U3[3], f3[3];
  bool ok = true, frac = false;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    U3[c] = rintf(u3[c]);
    f3[c] = u3[c] - U3[c];
    ok &= fabsf(U3[c]) < 1073741824.f;  // |U| < 2^30; false for NaN
    frac |= f3[c] != 0.f;
  }
  if (!ok) atomicOr(a.flags + FLAG_ERR, 1);
  if (frac) atomicOr(a.flags + FLAG_FRAC, 1);
  if (a.snap) {
    int packed = PAD_PACKED;
    int2 sp = make_int2(0, 1);
    const int s = a.snap[k];
    const int pr2 = a.pair[k];
    const int pm = pr2 & 0xffff, pn = (pr2 >> 16) & 0xffff;
    if (s < 0 || s >= a.S || pm >= a.nsat || pn >= a.nsat) atomicOr(a.flags + FLAG_ERR, 2);
    else {
      packed = (s * a.nsat + pm) | ((pn - pm + 32) << 26);
      sp = make_int2(s, (1 << pm) | (1 << pn));
    }
    if (a.rowsat) a.rowsat[pr] = packed;
    if (a.rowpm) a.rowpm[pr] = sp;
  }
  // PHASE_BIAS plus the per-row part of f_w * z: f_w * sn * n_offset; the
  // reconstruction folds the visibility's phase in too: y e^{ix} = |y| e^{i(x + arg y)}
  uint32_t bias = (uint32_t)PHASE_BIAS + (a.n_offset != 0.0 ? fix32((double)f3[2] * a.sn * a.n_offset) : 0u);
  float c = 0.f;
  if (recon) {
    const double wg = a.wgt ? (double)a.wgt[k] : 1.0;
    const double yr = wg * (double)a.V[2 * k], yi = wg * (double)a.V[2 * k + 1];
    c = (float)sqrt(yr * yr + yi * yi);
    if (c > 0.f) bias += fix32(atan2(yi, yr) * (0.5 / kPi));
    // every other row: half a turn more and -|y| (the same term), so that a
    // systematic error of the SFU's sin/cos cancels over the rows instead of
    // adding up with the all-positive weights |y|
    if (k & 1) {
      bias += 0x80000000u;
      c = -c;
    }
  }
  a.rows0[pr] = make_int4((int)(long long)U3[0], (int)(long long)U3[1], (int)(long long)U3[2], (int)bias);
  // the FP32 parts of the phase are summed in radians: coefficients times 2 pi
  a.rows1[pr] = make_float4(f3[0] * K2PI, f3[1] * K2PI, f3[2] * K2PI, c);
  if (a.uf) a.uf[pr] = make_float4(U3[0] * K2PI, U3[1] * K2PI, U3[2] * K2PI, 0.f);
  if (a.win) {
    int4 wv = recon ? make_int4(0, 0, 0, 0) : make_int4(1, 0, 0, 0);  // empty
    if (a.shade || a.shade_cols[0]) {
      const int M1 = a.shade ? a.shade[4 * k] : a.shade_cols[0][k], M2 = a.shade ? a.shade[4 * k + 1] : a.shade_cols[1][k],
                M3 = a.shade ? a.shade[4 * k + 2] : a.shade_cols[2][k],
                M4 = a.shade ? a.shade[4 * k + 3] : a.shade_cols[3][k];
      if (!recon) {
        if (a.mask_mode == VISS_MASK_REF_QUIRK) {
          if (M3 <= 0 && M4 >= 0) wv = make_int4(0, M4, M1, M2);
        } else if (a.mask_mode == VISS_MASK_REF_INTENDED) {
          if (M3 <= M4) wv = make_int4(M3, M4, M1, M2);
        }
      } else if (a.recon_mask == VISS_RECON_MASK_REF) {
        const float r1 = (float)M1 / (float)M2, r2 = (float)M3 / (float)M4;
        wv = make_int4(recon_ratio_tmax(r1), recon_ratio_tmax(r2), 0, 0);
      }
    } else if (a.ratios[0]) {
      // viss_imagerecon gives the ratios themselves.  Skip iff fabsf(t0 - thetaP) < dt &&
      // fabsf(p0 - phiP) < dp; the reference passes the same ratio array twice (t0 == dt,
      // p0 == dp, :514-517); rows of another form set flag bit 4 and the call is rejected.
      const float t0 = a.ratios[0][k], p0 = a.ratios[1][k], dt = a.ratios[2][k], dp = a.ratios[3][k];
      const bool same_t = (t0 == dt) || (t0 != t0 && dt != dt);
      const bool same_p = (p0 == dp) || (p0 != p0 && dp != dp);
      if (!same_t || !same_p) atomicOr(a.flags + FLAG_ERR, 4);
      wv = make_int4(recon_ratio_tmax(t0), recon_ratio_tmax(p0), 0, 0);
    }
    a.win[pr] = wv;
  }
}

// ------------------------------------------------------------- satellites
// satdir[i] = {p/|p|, cos(alpha)}, alpha = asin(R/|p|) the Moon's angular radius
// seen from the satellite.  Occluded <=> s_hat . p_hat < -cos(alpha).  A
// satellite inside the sphere (|p| <= R) gets cos(alpha) = 0 (occluded <=> s.p < 0),
// which is what the exact predicate gives there.
__device__ __forceinline__ float4 sat_direction(const float* pos, double R) {
  const double px = pos[0], py = pos[1], pz = pos[2];
  const double rr = px * px + py * py + pz * pz;
  if (!(rr > 0.0)) return make_float4(0.f, 0.f, 0.f, 0.f);
  const double inv = rsqrt(rr), q = R * inv;
  const float ca = rr > R * R ? sqrtf((float)(1.0 - q * q)) : 0.f;
  return make_float4((float)(px * inv), (float)(py * inv), (float)(pz * inv), ca);
}

// ------------------------------------------------------------- cones
// For a set of satellites {p_i} with shadow cones (axis -p_hat_i, half angle
// alpha_i): axis c = normalise(sum -p_hat_i), rho = max angle(c, -p_hat_i).
// A pixel s_hat with s_hat.c > cos(alpha_min - rho - eps) is occluded for every
// satellite of the set; with s_hat.c < cos(alpha_max + rho + eps) it is visible
// from every one.  cone[0] = {c, cos_occ}, cone[1] = {cos_vis, sin_occ, sin_vis, -}
// (the sines of the two angles, 0 where the cosine is the 2 / -2 of "never").
// Degenerate sets (a satellite at the origin) get cos_occ = 2, cos_vis = -2.
// In FP32: rho from the largest chord, good to 3e-7 rad, which the margins (1.2e-5 rad, 1.5e-6 in the
// cosine tested against) cover many times over; alpha from the extreme cosines, which are good to
// 6e-8 only and leave alpha itself uncertain by 6e-8 / sin(alpha) (6e-5 rad for a satellite a thousand
// radii away), so they are widened by that first.
constexpr float COS_ERR = 1.2e-7f;
__device__ void cone_write(const float4& axis, float c2, float wmin, float wmax, bool degen, float4* out) {
  const float eps = 1.2e-5f;
  float cos_occ = 2.f, cos_vis = -2.f, sin_occ = 0.f, sin_vis = 0.f;
  if (!degen) {
    const float rho = 2.f * asinf(fminf(1.f, 0.5f * sqrtf(c2)));
    const float lo = acosf(fminf(1.f, wmax + COS_ERR)) - rho - eps, hi = acosf(wmin - COS_ERR) + rho + eps;
    if (lo > 0.f) { cos_occ = cosf(lo) + 1.5e-6f; sin_occ = sinf(lo); }
    if (hi < 3.1415926f) { cos_vis = cosf(hi) - 1.5e-6f; sin_vis = sinf(hi); }
  }
  out[0] = make_float4(axis.x, axis.y, axis.z, cos_occ);
  out[1] = make_float4(cos_vis, sin_occ, sin_vis, 0.f);
}
// axis of a cone from the sum of -p_hat; no axis makes the set degenerate
__device__ __forceinline__ float4 cone_axis(float sx, float sy, float sz, bool* degen) {
  const float nn = sqrtf(fmaf(sx, sx, fmaf(sy, sy, sz * sz)));
  if (!(nn > 1e-6f)) {
    *degen = true;
    return make_float4(0.f, 0.f, 1.f, 0.f);
  }
  return make_float4(sx / nn, sy / nn, sz / nn, 0.f);
}
__device__ __forceinline__ float4 minus(const float4& d) { return make_float4(-d.x, -d.y, -d.z, d.w); }
// at the origin (no direction) or inside the sphere: no cone
__device__ __forceinline__ bool no_cone(const float4& d) { return d.w == 0.f; }

// Satellite directions and (cones != NULL) each snapshot's cone: a thread per satellite, G
// lanes (a power of two >= nsat) per snapshot, so that a pass of a hundred snapshots is a few
// short chains (one thread per snapshot with FP64 arc cosines took 20 us, the directions 5.5).
__device__ __forceinline__ void prep_satellite(const SatPrepArgs& a, int64_t t) {
  const int nsat = a.nsat, G = a.G;
  const int64_t S = a.S;
  float4* const satdir = a.satdir;
  float4* const cones = a.cones;
  const int64_t s = t / G;
  const int i = (int)(t & (G - 1));
  const bool live = s < S && i < nsat;
  float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
  if (live) {
    d = sat_direction(a.pos + 3 * (s * nsat + i), a.R);
    satdir[s * nsat + i] = d;
  }
  if (!cones) return;
  float sx = -d.x, sy = -d.y, sz = -d.z;
  float wmin = live ? d.w : 2.f, wmax = live ? d.w : -2.f;
  int dg = live && no_cone(d);
  for (int o = G >> 1; o; o >>= 1) {
    sx += __shfl_xor_sync(0xffffffffu, sx, o);
    sy += __shfl_xor_sync(0xffffffffu, sy, o);
    sz += __shfl_xor_sync(0xffffffffu, sz, o);
    wmin = fminf(wmin, __shfl_xor_sync(0xffffffffu, wmin, o));
    wmax = fmaxf(wmax, __shfl_xor_sync(0xffffffffu, wmax, o));
    dg |= __shfl_xor_sync(0xffffffffu, dg, o);
  }
  bool degen = dg != 0;
  const float4 axis = cone_axis(sx, sy, sz, &degen);
  float c2 = live ? chord2(axis, minus(d)) : 0.f;
  for (int o = G >> 1; o; o >>= 1) c2 = fmaxf(c2, __shfl_xor_sync(0xffffffffu, c2, o));
  if (s < S && i == 0) cone_write(axis, c2, wmin, wmax, degen, cones + 2 * s);
}

// The records of a pass in one launch: blocks of pixels, then of rows, then of satellites
// (they do not depend on each other, and for a small pass each is a launch's latency
// and little else: 3,360 x 2,048, vis and recon: 25 us in six launches, 10.5 in two).
template <bool CAPS>
__global__ void __launch_bounds__(PREP_THREADS) prep_kernel(const PixPrepArgs pix, const RowPrepArgs row, const SatPrepArgs sat,
                                                            int pix_blocks, int row_blocks, bool recon) {
  int b = (int)blockIdx.x;
  if (b < pix_blocks) {
    if (CAPS) prep_pixels_caps(pix, b, pix.wcaps);
    else {
      const int64_t pos = (int64_t)b * PREP_THREADS + threadIdx.x;
      if (pos < pix.Jpad) prep_pixel(pix, pos);
    }
    return;
  }
  b -= pix_blocks;
  if (b < row_blocks) {
    const int64_t pr = (int64_t)b * PREP_THREADS + threadIdx.x;
    if (pr < row.Kpad) prep_row(row, recon, pr);
    return;
  }
  prep_satellite(sat, (int64_t)(b - row_blocks) * PREP_THREADS + threadIdx.x);
}

static int64_t prep_blocks(int64_t n) { return (n + PREP_THREADS - 1) / PREP_THREADS; }

int launch_prep(const PixPrepArgs& pix, const RowPrepArgs& row, SatPrepArgs sat, bool recon, cudaStream_t st) {
  const bool caps = pix.wcaps != nullptr;
  const int64_t np = caps ? pix.Jpad / REC_PIX : prep_blocks(pix.Jpad), nr = prep_blocks(row.Kpad);
  int64_t ns = 0;
  if (sat.S > 0 && sat.nsat > 0) {
    for (sat.G = 1; sat.G < sat.nsat;) sat.G <<= 1;
    ns = prep_blocks(sat.S * sat.G);
  }
  const int64_t blocks = np + nr + ns;
  if (blocks <= 0) return VISS_OK;
  if (caps) prep_kernel<true><<<(unsigned)blocks, PREP_THREADS, 0, st>>>(pix, row, sat, (int)np, (int)nr, recon);
  else prep_kernel<false><<<(unsigned)blocks, PREP_THREADS, 0, st>>>(pix, row, sat, (int)np, (int)nr, recon);
  VISS_LAUNCH_CHECK("prep_kernel");
  return VISS_OK;
}

// One cone per padded block of VIS_ROWS rows, over the block's real rows; the
// sines in cone[1] (which the vis kernel does not use) are replaced by the range
// of satellite indices those rows use (y: the first, z: how many, as int bits;
// z = 0 for an empty block).  (With FP64 cosines and an FP64 arc cosine per satellite: 37 us
// however few the blocks, 320 us for 1,792.)
constexpr int CONE_THREADS = 256;
__global__ void __launch_bounds__(CONE_THREADS) rowblock_cones_kernel(const int* rowsat, const float4* satdir,
                                                                      const ChannelRows ch, float4* cones) {
  constexpr int NW = CONE_THREADS / 32, PER = VIS_ROWS / CONE_THREADS;
  __shared__ float red[NW][6];
  __shared__ int redi[NW][3];
  const int64_t b = blockIdx.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int c = 0;
  while (c + 1 < ch.nch && b >= ch.rb_off[c + 1]) ++c;
  int64_t cnt = (ch.row_off[c + 1] - ch.row_off[c]) - (b - ch.rb_off[c]) * VIS_ROWS;
  if (cnt > VIS_ROWS) cnt = VIS_ROWS;
  if (cnt < 0) cnt = 0;
  int pk[PER];
  float sx = 0.f, sy = 0.f, sz = 0.f, wmin = 2.f, wmax = -2.f;
  int lo = 0x7fffffff, hi = -1, dg = 0;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int r = threadIdx.x + i * CONE_THREADS;
    pk[i] = r < cnt ? rowsat[b * VIS_ROWS + r] : -1;
    if (pk[i] == -1) continue;
    const int gm = sat_gm(pk[i]), gn = sat_gn(pk[i]);
    const float4 d1 = satdir[gm], d2 = satdir[gn];
    sx -= d1.x + d2.x; sy -= d1.y + d2.y; sz -= d1.z + d2.z;
    wmin = fminf(wmin, fminf(d1.w, d2.w));
    wmax = fmaxf(wmax, fmaxf(d1.w, d2.w));
    dg |= no_cone(d1) || no_cone(d2);
    lo = min(lo, min(gm, gn));
    hi = max(hi, max(gm, gn));
  }
  sx = warp_sum(sx); sy = warp_sum(sy); sz = warp_sum(sz);
  wmin = warp_min(wmin);
  wmax = warp_max(wmax);
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  dg = __any_sync(0xffffffffu, dg);
  if (lane == 0) {
    red[wid][0] = sx; red[wid][1] = sy; red[wid][2] = sz; red[wid][3] = wmin; red[wid][4] = wmax;
    redi[wid][0] = lo; redi[wid][1] = hi; redi[wid][2] = dg;
  }
  __syncthreads();
  sx = sy = sz = 0.f;
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    sx += red[w][0]; sy += red[w][1]; sz += red[w][2];
    wmin = fminf(wmin, red[w][3]);
    wmax = fmaxf(wmax, red[w][4]);
    lo = min(lo, redi[w][0]);
    hi = max(hi, redi[w][1]);
    dg |= redi[w][2];
  }
  bool degen = dg != 0 || cnt == 0;
  const float4 axis = cone_axis(sx, sy, sz, &degen);
  float c2 = 0.f;
#pragma unroll
  for (int i = 0; i < PER; ++i)
    if (pk[i] != -1)
      c2 = fmaxf(c2, fmaxf(chord2(axis, minus(satdir[sat_gm(pk[i])])), chord2(axis, minus(satdir[sat_gn(pk[i])]))));
  c2 = warp_max(c2);
  if (lane == 0) red[wid][5] = c2;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < NW; ++w) c2 = fmaxf(c2, red[w][5]);
    cone_write(axis, c2, wmin, wmax, degen, cones + 2 * b);
    cones[2 * b + 1].y = __int_as_float(hi >= lo ? lo : 0);
    cones[2 * b + 1].z = __int_as_float(hi >= lo ? hi - lo + 1 : 0);
  }
}

int launch_prep_rowblock_cones(const int* rowsat, const float4* satdir, const ChannelRows& ch, int64_t nblocks,
                               float4* cones, cudaStream_t st) {
  if (nblocks <= 0) return VISS_OK;
  rowblock_cones_kernel<<<(unsigned)nblocks, CONE_THREADS, 0, st>>>(rowsat, satdir, ch, cones);
  VISS_LAUNCH_CHECK("rowblock_cones_kernel");
  return VISS_OK;
}

}  // namespace viss
