// recon.cu -- direct-DFT reconstruction (replaces imagerecon, vissGen10M_shade.cu:149-175,
// and the tiled optim2 form, vissGen10M_shade_optim2.cu:219-317).
//
// F_j = norm * sum_k [not masked] y_k exp(+2 pi i t_kj),  y_k = wgt_k V_k
//
// A work item of the unmasked and REF kernels is REC_PIX = 1024 pixels (4 per thread,
// fixed-point coordinates in registers) against one segment of visibility rows of one
// channel, streamed through shared memory in tiles of 2 REC_Q rows (REC_Q or REC_Q / 2 on
// request); one of the geometric kernel is a warp's 128 pixels against such a segment.
// The phase of y_k is folded into the
// row's fixed-point bias (y e^{ix} = |y| e^{i(x + arg y)}), so a term is the
// same as in the vis kernel: 3 IMAD [+3 FFMA fractional uvw] [+3 FFMA
// compensated], turns -> angle, __sincosf, 2 FFMA with |y_k|.
// Masks:
//   GEOMETRIC: a lane tests its row's snapshot cones against the cap bounding the warp's
//     128 pixels: rows hidden from all of them are dropped, rows that all of them see run
//     unmasked.  For a snapshot that this leaves open, every thread tests its pixels
//     against the cones and the warp votes; if that leaves it open too, the thread builds a
//     per-pixel satellite occlusion bitmask and tests each row's pair.
//   REF: the reference ratio mask can only fire on pixels (thetaP, phiP) with
//     1 <= thetaP <= tmax_k, 1 <= phiP <= pmax_k; tiles whose rows cannot touch
//     the item's pixels run unmasked.
// Persistent CTAs (geometric: warps) take items from an atomic counter, longest segments first.
// A channel split into several segments leaves partial sums per segment,
// reduced in a fixed order.
#include <type_traits>

#include "terms.cuh"
#include "viss_internal.cuh"

namespace viss {

// Exact decision near the limb (rare), out of line.
__device__ __noinline__ bool geo_exact_pix(const ReconParams& p, int j, int gidx) {
  count_limb(p.flags);
  return geo_occluded_exact(p.l[j], p.m[j], p.n[j], p.sat_pos + 3 * (int64_t)gidx, p.R);
}

template <bool FRAC, bool COMP>
__device__ __forceinline__ void rec_term(const int4& r0, const float4& r1, const float4& rf, float c, int A, int B,
                                         int C, float X, float Y, float Z, float lx, float ly, float lz, float& fr,
                                         float& fi) {
  const uint32_t q = (uint32_t)r0.x * (uint32_t)A + (uint32_t)r0.y * (uint32_t)B + (uint32_t)r0.z * (uint32_t)C +
                     (uint32_t)r0.w;
  float e = KM3PI;
  if (FRAC) e = fmaf(r1.x, X, fmaf(r1.y, Y, fmaf(r1.z, Z, e)));
  if (COMP) e = fmaf(rf.x, lx, fmaf(rf.y, ly, fmaf(rf.z, lz, e)));
  const float x = turns_to_angle(q, e);
  float sn, cs;
  __sincosf(x, &sn, &cs);
  fr = fmaf(c, cs, fr);
  fi = fmaf(c, sn, fi);
}

constexpr int RM_NONE = VISS_RECON_MASK_NONE, RM_REF = VISS_RECON_MASK_REF;

template <int RM, bool COMP, int Q>
struct RecSmem {  // unmasked and REF
  int4 r0[Q];                    // {U, V, W, bias}
  ulonglong2 r1[Q];              // {fu, fu, fv, fv}
  ulonglong2 r2[Q];              // {fw, fw, c, c}
  float4 rf[COMP ? Q : 1];
  int4 win[RM == RM_REF ? Q : 1];
  float4 acc[REC_PIX];           // running totals (re, im) and their Kahan compensation per pixel
};

// F = norm * (-fr - i fi)  (the angle carried an extra half turn)
__device__ __forceinline__ void recon_store(const ReconParams& p, const float4* acc, int64_t j0, float2* out, float norm,
                                            bool direct) {
#pragma unroll
  for (int i = 0; i < REC_TJ; ++i) {
    const int64_t pos = j0 + i;
    const float4 t = acc[threadIdx.x * REC_TJ + i];
    const float fr = t.x, fi = t.y;
    if (pos < p.J) {
      if (direct) {
        const int64_t j = p.perm ? (int64_t)p.perm[pos] : pos;
        out[j] = make_float2(-fr * norm, -fi * norm);
      } else {
        out[pos] = make_float2(fr, fi);
      }
    }
  }
}

// Unmasked and REF-mask items.  Every FP32 operation of a term but the SFU's runs packed, two pixels
// at a time, and of integer uvw a quarter of the terms are polynomials: the FMA pipe has room
// beside the SFU there (10 of its 16 cycles a warp-term).  What it measured against single
// operations is at recon_fast_kernel.
template <int RM, bool FRAC, bool COMP, int Q>
__device__ __forceinline__ void recon_rows(const ReconParams& p, RecSmem<RM, COMP, Q>& sm, int64_t pb, int64_t kb,
                                           int64_t ke, float2* out, float norm, bool direct) {
  const int tid = threadIdx.x;
  const int64_t j0 = pb * REC_PIX + (int64_t)tid * REC_TJ;
  int A[REC_TJ], B[REC_TJ], C[REC_TJ];
  // pixels in packed pairs (pixel 2h in the low half, 2h + 1 in the high one)
  f32x2 XF[REC_TJ / 2], YF[REC_TJ / 2], ZF[REC_TJ / 2];
  f32x2 LX[REC_TJ / 2], LY[REC_TJ / 2], LZ[REC_TJ / 2];
  // running totals live in sm.acc
#pragma unroll
  for (int i = 0; i < REC_TJ; ++i) {
    const int64_t pos = j0 + i;  // pixels padded to a whole block
    const int4 a = p.pix0[pos];
    A[i] = a.x; B[i] = a.y; C[i] = a.z;
    sm.acc[tid * REC_TJ + i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int h = 0; h < REC_TJ / 2; ++h) {
    XF[h] = YF[h] = ZF[h] = LX[h] = LY[h] = LZ[h] = 0ull;
    if (FRAC) {
      const float4* px = reinterpret_cast<const float4*>(p.pix1) + j0 + 2 * h;
      const float4 a = px[0], b = px[1];
      XF[h] = pack2(a.x, b.x); YF[h] = pack2(a.y, b.y); ZF[h] = pack2(a.z, b.z);
    }
    if (COMP) {
      const float4 a = p.plo[j0 + 2 * h], b = p.plo[j0 + 2 * h + 1];
      LX[h] = pack2(a.x, b.x); LY[h] = pack2(a.y, b.y); LZ[h] = pack2(a.z, b.z);
    }
  }
  const int64_t jfirst = pb * REC_PIX;
  int64_t jlast = jfirst + REC_PIX - 1;
  if (jlast > p.J - 1) jlast = p.J - 1;

  for (int64_t tile = kb; tile < ke; tile += Q) {
    const int nq = (int)((ke - tile) < Q ? (ke - tile) : Q);
    __syncthreads();
    bool hit = false;
    for (int r = tid; r < nq; r += REC_THREADS) {
      const int64_t k = tile + r;
      const float4 r1 = p.rows1[k];
      sm.r0[r] = p.rows0[k];
      sm.r1[r] = make_ulonglong2(pack2(r1.x, r1.x), pack2(r1.y, r1.y));
      sm.r2[r] = make_ulonglong2(pack2(r1.z, r1.z), pack2(r1.w, r1.w));
      if (COMP) sm.rf[r] = p.rowsf[k];
      if (RM == RM_REF) {
        const int4 wv = p.win[k];
        sm.win[r] = wv;
        if (wv.x >= 1 && wv.y >= 1) {
          const int64_t lo_idx = (int64_t)p.res + 1, hi_idx = (int64_t)wv.y * p.res + wv.x;
          if (lo_idx <= jlast && hi_idx >= jfirst) hit = true;
        }
      }
    }
    const bool masked_tile = __syncthreads_or(hit) != 0;
    f32x2 tr[REC_TJ / 2], ti[REC_TJ / 2];  // this tile's sums
#pragma unroll
    for (int h = 0; h < REC_TJ / 2; ++h) tr[h] = ti[h] = 0ull;
    static_assert(REC_TJ == 4, "two pixel pairs");
    // row r with all of the thread's pixels; poly: the second pair without the SFU
    auto row_term = [&](int r, auto poly) {
      const int4 r0 = sm.r0[r];
      const ulonglong2 fuv = FRAC ? sm.r1[r] : make_ulonglong2(0ull, 0ull), fwc = sm.r2[r];
      const float4 rf = COMP ? sm.rf[r] : make_float4(0.f, 0.f, 0.f, 0.f);
      term2<FRAC, COMP, false>(r0, fuv, fwc.x, rf, fwc.y, A, B, C, r0.w, r0.w, XF[0], YF[0], ZF[0], LX[0], LY[0], LZ[0], tr[0],
                                   ti[0]);
      term2<FRAC, COMP, decltype(poly)::value>(r0, fuv, fwc.x, rf, fwc.y, A + 2, B + 2, C + 2, r0.w, r0.w, XF[1], YF[1], ZF[1],
                                                   LX[1], LY[1], LZ[1], tr[1], ti[1]);
    };
    if (RM == RM_REF && masked_tile) {
      // the pixels' fine coordinates are read again here: held, they cost the unmasked tiles 8 of 80
      // registers (262,144 x 196,249: integer 21.4 -> 20.9 ms, fractional 23.9 -> 23.2)
      int TP[REC_TJ], PP[REC_TJ];
#pragma unroll
      for (int i = 0; i < REC_TJ; ++i) { const int2 qr = __ldg(p.pqr + j0 + i); PP[i] = qr.x; TP[i] = qr.y; }
      for (int r = 0; r < nq; ++r) {
        const int4 r0 = sm.r0[r], wv = sm.win[r];
        const ulonglong2 fuv = FRAC ? sm.r1[r] : make_ulonglong2(0ull, 0ull), fwc = sm.r2[r];
        const float4 rf = COMP ? sm.rf[r] : make_float4(0.f, 0.f, 0.f, 0.f);
        float c, c_;
        unpack2(fwc.y, c, c_);
#pragma unroll
        for (int h = 0; h < REC_TJ / 2; ++h) {
          float cm[2];
#pragma unroll
          for (int o = 0; o < 2; ++o) {
            const int i = 2 * h + o;
            cm[o] = TP[i] >= 1 && TP[i] <= wv.x && PP[i] >= 1 && PP[i] <= wv.y ? 0.f : c;
          }
          term2<FRAC, COMP, false>(r0, fuv, fwc.x, rf, pack2(cm[0], cm[1]), A + 2 * h, B + 2 * h, C + 2 * h, r0.w, r0.w, XF[h],
                                       YF[h], ZF[h], LX[h], LY[h], LZ[h], tr[h], ti[h]);
        }
      }
    } else {
      int r = 0;
      if (!FRAC && !COMP) {
        // the polynomial in two adjacent rows of four: the records alternate the sign of |y| so that
        // the SFU's systematic error cancels over the rows, which needs both signs in each kind of term
        // (in every other row: |mean error| of those pixels 9e-9 against 1e-10 at 65,536 rows).
        // Rows with and without it in turn: 262,144 x 196,249 in row order 2 % slower.
        for (; r + 4 <= nq; r += 4) {
          row_term(r, std::false_type{});
          row_term(r + 2, std::true_type{});
          row_term(r + 1, std::false_type{});
          row_term(r + 3, std::true_type{});
        }
      }
#pragma unroll 2
      for (; r < nq; ++r) row_term(r, std::false_type{});
    }
#pragma unroll
    for (int h = 0; h < REC_TJ / 2; ++h) {
      float r[2], im[2];
      unpack2(tr[h], r[0], r[1]);
      unpack2(ti[h], im[0], im[1]);
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        float4 t = sm.acc[tid * REC_TJ + 2 * h + o];  // owned by this thread alone
        kahan_add(t.x, t.z, r[o]);
        kahan_add(t.y, t.w, im[o]);
        sm.acc[tid * REC_TJ + 2 * h + o] = t;
      }
    }
  }
  recon_store(p, sm.acc, j0, out, norm, direct);
}

// Geometric items: a warp's own patch of 32 * REC_TJ positions against one segment.  With the
// spatial order of the geometric passes a patch is one compact piece of sky, so most snapshots
// hide or show it as a whole.  Bound by the SFU (16 cycles a warp-term) and register reads
// (15) as the other kernels are, but what a pass computes differs from warp to warp: a block
// that shares its row tiles waits at their barriers for the warp that sees the most (a third of
// the stalls on 28,672 x 12,288).  So nothing is shared: a warp stages 32 rows at a time in its
// own corner of shared memory (64 or 128 at a time: 1.2 and 1 % slower on 10 MHz), and one
// snapshot's bits are kept there for as long as it stays open.  Rows of an open snapshot
// whose satellites hide the whole patch are skipped.  Against blocks with shared row tiles:
// 3,360 x 2,048 19.8 -> 16.6 us, 28,672 x 12,288 254 -> 210 us, 458,752 x 49,152 11.28 -> 10.47 ms,
// 1,835,008 x 196,608 157.2 -> 150.1 ms (rows as 64-bit indexes: 152.4, they spill).  Tried: the
// packed terms of the other kernels (10 MHz +3 %), halves of a patch skipped by themselves
// (+1 to 4 %).
struct GeoWarp {
  int4 r0[32];
  float4 r1[32];
  uint32_t pm[32];          // the row's two satellites as bits of its snapshot's satellites
  float4 sat[32];           // the open snapshot's satellite directions
  uint32_t bits[REC_TJ][32];  // per pixel: the open snapshot's satellites that it is hidden from
  float4 acc[32 * REC_TJ];  // running totals (re, im) and their Kahan compensation per pixel
};
template <bool COMP>
struct GeoSmem {
  GeoWarp w[REC_THREADS / 32];
  float4 rf[COMP ? REC_THREADS : 1];
};

template <bool FRAC, bool COMP>
__device__ __forceinline__ void recon_geo(const ReconParams& p, GeoWarp& sm, float4* rfs, unsigned patch, unsigned kb,
                                          unsigned ke, float2* out, float norm, bool direct) {
  const int lane = threadIdx.x & 31;
  // J <= 2^30 and K <= 2^31: 32-bit positions and rows; pixel i stands at j0 + 32 i
  const unsigned j0 = patch * (32 * REC_TJ) + lane, nj = (unsigned)p.J;
  int A[REC_TJ], B[REC_TJ], C[REC_TJ];
  float XF[REC_TJ], YF[REC_TJ], ZF[REC_TJ];
  float LX[REC_TJ], LY[REC_TJ], LZ[REC_TJ];
#pragma unroll
  for (int i = 0; i < REC_TJ; ++i) {
    const unsigned pos = j0 + 32 * i;  // pixels padded to a whole block
    const int4 a = p.pix0[pos];
    A[i] = a.x; B[i] = a.y; C[i] = a.z;
    XF[i] = YF[i] = ZF[i] = 0.f;
    if (FRAC) {
      const int4 b = p.pix1[pos];
      XF[i] = __int_as_float(b.x); YF[i] = __int_as_float(b.y); ZF[i] = __int_as_float(b.z);
    }
    LX[i] = LY[i] = LZ[i] = 0.f;
    if (COMP) { const float4 lo = p.plo[pos]; LX[i] = lo.x; LY[i] = lo.y; LZ[i] = lo.z; }
    sm.acc[32 * i + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  int open = -1;         // the snapshot whose bits are in sm.bits
  uint32_t hides = 0u;   // its satellites that hide the whole patch
  for (unsigned tile = kb; tile < ke; tile += REC_Q) {
    const unsigned te = min(tile + REC_Q, ke);
    float tr[REC_TJ], ti[REC_TJ];  // this tile's sums
#pragma unroll
    for (int i = 0; i < REC_TJ; ++i) tr[i] = ti[i] = 0.f;
    for (unsigned b = tile; b < te; b += 32) {
      // each lane decides its row's snapshot against the patch's cap {a, r}:
      // all hidden when angle(a, c) + r < alpha_occ, i.e. a.c > cos(alpha_occ - r);
      // all visible when angle(a, c) - r > alpha_vis, i.e. a.c < cos(alpha_vis + r)
      // (alpha_vis + r < pi).  Margins of 1e-5 in the cosine.
      bool hid = true, vis = false;
      int sn = -1;
      __syncwarp();  // the last batch's rows are consumed
      if (b + lane < te) {
        const int2 sp = p.rowpm[b + lane];
        sn = sp.x;
        const float4 wc = __ldg(p.wcones + 2 * patch);
        const float ws = __ldg(p.wcones + 2 * patch + 1).x;
        const float4 c0 = __ldg(p.scones + 2 * (unsigned)sn), c1 = __ldg(p.scones + 2 * (unsigned)sn + 1);
        const float dw = fmaf(wc.x, c0.x, fmaf(wc.y, c0.y, wc.z * c0.z));
        hid = false;
        if (wc.w >= -1.f) {
          hid = c0.w <= 1.f && c0.w < wc.w && dw > fmaf(c0.w, wc.w, c1.y * ws) + 1e-5f;
          vis = c1.x >= -1.f && fmaf(c1.z, wc.w, c1.x * ws) > 0.f && dw < fmaf(c1.x, wc.w, -c1.z * ws) - 1e-5f;
        }
        if (!hid) {
          sm.r0[lane] = p.rows0[b + lane];
          sm.r1[lane] = p.rows1[b + lane];
          if (COMP) rfs[lane] = p.rowsf[b + lane];
          sm.pm[lane] = (uint32_t)sp.y;
        }
      }
      unsigned todo = __ballot_sync(0xffffffffu, !hid);
      unsigned seen = __ballot_sync(0xffffffffu, vis);
      __syncwarp();
      while (todo) {
        const int r = __ffs(todo) - 1;
        if ((seen >> r) & 1u) {
          // a run of rows that see the whole patch
          const unsigned gap = ~((todo & seen) >> r);
          const int re = gap ? r + __ffs(gap) - 1 : 32;
          todo &= re < 32 ? 0xffffffffu << re : 0u;
#pragma unroll 2
          for (int rr = r; rr < re; ++rr) {
            const int4 r0 = sm.r0[rr];
            const float4 r1 = sm.r1[rr];
            float4 rf = make_float4(0.f, 0.f, 0.f, 0.f);
            if (COMP) rf = rfs[rr];
#pragma unroll
            for (int i = 0; i < REC_TJ; ++i)
              rec_term<FRAC, COMP>(r0, r1, rf, r1.w, A[i], B[i], C[i], XF[i], YF[i], ZF[i], LX[i], LY[i], LZ[i],
                                   tr[i], ti[i]);
          }
          continue;
        }
        // the batch's rows of one snapshot that the cap leaves open: the pixels vote
        const int s = __shfl_sync(0xffffffffu, sn, r);
        const unsigned same = __ballot_sync(0xffffffffu, sn == s) & todo;
        if (s != open) {
          open = s;
          const float4 c0 = __ldg(p.scones + 2 * (unsigned)s), c1 = __ldg(p.scones + 2 * (unsigned)s + 1);
          bool all_vis = true, all_occ = true;
#pragma unroll
          for (int i = 0; i < REC_TJ; ++i) {
            const float4 g = __ldg(p.pgeo + j0 + 32 * i);
            const float d = fmaf(g.x, c0.x, fmaf(g.y, c0.y, g.z * c0.z));
            const bool v = j0 + 32 * i < nj;
            all_vis &= !v || d < c1.x;
            all_occ &= !v || d > c0.w;
          }
          all_occ = __all_sync(0xffffffffu, all_occ);
          all_vis = __all_sync(0xffffffffu, all_vis);
          hides = all_occ ? 0xffffffffu : 0u;
          if (all_occ || all_vis) {
#pragma unroll
            for (int i = 0; i < REC_TJ; ++i) sm.bits[i][lane] = hides;
          } else {
            // per-pixel satellite occlusion bits for snapshot s
            if (lane < p.nsat) sm.sat[lane] = __ldg(p.satdir + s * p.nsat + lane);
            __syncwarp();
            hides = 0xffffffffu;
#pragma unroll 1
            for (int i = 0; i < REC_TJ; ++i) {
              const float4 g = __ldg(p.pgeo + j0 + 32 * i);
              const bool v = j0 + 32 * i < nj;
              uint32_t bits = 0u;
#pragma unroll 4
              for (int sat = 0; sat < p.nsat; ++sat) {
                const float4 d = sm.sat[sat];
                const float e = fmaf(g.x, d.x, fmaf(g.y, d.y, fmaf(g.z, d.z, d.w)));
                bool occ = e < 0.f;
                if (fabsf(e) < GEO_EPS && v) occ = geo_exact_pix(p, __float_as_int(g.w), s * p.nsat + sat);
                bits |= (occ ? 1u : 0u) << sat;
              }
              sm.bits[i][lane] = bits;
              if (v) hides &= bits;
            }
            __syncwarp();
            hides = __reduce_and_sync(0xffffffffu, hides);
          }
        }
        todo &= ~same;
        uint32_t bits[REC_TJ];
#pragma unroll
        for (int i = 0; i < REC_TJ; ++i) bits[i] = sm.bits[i][lane];
        // a row whose satellites hide the whole patch is skipped
        for (unsigned m = __ballot_sync(0xffffffffu, !(sm.pm[lane] & hides)) & same; m; m &= m - 1) {
          const int rr = __ffs(m) - 1;
          const int4 r0 = sm.r0[rr];
          const float4 r1 = sm.r1[rr];
          float4 rf = make_float4(0.f, 0.f, 0.f, 0.f);
          if (COMP) rf = rfs[rr];
          const uint32_t pm = sm.pm[rr];
#pragma unroll
          for (int i = 0; i < REC_TJ; ++i) {
            const float c = (bits[i] & pm) ? 0.f : r1.w;
            rec_term<FRAC, COMP>(r0, r1, rf, c, A[i], B[i], C[i], XF[i], YF[i], ZF[i], LX[i], LY[i], LZ[i],
                                 tr[i], ti[i]);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < REC_TJ; ++i) {
      float4 t = sm.acc[32 * i + lane];  // owned by this thread alone
      kahan_add(t.x, t.z, tr[i]);
      kahan_add(t.y, t.w, ti[i]);
      sm.acc[32 * i + lane] = t;
    }
  }
  // F = norm * (-fr - i fi)  (the angle carried an extra half turn)
#pragma unroll
  for (int i = 0; i < REC_TJ; ++i) {
    const unsigned pos = j0 + 32 * i;
    const float4 t = sm.acc[32 * i + lane];
    if (pos < nj) {
      if (direct) out[p.perm ? (unsigned)p.perm[pos] : pos] = make_float2(-t.x * norm, -t.y * norm);
      else out[pos] = make_float2(t.x, t.y);
    }
  }
}

template <bool COMP>
__global__ void __launch_bounds__(REC_THREADS, rec_ctas(VISS_RECON_MASK_GEOMETRIC, COMP)) recon_geo_kernel(const ReconParams p) {
  __shared__ GeoSmem<COMP> sm;
  const bool frac = __ldg(p.flags + FLAG_FRAC) != 0;
  const int warp = threadIdx.x >> 5;
  const unsigned npatch = (unsigned)((p.J + 32 * REC_TJ - 1) / (32 * REC_TJ));
  for (;;) {
    unsigned item = 0;  // up to VISS_MAX_SEG * 2^23
    if ((threadIdx.x & 31) == 0) item = (unsigned)atomicAdd(p.flags + FLAG_REC_COUNTER, 1);
    item = __shfl_sync(0xffffffffu, item, 0);
    const unsigned seg = item / npatch;
    if (seg >= (unsigned)p.nseg) break;
    const unsigned patch = item - seg * npatch;
    const int ch = p.seg_ch[seg], slot = p.seg_slot[seg];
    const bool direct = slot < 0;
    float2* out = direct ? p.out + (int64_t)ch * p.J : p.partial + (int64_t)slot * p.J;
    float4* rf = sm.rf + (COMP ? 32 * warp : 0);
    if (frac) recon_geo<true, COMP>(p, sm.w[warp], rf, patch, (unsigned)p.seg_lo[seg], (unsigned)p.seg_hi[seg], out, p.ch_norm[ch], direct);
    else recon_geo<false, COMP>(p, sm.w[warp], rf, patch, (unsigned)p.seg_lo[seg], (unsigned)p.seg_hi[seg], out, p.ch_norm[ch], direct);
  }
}

// Persistent: grid = resident CTAs; each CTA takes the next work item (segment,
// pixel block) from an atomic counter until none are left.  The counter is
// reset by the host before the launch; no CTA waits on another.
// Resident CTAs per SM the instances are compiled for (rec_ctas).  The unmasked FAST one fits in
// 64 registers, and a fourth CTA hides its tile barriers better; the others need 80 (at 64 the
// geometric one spills, 10 MHz 155 -> 167 ms, the compensated one 8.44 against 7.56 ms on
// 200,003 x 65,537).  Packed against single operations (262,144 x 196,249,
// the instances at their best CTAs): unmasked fractional 23.4 -> 22.3 ms, compensated 29.2 -> 27.3
// (32.6 at four CTAs), integer with every fourth term a polynomial 21.5 -> 21.1, REF windows
// 21.45 -> 20.9.
template <int RM, bool COMP, int Q>
__global__ void __launch_bounds__(REC_THREADS, rec_ctas(RM, COMP)) recon_fast_kernel(const ReconParams p) {
  __shared__ RecSmem<RM, COMP, Q> sm;
  __shared__ int s_item;
  const bool frac = __ldg(p.flags + FLAG_FRAC) != 0;
  for (;;) {
    __syncthreads();  // everyone has read the previous item
    if (threadIdx.x == 0) s_item = atomicAdd(p.flags + FLAG_REC_COUNTER, 1);
    __syncthreads();
    const int item = s_item;
    if (item >= p.nitems) break;
    const int seg = item / p.npb;
    const int64_t pb = item - (int64_t)seg * p.npb;
    const int ch = p.seg_ch[seg], slot = p.seg_slot[seg];
    const bool direct = slot < 0;
    float2* out = direct ? p.out + (int64_t)ch * p.J : p.partial + (int64_t)slot * p.J;
    if (frac) recon_rows<RM, true, COMP, Q>(p, sm, pb, p.seg_lo[seg], p.seg_hi[seg], out, p.ch_norm[ch], direct);
    else recon_rows<RM, false, COMP, Q>(p, sm, pb, p.seg_lo[seg], p.seg_hi[seg], out, p.ch_norm[ch], direct);
  }
}

template <int RM, bool COMP, int Q>
static void launch_tile(const ReconParams& p, int ctas_per_sm, cudaStream_t st) {
  const int g = persistent_grid(recon_fast_kernel<RM, COMP, Q>, REC_THREADS, ctas_per_sm, p.nitems);
  recon_fast_kernel<RM, COMP, Q><<<g, REC_THREADS, 0, st>>>(p);
}

// Row tiles of 2 REC_Q visibilities (the default), REC_Q or REC_Q / 2 (tuning).
template <int RM>
static void launch_rm(const ReconParams& p, int ctas_per_sm, bool comp, cudaStream_t st) {
  if (p.row_tile == 1) {
    if (comp) launch_tile<RM, true, REC_Q / 2>(p, ctas_per_sm, st);
    else launch_tile<RM, false, REC_Q / 2>(p, ctas_per_sm, st);
  } else if (p.row_tile == 2) {
    if (comp) launch_tile<RM, true, 2 * REC_Q>(p, ctas_per_sm, st);
    else launch_tile<RM, false, 2 * REC_Q>(p, ctas_per_sm, st);
  } else {
    if (comp) launch_tile<RM, true, REC_Q>(p, ctas_per_sm, st);
    else launch_tile<RM, false, REC_Q>(p, ctas_per_sm, st);
  }
}

template <bool COMP>
static void launch_geo(const ReconParams& p, int ctas_per_sm, cudaStream_t st) {
  const int g = persistent_grid(recon_geo_kernel<COMP>, REC_THREADS, ctas_per_sm, p.nitems);
  recon_geo_kernel<COMP><<<g, REC_THREADS, 0, st>>>(p);
}

int launch_recon_fast(const ReconParams& p, int ctas_per_sm, bool comp, cudaStream_t st) {
  if (p.nitems <= 0) return VISS_OK;
  switch (p.recon_mask) {
    case VISS_RECON_MASK_NONE: launch_rm<RM_NONE>(p, ctas_per_sm, comp, st); break;
    case VISS_RECON_MASK_REF: launch_rm<RM_REF>(p, ctas_per_sm, comp, st); break;
    case VISS_RECON_MASK_GEOMETRIC:
      if (comp) launch_geo<true>(p, ctas_per_sm, st);
      else launch_geo<false>(p, ctas_per_sm, st);
      break;
    default: return fail(VISS_ERR_INVALID, "unknown recon mask");
  }
  VISS_LAUNCH_CHECK("recon_fast_kernel");
  return VISS_OK;
}

// (s + e) * f, rounded once (but for the last bits of e)
__device__ __forceinline__ float pair_times(const FloatPair& v, float f) {
  const float h = __fmul_rn(v.s, f);
  if (isinf(h)) return h;
  return h + __fmaf_rn(v.e, f, __fmaf_rn(v.s, f, -h));
}

// F[c] = norm_c * -(sum of channel c's partial slots), slots summed in a fixed order.
// 10 MHz (256 slots x 196,608 pixels, 400 MB): 262 -> 48 us.
__global__ void __launch_bounds__(32 * RED_GROUPS) recon_reduce_kernel(const RecReduceParams p) {
  const int64_t pos = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31);
  const int c = blockIdx.y;
  if (p.nslot[c] == 0) return;
  FloatPair re, im;
  const float2* const part = p.partial + (int64_t)p.slot0[c] * p.J + pos;
  const float norm = p.norm[c];
  reduce_partials(part, p.nslot[c], p.J, pos < p.J, re, im);
  if (threadIdx.x < 32 && pos < p.J) {
    const int64_t j = p.perm ? (int64_t)p.perm[pos] : pos;
    float2 o = make_float2(pair_times(re, -norm), pair_times(im, -norm));
    if (!re.in_range() || !im.in_range()) {
      const double2 d = sum_partials_f64(part, p.nslot[c], p.J);
      o = make_float2((float)(-d.x * norm), (float)(-d.y * norm));
    }
    p.out[(int64_t)c * p.J + j] = o;
  }
}

int launch_recon_reduce(const RecReduceParams& p, cudaStream_t st) {
  if (p.J <= 0 || p.nch <= 0) return VISS_OK;
  recon_reduce_kernel<<<dim3((unsigned)((p.J + 31) / 32), (unsigned)p.nch), 32 * RED_GROUPS, 0, st>>>(p);
  VISS_LAUNCH_CHECK("recon_reduce_kernel");
  return VISS_OK;
}

// ---------------------------------------------------------------- plain
// The reference's plain recon, restated: one thread per pixel, FP32 phase
//   ph = u*l/d + v*m/d + w*(n + n_offset)/d,  x = +2 pi ph   (vissGen10M_shade.cu:169)
// precise sincosf, register accumulator (optim1, :235-271); reference ratio
// mask evaluated per term from r1 = M1/M2, r2 = M3/M4 (:166).
// F64 (the FP64-phase arm of precision sweeps): the phase in FP64, reduced to
// [-1/2, 1/2] turn in FP64, sincosf of the float angle, Kahan sums.
struct PlainRecArgs {
  const float *u, *v, *w, *wgt, *V, *l, *m, *n;
  const float* r1;
  const float* r2;
  const int32_t* snap;
  const int32_t* pair;
  const float* sat_pos;
  const float4* satdir;
  int64_t K, J;
  int nsat;
  int rmask;
  int res;
  float dl, dm, dn;
  float noff;
  double noff64;
  float norm;
  double R;
  float2* out;
  int* flags;  // near-limb count (may be null)
};

template <bool F64>
__global__ void recon_plain_kernel(const PlainRecArgs a) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= a.J) return;
  const float phiP = floorf((float)(j / a.res));
  const float thetaP = (float)j - phiP * (float)a.res;
  const float lj = a.l[j], mj = a.m[j], nj = a.n[j] + a.noff;
  // FP64-phase arm: l/d, m/d, (n + n_offset)/d in double
  const double ld = (double)a.l[j] / (double)a.dl, md = (double)a.m[j] / (double)a.dm;
  const double nd = ((double)a.n[j] + a.noff64) / (double)a.dn;
  const float p2 = 2.0f * (float)kPi;
  float fr = 0.f, fi = 0.f, cr = 0.f, ci = 0.f;
  for (int64_t k = 0; k < a.K; ++k) {
    if (a.rmask == VISS_RECON_MASK_REF) {
      const float t0 = a.r1[k], p0 = a.r2[k];
      if (fabsf(t0 - thetaP) < t0 && fabsf(p0 - phiP) < p0) continue;
    } else if (a.rmask == VISS_RECON_MASK_GEOMETRIC) {
      const int s = a.snap[k], pr = a.pair[k];
      const int64_t g1 = (int64_t)s * a.nsat + (pr & 0xffff), g2 = (int64_t)s * a.nsat + ((pr >> 16) & 0xffff);
      if (geo_test_plain(a.l[j], a.m[j], a.n[j], a.satdir[g1], a.sat_pos + 3 * g1, a.R, a.flags) ||
          geo_test_plain(a.l[j], a.m[j], a.n[j], a.satdir[g2], a.sat_pos + 3 * g2, a.R, a.flags))
        continue;
    }
    float sn, cs;
    if (F64) {
      const double t = fma((double)a.u[k], ld, fma((double)a.v[k], md, (double)a.w[k] * nd));
      sincosf((float)((t - rint(t)) * (2.0 * kPi)), &sn, &cs);
    } else {
      const float ph = a.u[k] * lj / a.dl + a.v[k] * mj / a.dm + a.w[k] * nj / a.dn;
      sincosf(p2 * ph, &sn, &cs);
    }
    const float wg = a.wgt ? a.wgt[k] : 1.0f;
    const float yr = wg * a.V[2 * k], yi = wg * a.V[2 * k + 1];
    if (F64) {
      kahan_add(fr, cr, yr * cs - yi * sn);
      kahan_add(fi, ci, yr * sn + yi * cs);
    } else {
      fr += yr * cs - yi * sn;
      fi += yr * sn + yi * cs;
    }
  }
  a.out[j] = make_float2(fr * a.norm, fi * a.norm);
}

int launch_recon_plain(const viss_dft_cfg& cfg, const viss_sky& sky, const viss_vis_set& vis,
                       const viss_geometry* geo, const float* V, const float* ratios, const float4* satdir,
                       const float* dlmn, float2* out, cudaStream_t st, int* flags) {
  PlainRecArgs a{};
  a.flags = flags;
  a.satdir = satdir;
  a.u = vis.u; a.v = vis.v; a.w = vis.w; a.wgt = vis.wgt; a.V = V;
  a.l = sky.l; a.m = sky.m; a.n = sky.n;
  a.r1 = ratios; a.r2 = ratios ? ratios + vis.K : nullptr;
  a.snap = vis.snap; a.pair = vis.pair;
  a.sat_pos = geo ? geo->sat_pos : nullptr;
  a.nsat = geo ? geo->nsat : 0;
  a.K = vis.K; a.J = sky.J;
  a.rmask = cfg.recon_mask;
  a.res = cfg.res > 0 ? cfg.res : 1;
  a.dl = dlmn[0]; a.dm = dlmn[1]; a.dn = dlmn[2];
  a.noff = (float)cfg.n_offset;
  a.noff64 = cfg.n_offset;
  a.norm = (float)cfg.norm;
  a.R = cfg.moon_radius_km;
  a.out = out;
  if (a.J <= 0) return VISS_OK;
  if (cfg.precision == VISS_PREC_F64_PHASE) recon_plain_kernel<true><<<(unsigned)((a.J + 255) / 256), 256, 0, st>>>(a);
  else recon_plain_kernel<false><<<(unsigned)((a.J + 255) / 256), 256, 0, st>>>(a);
  VISS_LAUNCH_CHECK("recon_plain_kernel");
  return VISS_OK;
}

}  // namespace viss
