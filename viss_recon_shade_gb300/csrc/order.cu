// order.cu -- spatial permutation of the sky (cube-face Morton order), used by
// the geometric-mask passes so that a warp's pixels form a compact patch.
#include <cub/cub.cuh>

#include "viss_internal.cuh"

namespace viss {

// ------------------------------------------------------------- pixel order
// Spatial order of the sky for the geometric mask: the direction is projected
// on the face of the cube it points to and the face coordinates (10 bits each)
// are interleaved (Morton), so consecutive positions are neighbouring pixels
// and a warp's pixels see the Moon's limb together.
// 10 bits -> the even bits of 20 (2-D Morton interleave)
__device__ __forceinline__ uint32_t spread10(uint32_t x) {
  x &= 0x3ff;
  x = (x | (x << 8)) & 0x00ff00ffu;
  x = (x | (x << 4)) & 0x0f0f0f0fu;
  x = (x | (x << 2)) & 0x33333333u;
  x = (x | (x << 1)) & 0x55555555u;
  return x;
}

__device__ __forceinline__ uint32_t pixel_key(float x, float y, float z) {
  const float ax = fabsf(x), ay = fabsf(y), az = fabsf(z);
  uint32_t face;
  float a, b, d;
  if (ax >= ay && ax >= az) { face = x >= 0 ? 0 : 1; a = y; b = z; d = ax; }
  else if (ay >= az) { face = y >= 0 ? 2 : 3; a = x; b = z; d = ay; }
  else { face = z >= 0 ? 4 : 5; a = x; b = y; d = az; }
  const float inv = d > 0.f ? 1.0f / d : 0.f;
  const uint32_t ia = (uint32_t)fminf(1023.f, fmaxf(0.f, (a * inv + 1.0f) * 511.5f));
  const uint32_t ib = (uint32_t)fminf(1023.f, fmaxf(0.f, (b * inv + 1.0f) * 511.5f));
  return (face << 20) | (spread10(ia) << 1) | spread10(ib);
}

__global__ void pixel_keys_kernel(const float* l, const float* m, const float* n, int64_t J, uint32_t* keys,
                                  int32_t* idx) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= J) return;
  keys[j] = pixel_key(l[j], m[j], n[j]);
  idx[j] = (int32_t)j;
}

static int launch_pixel_keys(const float* l, const float* m, const float* n, int64_t J, uint32_t* keys, int32_t* idx,
                             cudaStream_t st) {
  pixel_keys_kernel<<<(unsigned)((J + 255) / 256), 256, 0, st>>>(l, m, n, J, keys, idx);
  VISS_LAUNCH_CHECK("pixel_keys_kernel");
  return VISS_OK;
}

namespace {
struct OrderScratch {
  uint32_t *k0 = nullptr, *k1 = nullptr;
  int32_t* i0 = nullptr;
  void* cub = nullptr;
  size_t cub_bytes = 0, bytes = 0;
  void layout(void* ws, int64_t J) {
    Carver c(ws);
    k0 = c.take<uint32_t>(J);
    k1 = c.take<uint32_t>(J);
    i0 = c.take<int32_t>(J);
    size_t a = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, a, (uint32_t*)nullptr, (uint32_t*)nullptr, (int32_t*)nullptr,
                                    (int32_t*)nullptr, (int64_t)J, 0, 23);
    cub_bytes = a;
    cub = c.take<char>(a);
    bytes = c.size();
  }
};
}  // namespace

// Small skies in one block and one launch: a counting sort by the 13 upper bits of the key
// (6 x 32 x 32 cells, a few pixels each), then each cell's few pixels by index.  A sky that crowds
// more than SMALL_SORT pixels into a cell (a narrow field) is sorted by its whole keys instead:
// left as the cell was filled, a pixel's patch would vary from call to call, and with it the order
// in which its rows are added where they are not in snapshot order; and patches scattered over a
// cell are seen or hidden as a whole less often (16,384 pixels in a few degrees, 28,672 rows: 205 -> 199
// us).  The device-wide sort takes 2 launches up to ~4,000 pixels and 6 with 5 memsets above: 30 us for
// 12,288 and 16,384 pixels, here 17 and 22 (2,048: 10.5, 6.6); a field of 16,384 pixels in a few
// degrees 29, here 32 (4,096: 11, 13).
constexpr int SMALL_THREADS = 1024;
constexpr int SMALL_WARPS = SMALL_THREADS / 32;
constexpr int SMALL_ITEMS = 16;  // most pixels per thread, their keys in registers
constexpr int SMALL_MAX = SMALL_ITEMS * SMALL_THREADS;
constexpr int SMALL_BITS = 13;
constexpr int SMALL_CELLS = 6 << (SMALL_BITS - 3);
constexpr int SMALL_SORT = 32;  // cells of up to so many pixels are put in order one by one
constexpr int SMALL_DIGITS = 256;
constexpr int SMALL_ROW = SMALL_DIGITS + 1;  // a warp's counts, padded: the scan reads a digit of eight warps
constexpr uint32_t SMALL_PAD = 0x7fffff;     // key of the positions past the last pixel: above every pixel's (6 << 20)

// Shared memory: the counting sort's counts and order, or the radix sort's keys, counts and order.
static size_t small_smem_bytes(int items) {
  const size_t n = (size_t)items * SMALL_THREADS;
  const size_t cells = sizeof(int) * (SMALL_CELLS + n);
  const size_t radix = n * (sizeof(uint32_t) + sizeof(uint16_t)) + sizeof(int) * SMALL_WARPS * SMALL_ROW;
  return cells > radix ? cells : radix;
}

// The exclusive sum of x over the block's threads.
__device__ __forceinline__ int small_scan(int x, int* warp_sum) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_sum[wid] = incl;
  __syncthreads();
  return incl - x + __reduce_add_sync(0xffffffffu, lane < wid ? warp_sum[lane] : 0);
}

// The lanes that hold the same digit: eight ballots (__match_any_sync takes a step per distinct value).
__device__ __forceinline__ unsigned digit_peers(uint32_t d) {
  unsigned peers = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const bool bit = (d >> b) & 1u;
    const unsigned v = __ballot_sync(0xffffffffu, bit);
    peers &= bit ? v : ~v;
  }
  return peers;
}

// The crowded case: a stable radix sort of the whole keys, up to three passes of 8 bits, which is the
// device-wide sort's order.  A warp takes a run of 32 x items positions, ranks 32 at a time and
// keeps its own counts.
__device__ __forceinline__ void small_radix(const uint32_t* key, int J, int items, uint32_t* smem, int* warp_sum,
                                            int32_t* perm) {
  uint32_t* const keys = smem;                                                           // [items * 1024] by pixel
  int* const count = reinterpret_cast<int*>(smem + items * SMALL_THREADS);               // [warp][SMALL_ROW]
  uint16_t* const order = reinterpret_cast<uint16_t*>(count + SMALL_WARPS * SMALL_ROW);  // [items * 1024]
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int p0 = wid * 32 * items + lane;  // the thread's positions are p0 + 32 i
  int* const mine = count + wid * SMALL_ROW;
#pragma unroll
  for (int i = 0; i < SMALL_ITEMS; ++i) {
    if (i < items) {
      const int j = tid + i * SMALL_THREADS;
      keys[j] = key[i];
      order[j] = (uint16_t)j;
    }
  }
  __shared__ uint32_t differ;  // the bits in which the pixels' keys differ
  if (tid == 0) differ = 0;
  __syncthreads();
  uint32_t mix = 0;
#pragma unroll
  for (int i = 0; i < SMALL_ITEMS; ++i)
    if (key[i] != SMALL_PAD) mix |= key[i] ^ keys[0];
  mix = __reduce_or_sync(0xffffffffu, mix);
  if (lane == 0) atomicOr(&differ, mix);
  __syncthreads();
  static_assert(SMALL_MAX <= 1 << 14 && SMALL_DIGITS <= 1 << 8 && 32 * SMALL_ITEMS <= 1 << 9, "fields of a packed position");
#pragma unroll 1
  for (int shift = 0; shift < 23; shift += 8) {
    if (((differ >> shift) & (SMALL_DIGITS - 1)) == 0) continue;  // one digit (the padding stays behind the pixels)
    uint32_t pos[SMALL_ITEMS];  // pixel | digit << 14 | rank among the warp's positions of that digit << 22
#pragma unroll
    for (int i = 0; i < SMALL_ITEMS; ++i) {
      if (i < items) {
        const uint32_t id = order[p0 + 32 * i];
        pos[i] = id | ((keys[id] >> shift) & (SMALL_DIGITS - 1)) << 14;
      }
    }
    for (int d = lane; d < SMALL_DIGITS; d += 32) mine[d] = 0;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < SMALL_ITEMS; ++i) {
      if (i < items) {
        const uint32_t d = pos[i] >> 14;
        const unsigned peers = digit_peers(d);
        const int before = mine[d];
        __syncwarp();
        if (lane == __ffs(peers) - 1) mine[d] = before + __popc(peers);
        __syncwarp();
        pos[i] |= (uint32_t)(before + __popc(peers & ((1u << lane) - 1u))) << 22;
      }
    }
    __syncthreads();
    // counts -> first positions, digits in order and a digit's warps in order: a thread has eight warps of one digit
    int c[8], sum = 0;
    int* const eight = count + (tid & 3) * 8 * SMALL_ROW + (tid >> 2);
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      c[w] = sum;
      sum += eight[w * SMALL_ROW];
    }
    const int first = small_scan(sum, warp_sum);
#pragma unroll
    for (int w = 0; w < 8; ++w) eight[w * SMALL_ROW] = first + c[w];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < SMALL_ITEMS; ++i)
      if (i < items) order[mine[(pos[i] >> 14) & (SMALL_DIGITS - 1)] + (pos[i] >> 22)] = (uint16_t)(pos[i] & 0x3fff);
    __syncthreads();
  }
  for (int j = tid; j < J; j += SMALL_THREADS) perm[j] = order[j];
}

__global__ void __launch_bounds__(SMALL_THREADS) small_order_kernel(const float* l, const float* m, const float* n, int J,
                                                                    int items, int32_t* perm) {
  constexpr int PER = SMALL_CELLS / SMALL_THREADS;
  static_assert(SMALL_CELLS % SMALL_THREADS == 0, "whole cells per thread");
  extern __shared__ uint32_t small_smem[];
  int* const count = reinterpret_cast<int*>(small_smem);
  int* const order = count + SMALL_CELLS;  // [J]
  __shared__ int warp_sum[SMALL_WARPS];
  const int tid = threadIdx.x;
  __shared__ int crowded;
  for (int i = tid; i < SMALL_CELLS; i += SMALL_THREADS) count[i] = 0;
  if (tid == 0) crowded = 0;
  uint32_t key[SMALL_ITEMS];
#pragma unroll
  for (int i = 0; i < SMALL_ITEMS; ++i) {
    const int j = tid + i * SMALL_THREADS;
    key[i] = j < J ? pixel_key(l[j], m[j], n[j]) : SMALL_PAD;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < SMALL_ITEMS; ++i) {
    // a crowded cell's counts queue on one address: none once one is known
    if (key[i] != SMALL_PAD && !*(volatile int*)&crowded &&
        atomicAdd(&count[key[i] >> (23 - SMALL_BITS)], 1) >= SMALL_SORT)
      crowded = 1;
  }
  __syncthreads();
  if (crowded) {
    __syncthreads();
    small_radix(key, J, items, small_smem, warp_sum, perm);
    return;
  }
  int c[PER], mine = 0;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    c[i] = count[tid * PER + i];
    mine += c[i];
  }
  const int start = small_scan(mine, warp_sum);
  int at = start;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    count[tid * PER + i] = at;
    at += c[i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < SMALL_ITEMS; ++i)
    if (key[i] != SMALL_PAD) order[atomicAdd(&count[key[i] >> (23 - SMALL_BITS)], 1)] = tid + i * SMALL_THREADS;
  __syncthreads();
  at = start;
#pragma unroll 1
  for (int i = 0; i < PER; ++i) {
    for (int x = at + 1; x < at + c[i]; ++x) {
      const int v = order[x];
      int y = x;
      while (y > at && order[y - 1] > v) { order[y] = order[y - 1]; --y; }
      order[y] = v;
    }
    at += c[i];
  }
  __syncthreads();
  for (int j = tid; j < J; j += SMALL_THREADS) perm[j] = order[j];
}

size_t pixel_order_scratch(int64_t J) {
  if (J <= SMALL_MAX) return 0;
  OrderScratch s;
  s.layout(nullptr, J);
  return s.bytes;
}

int pixel_order(const float* l, const float* m, const float* n, int64_t J, void* scratch, size_t scratch_bytes,
                int32_t* perm, cudaStream_t st) {
  if (J <= 0) return VISS_OK;
  if (J <= SMALL_MAX) {
    const int items = (int)((J + SMALL_THREADS - 1) / SMALL_THREADS);
    VISS_CUDA(cudaFuncSetAttribute(small_order_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)small_smem_bytes(SMALL_ITEMS)));
    small_order_kernel<<<1, SMALL_THREADS, small_smem_bytes(items), st>>>(l, m, n, (int)J, items, perm);
    VISS_LAUNCH_CHECK("small_order_kernel");
    return VISS_OK;
  }
  OrderScratch s;
  s.layout(nullptr, J);
  if (!scratch || scratch_bytes < s.bytes) return fail(VISS_ERR_WORKSPACE, "pixel order scratch too small");
  s.layout(scratch, J);
  int rc = launch_pixel_keys(l, m, n, J, s.k0, s.i0, st);
  if (rc) return rc;
  size_t cb = s.cub_bytes;
  VISS_CUDA(cub::DeviceRadixSort::SortPairs(s.cub, cb, s.k0, s.k1, s.i0, perm, J, 0, 23, st));
  return VISS_OK;
}

}  // namespace viss
