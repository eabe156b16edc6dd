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
// (6 x 32 x 32 cells, a few pixels each), then each cell's few pixels by index, so that
// the order is the same every time (a crowded cell keeps the order it was filled in: no result
// depends on it, the reconstruction sums a pixel's rows in the same order wherever it stands).
// The device-wide sort takes 2 launches up to ~4,000 pixels and 6 with 5 memsets above: 39 us
// for 12,288 pixels, 17 here (2,048: 10.5, 6.6).
constexpr int SMALL_THREADS = 1024;
constexpr int SMALL_ITEMS = 16;  // pixels per thread, their cells in registers
constexpr int SMALL_MAX = SMALL_ITEMS * SMALL_THREADS;
constexpr int SMALL_BITS = 13;
constexpr int SMALL_CELLS = 6 << (SMALL_BITS - 3);
constexpr int SMALL_SORT = 32;  // cells of up to so many pixels are put in order

__global__ void __launch_bounds__(SMALL_THREADS) small_order_kernel(const float* l, const float* m, const float* n, int J,
                                                                    int32_t* perm) {
  constexpr int PER = SMALL_CELLS / SMALL_THREADS;
  static_assert(SMALL_CELLS % SMALL_THREADS == 0, "whole cells per thread");
  extern __shared__ int small_smem[];
  int* const count = small_smem;
  int* const order = small_smem + SMALL_CELLS;  // [J]
  __shared__ int warp_sum[32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int i = tid; i < SMALL_CELLS; i += SMALL_THREADS) count[i] = 0;
  int cell[SMALL_ITEMS];
#pragma unroll
  for (int i = 0; i < SMALL_ITEMS; ++i) {
    const int j = tid + i * SMALL_THREADS;
    cell[i] = j < J ? (int)(pixel_key(l[j], m[j], n[j]) >> (23 - SMALL_BITS)) : -1;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < SMALL_ITEMS; ++i)
    if (cell[i] >= 0) atomicAdd(&count[cell[i]], 1);
  __syncthreads();
  int c[PER], mine = 0;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    c[i] = count[tid * PER + i];
    mine += c[i];
  }
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_sum[wid] = incl;
  __syncthreads();
  int start = incl - mine;
  for (int w = 0; w < wid; ++w) start += warp_sum[w];
  int at = start;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    count[tid * PER + i] = at;
    at += c[i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < SMALL_ITEMS; ++i)
    if (cell[i] >= 0) order[atomicAdd(&count[cell[i]], 1)] = tid + i * SMALL_THREADS;
  __syncthreads();
  at = start;
#pragma unroll 1
  for (int i = 0; i < PER; ++i) {
    if (c[i] > 1 && c[i] <= SMALL_SORT) {
      for (int x = at + 1; x < at + c[i]; ++x) {
        const int v = order[x];
        int y = x;
        while (y > at && order[y - 1] > v) { order[y] = order[y - 1]; --y; }
        order[y] = v;
      }
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
    constexpr int most = (SMALL_CELLS + SMALL_MAX) * (int)sizeof(int);
    VISS_CUDA(cudaFuncSetAttribute(small_order_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    small_order_kernel<<<1, SMALL_THREADS, (SMALL_CELLS + (size_t)J) * sizeof(int), st>>>(l, m, n, (int)J, perm);
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
