// The order in which receivers are walked: Morton order of their positions.
//
// A warp walks up to 32 cones together: one object hierarchy walk visits the
// union of the nodes its cones need, and their mesh walks share what they load,
// so cones in a warp should see the same geometry. Callers
// list receivers in their own order (image rows, texels of many pages); here
// each receiver gets a Morton code of its position quantized in the scene's
// bounds, and a device radix sort yields the walk order. Results do
// not depend on the order — only which cones share a warp.
#include <cub/device/device_radix_sort.cuh>

#include <cstdint>

#include "kernels.h"

namespace cc {

namespace {

__device__ __forceinline__ uint32_t grid_code(const OrderGrid& g, float4 p) {
  const float x[3] = {p.x, p.y, p.z};
  uint32_t c[3];
  int top = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float most = (float)((1u << g.bits[k]) - 1u);
    c[k] = (uint32_t)fminf(fmaxf((x[k] - g.lo[k]) * g.inv, 0.0f), most);  // NaN clamps to 0
    top = max(top, g.bits[k]);
  }
  uint32_t code = 0;
  for (int b = top - 1; b >= 0; --b) {
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (b < g.bits[k]) code = (code << 1) | ((c[k] >> b) & 1u);
  }
  return code;
}

__global__ void morton_keys(const float4* __restrict__ receivers, uint64_t n, OrderGrid grid, uint32_t* __restrict__ keys,
                            uint32_t* __restrict__ index) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  keys[i] = grid_code(grid, __ldg(&receivers[2 * i]));
  index[i] = (uint32_t)i;
}

// Batch keys: the job's index above the point's code; values: the point's
// index within its job.
__global__ void batch_morton_keys(BatchLaunch b, unsigned long long* __restrict__ keys,
                                  uint32_t* __restrict__ index) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.points) return;
  uint32_t lo = 0, hi = b.njobs;  // jobs[lo].point_start <= i < jobs[hi].point_start
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(&b.jobs[mid].point_start) <= i) lo = mid; else hi = mid;
  }
  const JobGpu& J = b.jobs[lo];
  const uint64_t local = i - J.point_start;
  keys[i] = ((unsigned long long)lo << kCodeBits) | grid_code(J.grid, __ldg(&J.query.receivers[2 * local]));
  index[i] = (uint32_t)local;
}

int job_bits(uint32_t njobs) {
  int bits = 0;
  while ((1ull << bits) < njobs) ++bits;
  return bits;
}

}  // namespace

OrderGrid grid_over(const float* lo, const float* hi) {
  OrderGrid g;
  float e[3], longest = 0.0f;
  for (int k = 0; k < 3; ++k) {
    g.lo[k] = lo[k];
    e[k] = hi[k] - lo[k];
    if (!(e[k] > 0.0f)) e[k] = 0.0f;
    longest = e[k] > longest ? e[k] : longest;
    g.bits[k] = 0;
  }
  g.inv = 0.0f;
  if (!(longest > 0.0f) || !(longest < 1e30f)) return g;
  // Halve the cell from the longest axis's length while the codes fit.
  float side = longest;
  for (;;) {
    int bits[3], sum = 0;
    for (int k = 0; k < 3; ++k) {
      bits[k] = 0;
      while (bits[k] < kCodeBits && side * 0.5f * (float)(1u << bits[k]) < e[k] && bits[k] < 31) ++bits[k];
      sum += bits[k];
    }
    if (sum > kCodeBits || bits[0] > 20 || bits[1] > 20 || bits[2] > 20) break;
    for (int k = 0; k < 3; ++k) g.bits[k] = bits[k];
    side *= 0.5f;
  }
  g.inv = 1.0f / side;
  return g;
}

size_t batch_order_scratch_bytes(uint64_t points) {
  size_t temp = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, temp, (const unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                  (const uint32_t*)nullptr, (uint32_t*)nullptr, (int)points, 0, 62);
  return points * (2 * sizeof(unsigned long long) + sizeof(uint32_t)) + temp + 512;
}

cudaError_t batch_order(const BatchLaunch& b, void* scratch, size_t scratch_bytes, uint32_t* order,
                        cudaStream_t stream) {
  if (b.points == 0 || b.njobs == 0) return cudaSuccess;
  const uint64_t n = b.points;
  auto align = [](uint8_t* p) {
    return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 255) & ~uintptr_t(255));
  };
  uint8_t* base = align(static_cast<uint8_t*>(scratch));
  unsigned long long* keys_in = reinterpret_cast<unsigned long long*>(base);
  unsigned long long* keys_out = keys_in + n;
  uint32_t* idx_in = reinterpret_cast<uint32_t*>(keys_out + n);
  uint8_t* temp = align(reinterpret_cast<uint8_t*>(idx_in + n));
  const size_t used = static_cast<size_t>(temp - static_cast<uint8_t*>(scratch));
  if (used > scratch_bytes) return cudaErrorInvalidValue;
  size_t temp_bytes = scratch_bytes - used;
  const unsigned threads = 256;
  const unsigned blocks = (unsigned)((n + threads - 1) / threads);
  batch_morton_keys<<<blocks, threads, 0, stream>>>(b, keys_in, idx_in);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return cub::DeviceRadixSort::SortPairs(temp, temp_bytes, keys_in, keys_out, idx_in, order, (int)n, 0,
                                         kCodeBits + job_bits(b.njobs), stream);
}

size_t walk_order_scratch_bytes(uint64_t npoints) {
  size_t temp = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, temp, (const uint32_t*)nullptr, (uint32_t*)nullptr,
                                  (const uint32_t*)nullptr, (uint32_t*)nullptr, (int)npoints, 0, kCodeBits);
  return 4 * npoints * sizeof(uint32_t) + temp + 256;
}

cudaError_t walk_order(const float4* receivers, uint64_t npoints, const float* scene_lo, const float* scene_hi,
                       void* scratch, size_t scratch_bytes, uint32_t* order, cudaStream_t stream) {
  if (npoints == 0) return cudaSuccess;
  uint32_t* keys_in = static_cast<uint32_t*>(scratch);
  uint32_t* keys_out = keys_in + npoints;
  uint32_t* idx_in = keys_out + npoints;
  uint8_t* temp = reinterpret_cast<uint8_t*>(idx_in + npoints);
  // 256-byte alignment for the sort's temporary storage.
  temp = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(temp) + 255) & ~uintptr_t(255));
  const size_t used = static_cast<size_t>(temp - static_cast<uint8_t*>(scratch));
  if (used > scratch_bytes) return cudaErrorInvalidValue;
  size_t temp_bytes = scratch_bytes - used;
  const OrderGrid grid = grid_over(scene_lo, scene_hi);
  const unsigned threads = 256;
  const unsigned blocks = (unsigned)((npoints + threads - 1) / threads);
  morton_keys<<<blocks, threads, 0, stream>>>(receivers, npoints, grid, keys_in, idx_in);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return cub::DeviceRadixSort::SortPairs(temp, temp_bytes, keys_in, keys_out, idx_in, order, (int)npoints, 0,
                                         max(grid.bits[0] + grid.bits[1] + grid.bits[2], 1), stream);
}

}  // namespace cc
