// CSR validation and per-row sorting on the device.
//
// The reference validates shards on the host (InvalidShard, scx-gpu/src/
// error.rs) and sorts indices before the GPU call (ensure_csr,
// pyscx/src/accel/pca.rs:900).  Here both run where the matrix lives.
#include <algorithm>

#include "common.cuh"
#include "launch.h"

namespace scx {

// One warp per row, 128 entries a step: each lane has four indices and four
// values on the way, which is what keeps HBM busy (one of each: 246 us for 92M
// FP32 entries; four, and blocks enough for a short last wave: 211; the bytes
// alone take 114).  A row's order is
// checked between neighbouring lanes and across steps by shuffles.
template <typename ValT>
__global__ void __launch_bounds__(256) k_validate_csr(const int64_t* __restrict__ indptr,
                                                      const int32_t* __restrict__ idx, const ValT* __restrict__ val,
                                                      int64_t n, int64_t g, int64_t nnz, int32_t* __restrict__ flags) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  bool bad_ptr = false, bad_idx = false, bad_order = false, bad_val = false;
  for (int64_t row = warp; row < n; row += nwarps) {
    const int64_t s = indptr[row], e = indptr[row + 1];
    if (s < 0 || e < s || e > nnz) {
      bad_ptr = true;
      continue;
    }
    int32_t before = INT32_MIN;  // the index in front of the step's first
    for (int64_t b = s; b < e; b += 128) {
      int32_t j[4];
      ValT x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t p = b + 32 * u + lane;
        j[u] = p < e ? __ldg(idx + p) : INT32_MAX;
        x[u] = p < e ? val[p] : ValT();
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t p = b + 32 * u + lane;
        int32_t prev = __shfl_up_sync(0xffffffffu, j[u], 1);
        if (lane == 0) prev = before;
        before = __shfl_sync(0xffffffffu, j[u], 31);
        if (p < e) {
          bad_idx |= j[u] < 0 || (int64_t)j[u] >= g;
          bad_order |= p > s && prev >= j[u];
          bad_val |= !isfinite(to_f32(x[u]));
        }
      }
    }
  }
  if (bad_ptr) atomicOr(&flags[0], 1);
  if (bad_idx) atomicOr(&flags[1], 1);
  if (bad_order) atomicOr(&flags[2], 1);
  if (bad_val) atomicOr(&flags[3], 1);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (indptr[0] != 0 || indptr[n] != nnz) atomicOr(&flags[0], 1);
  }
}

// The row pointers and the index range alone (flags[0], flags[1]), for callers
// that read neither order nor values here: half the bytes, and no row
// structure to follow, so the entries go as one array.
__global__ void __launch_bounds__(256) k_check_indices(const int64_t* __restrict__ indptr,
                                                       const int32_t* __restrict__ idx, int64_t n, int64_t g,
                                                       int64_t nnz, int32_t* __restrict__ flags) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
  bool bad_ptr = false, bad_idx = false;
  for (int64_t i = t; i < n; i += nt) {
    const int64_t s = indptr[i], e = indptr[i + 1];
    bad_ptr |= s < 0 || e < s || e > nnz;
  }
  for (int64_t p = t; p < nnz; p += 8 * nt) {
    int32_t j[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) j[u] = p + u * nt < nnz ? __ldg(idx + p + u * nt) : 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) bad_idx |= j[u] < 0 || (int64_t)j[u] >= g;
  }
  if (t == 0) bad_ptr |= indptr[0] != 0 || indptr[n] != nnz;
  if (bad_ptr) atomicOr(&flags[0], 1);
  if (bad_idx) atomicOr(&flags[1], 1);
}

cudaError_t launch_check_indices(const int64_t* indptr, const int32_t* idx, int64_t n, int64_t g, int64_t nnz,
                                 int32_t* flags, cudaStream_t st, int num_sms) {
  note_launches(1);
  k_check_indices<<<grid_for(std::max(n, nnz / 8) + 1, 256, num_sms, 8), 256, 0, st>>>(indptr, idx, n, g, nnz, flags);
  return cudaGetLastError();
}

cudaError_t launch_validate_csr(int dtype, const int64_t* indptr, const int32_t* idx,
                                const void* val, int64_t n, int64_t g, int64_t nnz,
                                int32_t* flags, cudaStream_t st, int num_sms) {
  int grid = grid_for(n * 32 + 32, 256, num_sms, 64);
  note_launches(1);
  switch (dtype) {
    case 0: k_validate_csr<float><<<grid, 256, 0, st>>>(indptr, idx, (const float*)val, n, g, nnz, flags); break;
    case 1: k_validate_csr<__nv_bfloat16><<<grid, 256, 0, st>>>(indptr, idx, (const __nv_bfloat16*)val, n, g, nnz, flags); break;
    default: k_validate_csr<__half><<<grid, 256, 0, st>>>(indptr, idx, (const __half*)val, n, g, nnz, flags); break;
  }
  return cudaGetLastError();
}

// Sort a row by gene: rows up to 1024 entries with a bitonic sort in shared
// memory (one block of 256 threads per row batch); longer rows by a
// single-thread insertion sort (rare for cells x genes data).  Equal genes
// keep both entries (duplicates are summed by every product kernel).
template <typename ValT>
__global__ void k_sort_rows(const int64_t* __restrict__ indptr, int32_t* __restrict__ idx,
                            ValT* __restrict__ val, int64_t n) {
  constexpr int CAP = 1024;
  __shared__ int32_t key[CAP];
  __shared__ ValT vv[CAP];
  for (int64_t row = blockIdx.x; row < n; row += gridDim.x) {
    const int64_t s = indptr[row], e = indptr[row + 1];
    const int len = (int)(e - s);
    if (len <= 1) continue;
    if (len > CAP) {
      if (threadIdx.x == 0) {
        for (int64_t a = s + 1; a < e; ++a) {
          int32_t kj = idx[a];
          ValT kv = val[a];
          int64_t b = a - 1;
          while (b >= s && idx[b] > kj) {
            idx[b + 1] = idx[b];
            val[b + 1] = val[b];
            --b;
          }
          idx[b + 1] = kj;
          val[b + 1] = kv;
        }
      }
      __syncthreads();
      continue;
    }
    int pow2 = 1;
    while (pow2 < len) pow2 <<= 1;
    for (int t = threadIdx.x; t < pow2; t += blockDim.x) {
      key[t] = t < len ? idx[s + t] : INT32_MAX;
      if (t < len) vv[t] = val[s + t];
    }
    __syncthreads();
    for (int size = 2; size <= pow2; size <<= 1) {
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        for (int t = threadIdx.x; t < pow2; t += blockDim.x) {
          int partner = t ^ stride;
          if (partner > t) {
            bool up = (t & size) == 0;
            int32_t a = key[t], b = key[partner];
            if ((a > b) == up) {
              key[t] = b;
              key[partner] = a;
              if (t < CAP && partner < CAP) {
                ValT tv = vv[t];
                vv[t] = vv[partner];
                vv[partner] = tv;
              }
            }
          }
        }
        __syncthreads();
      }
    }
    for (int t = threadIdx.x; t < len; t += blockDim.x) {
      idx[s + t] = key[t];
      val[s + t] = vv[t];
    }
    __syncthreads();
  }
}

cudaError_t launch_sort_rows(int dtype, const int64_t* indptr, int32_t* idx, void* val, int64_t n,
                             cudaStream_t st, int num_sms) {
  if (n == 0) return cudaSuccess;
  int grid = grid_for(n, 1, num_sms, 8);
  note_launches(1);
  switch (dtype) {
    case 0: k_sort_rows<float><<<grid, 256, 0, st>>>(indptr, idx, (float*)val, n); break;
    case 1: k_sort_rows<__nv_bfloat16><<<grid, 256, 0, st>>>(indptr, idx, (__nv_bfloat16*)val, n); break;
    default: k_sort_rows<__half><<<grid, 256, 0, st>>>(indptr, idx, (__half*)val, n); break;
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Exclusive prefix sum of n int64 counts into out[0..n] (out[n] = total), in
// three launches: the sum of every tile to out[end of the tile], one block
// turns those into running totals in place, and each tile is scanned from the
// total in front of it.  It needs no scratch (a library scan's, taken from the
// default pool and given back, cost 290 us of unmapping and mapping per call).
// ---------------------------------------------------------------------------
constexpr int kScanTile = 2048;  // 256 threads x 8

__device__ __forceinline__ int64_t block_inclusive(int64_t x, int64_t* warp_sums) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[w] = x;
  __syncthreads();
  for (int u = 0; u < w; ++u) x += warp_sums[u];
  __syncthreads();
  return x;
}

// `flags` (may be null): with flags[0] or flags[1] set, nothing is written.
__device__ __forceinline__ bool refused(const int32_t* flags) { return flags && (flags[0] | flags[1]); }

__global__ void __launch_bounds__(256) k_scan_sums(const int64_t* __restrict__ in, int64_t n, int64_t* out,
                                                   const int32_t* __restrict__ flags) {
  __shared__ int64_t warp_sums[8];
  if (refused(flags)) return;
  const int64_t b = (int64_t)blockIdx.x * kScanTile, e = min(n, b + kScanTile);
  int64_t x = 0;
  for (int64_t i = b + threadIdx.x; i < e; i += 256) x += in[i];
  x = block_inclusive(x, warp_sums);
  if (threadIdx.x == 255) out[e] = x;
}

__global__ void __launch_bounds__(256) k_scan_tops(int64_t n, int64_t* out, const int32_t* __restrict__ flags) {
  __shared__ int64_t warp_sums[8];
  __shared__ int64_t total;
  if (refused(flags)) return;
  const int64_t tiles = (n + kScanTile - 1) / kScanTile;
  if (threadIdx.x == 0) {
    out[0] = 0;
    total = 0;
  }
  __syncthreads();
  for (int64_t b = 0; b < tiles; b += 256) {
    const int64_t t = b + threadIdx.x, at = min(n, (t + 1) * kScanTile);
    const int64_t x = block_inclusive(t < tiles ? out[at] : 0, warp_sums) + total;
    if (t < tiles) out[at] = x;
    __syncthreads();  // everyone has read the total
    if (threadIdx.x == 255) total = x;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) k_scan_tiles(const int64_t* __restrict__ in, int64_t n, int64_t* out,
                                                    const int32_t* __restrict__ flags) {
  __shared__ int64_t warp_sums[8];
  if (refused(flags)) return;
  const int64_t b = (int64_t)blockIdx.x * kScanTile;
  const int64_t base = out[b];  // the tile in front writes this place too, with the value it holds
  const int64_t i0 = b + threadIdx.x * 8;
  int64_t x[8], sum = 0;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    x[u] = i0 + u < n ? in[i0 + u] : 0;
    sum += x[u];
  }
  int64_t run = block_inclusive(sum, warp_sums) - sum + base;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    run += x[u];
    if (i0 + u < n) out[i0 + u + 1] = run;
  }
}

cudaError_t launch_exclusive_scan_i64(const int64_t* in, int64_t n, int64_t* out, cudaStream_t st,
                                      const int32_t* flags) {
  const unsigned tiles = (unsigned)((n + kScanTile - 1) / kScanTile);
  note_launches(tiles ? 3 : 1);
  if (tiles) k_scan_sums<<<tiles, 256, 0, st>>>(in, n, out, flags);
  k_scan_tops<<<1, 256, 0, st>>>(n, out, flags);
  if (tiles) k_scan_tiles<<<tiles, 256, 0, st>>>(in, n, out, flags);
  return cudaGetLastError();
}

}  // namespace scx
