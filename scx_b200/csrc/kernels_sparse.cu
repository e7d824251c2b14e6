// Sparse-side kernels: per-gene statistics, value transforms, the forward
// product Y = (X - 1 mu^T) V and the transposed product W = X^T Q on the
// CUDA cores (FP32 products, FP32/FP64 accumulation).
//
// Layouts (all device memory):
//   CSR    : int64 indptr[n+1], int32 indices[nnz], values[nnz] (f32/bf16/f16)
//   V      : float [n_vars][ld]   gene-major, ld = k padded to 32, pad = 0
//   Y, Q   : float [n_obs][ld]    cell-major
//   partial: float [n_chunks][n_vars][ld] per-chunk partial X^T Q
#include <algorithm>

#include "common.cuh"
#include "launch.h"

namespace scx {

// ---------------------------------------------------------------------------
// Per-gene sums and sums of squares (FP64), in a fixed order: the result is
// bit-identical from run to run.  Restates ScxCsr::col_sums_and_sum_sq
// (scx-sparse/src/csr.rs:570-580).
//
// Part b of the partition owns the stored entries [b * per, (b + 1) * per) and
// one FP64 accumulator pair per gene in shared memory.  A warp walks the part's
// entries 32 at a time; where few parts fit an SM, several warps walk the same
// part, each adding its own range of the genes.  No two warps touch one
// accumulator, so there are no atomics and no barriers.  Inside one 32-entry
// step two lanes may name the same gene only across a row boundary (a sorted row
// holds a gene once); the step is cut into runs of strictly increasing gene
// index, applied one after another in lane order.  Every gene's adds therefore
// happen in entry order, whatever the rows look like (unsorted rows and
// duplicates included) and however many warps share the part.  Genes beyond the
// shared-memory accumulators take further passes over the part's entries, of at
// most kStatsPassGenes genes each.  Each part writes one partial row pair
// [sum | sum sq] (n_vars each); reduce_rows_f64 adds the partials in order.
//
// What bounds it is latency: of a step's read-modify-write of 32 scattered
// 16-byte pairs, and of the loads when few warps run.  As many parts run on an
// SM as have room for their accumulators (6 at 2,000 genes); a warp takes two
// steps at once where their 64 genes increase, so their updates cannot meet
// (most pairs: a row has some 190 entries), and loads eight steps ahead, as
// stored (a conversion in the load would wait for it).  92M entries: 366 us
// FP32, 373 BF16, against 825 and 912 for one accumulator set per block, its
// genes dealt to four warps through a bucket sort of every 1,024-entry window.
// (One step at a time: 526.)
//
// Above 4,266 genes at most two parts fit.  Their warps are made up to
// kStatsLeast by ranges and load sixteen steps ahead, and where the entries are
// worth the partials there are four parts per SM, in turn, so that a piece of an
// upload still fills half of the SMs.
// 46M entries, one warp a part and eight steps against this: 8,000 genes 850 ->
// 660 us, 12,800 855 -> 656, 30,000 2,468 -> 1,627 (the bucket sort: 1,071,
// 1,608, 2,146); in a plan from host memory at 30,000 genes they take 10 ms less,
// as the pieces no longer outlast the copy.  Ranges without the longer loads
// gain nothing, the loads alone 17 % at 30,000 genes and nothing at 12,800; with
// three parts an SM neither gains.
// ---------------------------------------------------------------------------
constexpr int kStatsMaxWarps = 16;  // warps of a block
constexpr int kStatsPassGenes = (int)(kStatsSmemMax / 16);
constexpr int kStatsLeast = 4;      // warps of a block whose parts are shared
constexpr int kStatsOwn = 3;        // parts of a block from which on each has one warp
constexpr int kStatsWorth = 16384;  // entries that are worth a partial of a wide matrix

// Parts whose accumulators fit an SM's shared memory.
static int stats_sets(int64_t g) {
  const int64_t pass = std::min<int64_t>(std::max<int64_t>(g, 1), kStatsPassGenes);
  return (int)std::min<int64_t>(kStatsMaxWarps, (int64_t)kStatsSmemMax / (16 * pass));
}

int col_stats_parts(int64_t g, int64_t nnz, int num_sms) {
  const int sets = stats_sets(g), four = 4 * num_sms;
  return sets < kStatsOwn && nnz >= (int64_t)four * kStatsWorth ? four : num_sms * sets;
}

// SHARED: `ranges` warps walk a part, and a step may hold none of a warp's genes.
template <typename ValT, bool SHARED>
__global__ void __launch_bounds__(SHARED ? kStatsLeast * 32 : kStatsMaxWarps * 32)
    k_col_stats(const int32_t* __restrict__ idx, const ValT* __restrict__ val, int64_t nnz, int32_t g,
                int32_t pass_genes, int ranges, int nparts, int part0, int part1, double* __restrict__ partial) {
  constexpr int AHEAD = SHARED ? 16 : 8;  // 32-entry steps a warp loads at once, before it needs them
  extern __shared__ __align__(16) double2 stats_sm[];  // [parts of the block][pass_genes]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, set = warp / ranges, range = warp % ranges;
  const unsigned lanemask_le = 0xffffffffu >> (31 - lane);
  // this launch runs parts part0 .. part1 - 1 of the partition
  const int b = part0 + (int)blockIdx.x * ((int)(blockDim.x >> 5) / ranges) + set;
  if (b >= part1) return;
  double2* acc = stats_sm + (int64_t)set * pass_genes;
  const int64_t per = (nnz + nparts - 1) / nparts;
  const int64_t s = min(nnz, (int64_t)b * per);
  const int64_t e = min(nnz, s + per);
  double* out = partial + (int64_t)b * 2 * g;
  for (int32_t lo = 0; lo < g; lo += pass_genes) {
    const int32_t gp = min(pass_genes, g - lo);
    // the warp's genes of this pass, lo + [i0, i1): the same accumulators in
    // every pass, as the part's other warps may be a pass behind
    const int32_t i0 = min(gp, pass_genes * range / ranges), i1 = min(gp, pass_genes * (range + 1) / ranges);
    for (int i = i0 + lane; i < i1; i += 32) acc[i] = make_double2(0.0, 0.0);
    int32_t nj[AHEAD];
    ValT nx[AHEAD];
    auto load = [&](int64_t w) {
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const int64_t p = w + 32 * u + lane;
        nj[u] = p < e ? __ldg(idx + p) : INT32_MAX;
        nx[u] = p < e ? val[p] : ValT();
      }
    };
    // (an index out of range is no warp's)
    auto in_range = [&](int32_t j) { return j >= lo + i0 && j - lo < i1; };
    auto add = [](double2& a, double x) {
      a.x += x;
      a.y += x * x;
    };
    load(s);
    __syncwarp();  // the accumulators are zeroed
    for (int64_t w0 = s; w0 < e; w0 += 32 * AHEAD) {
      int32_t cj[AHEAD];
      double cx[AHEAD];
      unsigned starts[AHEAD];  // lanes whose gene is not above the lane before's
      bool follows[AHEAD];     // the step's first gene is above the last one of the step before
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        cj[u] = nj[u];
        cx[u] = (double)to_f32(nx[u]);
      }
      load(w0 + 32 * AHEAD);
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const int32_t jl = __shfl_up_sync(0xffffffffu, cj[u], 1);
        starts[u] = __ballot_sync(0xffffffffu, lane > 0 && cj[u] != INT32_MAX && cj[u] <= jl);
        follows[u] = u > 0 && __shfl_sync(0xffffffffu, cj[u], 0) > __shfl_sync(0xffffffffu, cj[u ? u - 1 : 0], 31);
      }
#pragma unroll
      for (int u = 0; u < AHEAD; u += 2) {
        const bool in0 = in_range(cj[u]), in1 = in_range(cj[u + 1]);
        if (SHARED && !__any_sync(0xffffffffu, in0 || in1)) continue;
        if (starts[u] == 0 && starts[u + 1] == 0 && follows[u + 1]) {
          // 64 increasing genes: the two steps' updates do not meet
          double2 a0, a1;
          if (in0) a0 = acc[cj[u] - lo];
          if (in1) a1 = acc[cj[u + 1] - lo];
          if (in0) {
            add(a0, cx[u]);
            acc[cj[u] - lo] = a0;
          }
          if (in1) {
            add(a1, cx[u + 1]);
            acc[cj[u + 1] - lo] = a1;
          }
          __syncwarp();  // the next step's lanes see these updates
        } else {
#pragma unroll
          for (int v = u; v < u + 2; ++v) {
            const int run = __popc(starts[v] & lanemask_le);
            const int runs = __popc(starts[v]) + 1;
            for (int r = 0; r < runs; ++r) {
              if ((v == u ? in0 : in1) && run == r) {
                double2 a = acc[cj[v] - lo];
                add(a, cx[v]);
                acc[cj[v] - lo] = a;
              }
              __syncwarp();
            }
          }
        }
      }
    }
    for (int i = i0 + lane; i < i1; i += 32) {
      out[lo + i] = acc[i].x;
      out[g + lo + i] = acc[i].y;
    }
    __syncwarp();
  }
}

// The value transform of one entry (k_transform_values, below): the working
// value as stored.
template <typename InT, typename OutT>
__device__ __forceinline__ OutT transform_value(InT v, int32_t j, int mode, const double* mu, const double* inv_std,
                                                const double* cshift, double clip) {
  double x = (double)to_f32(v);
  if (mode != 0) {
    const double is = inv_std[j];
    if (mode == 1) {
      double sv = (x - mu[j]) * is;
      if (clip > 0.0) sv = fmin(fmax(sv, -clip), clip);
      x = sv - cshift[j];
    } else {
      x = x * is;
      if (clip > 0.0) x = fmin(x, clip);
    }
  }
  return from_f32<OutT>((float)x);
}

// out[i] (+)= sum_{b < nparts} part[b * len + i] in FP64.  A block takes 32
// consecutive outputs (one per lane, coalesced); warp w sums the partials
// b = w, w + 8, ... with four loads in flight, and warp 0 adds the eight warp
// sums in warp order: a fixed order, so the result is deterministic.
// With width > 0 the output is a column panel of a wider matrix: element i
// goes to out[(i / width) * ldo + i % width].
// FP32 partials with len a multiple of 4: the same sums (warp w adds the
// parts w, w + 8, ... in that order, warp 0 the eight warp sums), but a lane
// takes four consecutive outputs with one 16-byte load per part, so a block
// step covers 128 outputs.  A pass over many small partials (the segments of a
// batch) is bound by the latency of its steps, not by bandwidth.
__device__ __forceinline__ void reduce_rows_body_f4(const float* __restrict__ part, int nparts, int64_t len,
                                                    double* __restrict__ out, int accumulate, int width, int ldo,
                                                    int blk, int nblk) {
  __shared__ double red4[8][4 * 32 + 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (nparts <= 8) {
    // Warp w of the eight would hold part w alone, and warp 0 would add them
    // in warp order: out + p_0 + p_1 + ... .  The same sums, each warp on its
    // own 128 outputs: one step per chunk instead of a block-wide step with
    // most warps idle (the partials of a batch's small segments).
    for (int64_t base = ((int64_t)blk * 8 + w) * 128; base < len; base += (int64_t)nblk * 8 * 128) {
      const int64_t i = base + 4 * lane;
      if (i >= len) continue;
      float4 v[8];
#pragma unroll
      for (int b = 0; b < 8; ++b)
        if (b < nparts) v[b] = *reinterpret_cast<const float4*>(part + (int64_t)b * len + i);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int64_t ie = i + e;
        const int64_t oi = width > 0 ? (ie / width) * ldo + ie % width : ie;
        double acc = accumulate ? out[oi] : 0.0;
#pragma unroll
        for (int b = 0; b < 8; ++b)
          if (b < nparts) acc += (double)(e == 0 ? v[b].x : e == 1 ? v[b].y : e == 2 ? v[b].z : v[b].w);
        out[oi] = acc;
      }
    }
    return;
  }
  for (int64_t base = (int64_t)blk * 128; base < len; base += (int64_t)nblk * 128) {
    const int64_t i = base + 4 * lane;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    if (i < len) {
      int b = w;
      for (; b + 24 < nparts; b += 32) {
        const float4 v0 = *reinterpret_cast<const float4*>(part + (int64_t)b * len + i);
        const float4 v1 = *reinterpret_cast<const float4*>(part + (int64_t)(b + 8) * len + i);
        const float4 v2 = *reinterpret_cast<const float4*>(part + (int64_t)(b + 16) * len + i);
        const float4 v3 = *reinterpret_cast<const float4*>(part + (int64_t)(b + 24) * len + i);
        acc[0] += (double)v0.x; acc[1] += (double)v0.y; acc[2] += (double)v0.z; acc[3] += (double)v0.w;
        acc[0] += (double)v1.x; acc[1] += (double)v1.y; acc[2] += (double)v1.z; acc[3] += (double)v1.w;
        acc[0] += (double)v2.x; acc[1] += (double)v2.y; acc[2] += (double)v2.z; acc[3] += (double)v2.w;
        acc[0] += (double)v3.x; acc[1] += (double)v3.y; acc[2] += (double)v3.z; acc[3] += (double)v3.w;
      }
      for (; b < nparts; b += 8) {
        const float4 v = *reinterpret_cast<const float4*>(part + (int64_t)b * len + i);
        acc[0] += (double)v.x; acc[1] += (double)v.y; acc[2] += (double)v.z; acc[3] += (double)v.w;
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) red4[w][4 * lane + e] = acc[e];
    __syncthreads();
    if (w == 0 && i < len) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int64_t ie = i + e;
        const int64_t oi = width > 0 ? (ie / width) * ldo + ie % width : ie;
        double s = accumulate ? out[oi] : 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u) s += red4[u][4 * lane + e];
        out[oi] = s;
      }
    }
    __syncthreads();
  }
}

template <typename T>
__device__ __forceinline__ void reduce_rows_body(const T* __restrict__ part, int nparts, int64_t len,
                                                 double* __restrict__ out, int accumulate, int width, int ldo,
                                                 int blk, int nblk) {
  if constexpr (sizeof(T) == 4) {
    if ((len & 3) == 0 && (reinterpret_cast<uintptr_t>(part) & 15) == 0) {
      reduce_rows_body_f4(part, nparts, len, out, accumulate, width, ldo, blk, nblk);
      return;
    }
  }
  __shared__ double red[8][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int64_t base = (int64_t)blk * 32; base < len; base += (int64_t)nblk * 32) {
    const int64_t i = base + lane;
    double acc = 0.0;
    if (i < len) {
      int b = w;
      for (; b + 24 < nparts; b += 32) {
        const double v0 = (double)part[(int64_t)b * len + i];
        const double v1 = (double)part[(int64_t)(b + 8) * len + i];
        const double v2 = (double)part[(int64_t)(b + 16) * len + i];
        const double v3 = (double)part[(int64_t)(b + 24) * len + i];
        acc += v0;
        acc += v1;
        acc += v2;
        acc += v3;
      }
      for (; b < nparts; b += 8) acc += (double)part[(int64_t)b * len + i];
    }
    red[w][lane] = acc;
    __syncthreads();
    if (w == 0 && i < len) {
      const int64_t oi = width > 0 ? (i / width) * ldo + i % width : i;
      double s = accumulate ? out[oi] : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u) s += red[u][lane];
      out[oi] = s;
    }
    __syncthreads();
  }
}

template <typename T>
__global__ void __launch_bounds__(256) k_reduce_rows(const T* __restrict__ part, int nparts, int64_t len,
                                                     double* __restrict__ out, int accumulate, int width = 0,
                                                     int ldo = 0) {
  reduce_rows_body<T>(part, nparts, len, out, accumulate, width, ldo, blockIdx.x, gridDim.x);
}

// One reduction per grid row y (batched segments): the task's part into its G.
__global__ void __launch_bounds__(256) k_reduce_rows_batch(const GramTask* __restrict__ tasks, int nparts,
                                                           int64_t len) {
  const GramTask t = tasks[blockIdx.y];
  reduce_rows_body<double>(t.part, nparts, len, t.G, 0, 0, 0, blockIdx.x, gridDim.x);
}

// One reduction per grid row y with its own part count (the segments of a
// batch); the sums have the bits of k_reduce_rows on the same partials.
template <typename T>
__global__ void __launch_bounds__(256) k_reduce_rows_sum(const SumTask* __restrict__ tasks, int64_t len) {
  const SumTask t = tasks[blockIdx.y];
  reduce_rows_body<T>(static_cast<const T*>(t.part), t.nparts, len, t.out, 0, 0, 0, blockIdx.x, gridDim.x);
}

cudaError_t launch_reduce_rows_batch(int part_dtype_f32, const SumTask* tasks, int ntasks, int64_t len,
                                     cudaStream_t st) {
  if (ntasks <= 0 || len <= 0) return cudaSuccess;
  const dim3 grid((unsigned)std::max<int64_t>(1, std::min<int64_t>((len + 31) / 32, 64)), (unsigned)ntasks);
  note_launches(1);
  if (part_dtype_f32)
    k_reduce_rows_sum<float><<<grid, 256, 0, st>>>(tasks, len);
  else
    k_reduce_rows_sum<double><<<grid, 256, 0, st>>>(tasks, len);
  return cudaGetLastError();
}

cudaError_t launch_reduce_rows_f64_batch(const GramTask* tasks, int ntasks, int nparts, int64_t len, cudaStream_t st,
                                         int num_sms) {
  if (ntasks <= 0) return cudaSuccess;
  const int gx = (int)std::max<int64_t>(1, std::min<int64_t>((len + 31) / 32, 16));
  note_launches(1);
  k_reduce_rows_batch<<<dim3((unsigned)gx, (unsigned)ntasks), 256, 0, st>>>(tasks, nparts, len);
  (void)num_sms;
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Value transform: convert to the compute type, optionally scale and clip.
//   mode 0: p = x
//   mode 1 (scale, centred):   p = clip((x - mu) * inv_std, +-clip) - c_g
//   mode 2 (scale, uncentred): p = min(x * inv_std, clip)
// c_g = clip(-mu * inv_std) is the value every stored zero takes, so the dense
// scaled matrix is P + 1 c^T with P on X's sparsity pattern.
// ---------------------------------------------------------------------------
// Four entries a thread, their loads in flight together.  With SMEM a block
// stages the three per-gene vectors (mode != 0): an entry's three lookups are
// random genes, and 32 of them cost the L1 a tag lookup per line touched
// (92M FP32 entries to scaled BF16: 234 us against 282).
template <typename InT, typename OutT, bool SMEM>
__global__ void __launch_bounds__(512) k_transform_values(const int32_t* __restrict__ idx, const InT* __restrict__ in,
                                                          OutT* __restrict__ out, int64_t nnz, int32_t g, int mode,
                                                          const double* __restrict__ mu,
                                                          const double* __restrict__ inv_std,
                                                          const double* __restrict__ cshift, double clip) {
  extern __shared__ double vec_sm[];  // [3][g]
  if (SMEM) {
    for (int i = threadIdx.x; i < g; i += blockDim.x) {
      vec_sm[i] = mu[i];
      vec_sm[g + i] = inv_std[i];
      vec_sm[2 * g + i] = cshift[i];
    }
    __syncthreads();
    mu = vec_sm;
    inv_std = vec_sm + g;
    cshift = vec_sm + 2 * g;
  }
  const int64_t nt = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < nnz; p += 4 * nt) {
    int32_t j[4];
    InT x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool ok = p + u * nt < nnz;
      j[u] = ok && mode != 0 ? __ldg(idx + p + u * nt) : 0;
      x[u] = ok ? in[p + u * nt] : InT();
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (p + u * nt < nnz) out[p + u * nt] = transform_value<InT, OutT>(x[u], j[u], mode, mu, inv_std, cshift, clip);
  }
}

// ---------------------------------------------------------------------------
// Row-block pointer table for the transposed product: for row i and gene
// block b, rbp[i * (nb + 1) + b] = offset (from indptr[i]) of the first stored
// entry of row i whose gene is >= b * gb.  Rows must be sorted by gene.
// ---------------------------------------------------------------------------
__global__ void k_row_block_ptr(const int64_t* __restrict__ indptr, const int32_t* __restrict__ idx,
                                int64_t n_obs, int nb, int gb, int32_t* __restrict__ rbp) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t row = warp; row < n_obs; row += nwarps) {
    const int64_t s = indptr[row], e = indptr[row + 1];
    for (int b = lane; b <= nb; b += 32) {
      const int32_t key = b * gb;
      int64_t lo = s, hi = e;  // first position with idx >= key
      while (lo < hi) {
        int64_t mid = (lo + hi) >> 1;
        if (__ldg(idx + mid) < key) lo = mid + 1; else hi = mid;
      }
      rbp[row * (nb + 1) + b] = (int32_t)(lo - s);
    }
  }
}

// ---------------------------------------------------------------------------
// Transposed product, CUDA-core path: block (chunk, b) owns genes
// [b*GB, (b+1)*GB) and the rows of one chunk, accumulates W_part[gene, :] in
// shared memory (FP32 shared atomics) and writes one partial.  Partials are
// reduced in fixed chunk order into FP64 by k_reduce_rows.
// Restates spmm_transpose_block (scx-accel/src/pca/cpu.rs:1282-1328).
// ---------------------------------------------------------------------------
template <int C, typename ValT, int GB>
__global__ void __launch_bounds__(512) k_spmm_t(const int64_t* __restrict__ indptr,
                                                const int32_t* __restrict__ idx,
                                                const ValT* __restrict__ val, int64_t n_obs,
                                                int32_t g, const int32_t* __restrict__ rbp, int nb,
                                                int64_t rows_per_chunk,
                                                const float* __restrict__ Q, int ldq,
                                                float* __restrict__ part) {
  constexpr int LD = 32 * C;
  extern __shared__ float acc[];  // [GB][LD]
  const int b = blockIdx.y;
  const int chunk = blockIdx.x;
  for (int i = threadIdx.x; i < GB * LD; i += blockDim.x) acc[i] = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int wid = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5;
  const int64_t r0 = (int64_t)chunk * rows_per_chunk;
  const int64_t r1 = min(n_obs, r0 + rows_per_chunk);
  const int g0 = b * GB;
  for (int64_t row = r0 + wid; row < r1; row += nw) {
    const int64_t base_row = indptr[row];
    const int32_t* rb = rbp + row * (nb + 1);
    const int64_t s = base_row + rb[b], e = base_row + rb[b + 1];
    if (s >= e) continue;
    float q[C];
#pragma unroll
    for (int c = 0; c < C; ++c) q[c] = __ldg(Q + row * (int64_t)ldq + lane + 32 * c);
    for (int64_t base = s; base < e; base += 32) {
      const int64_t p = base + lane;
      int32_t j = 0;
      float x = 0.f;
      if (p < e) {
        j = __ldg(idx + p) - g0;
        x = to_f32(val[p]);
      }
      const int cnt = (int)min((int64_t)32, e - base);
      for (int t = 0; t < cnt; ++t) {
        const int jt = __shfl_sync(0xffffffffu, j, t);
        const float xt = __shfl_sync(0xffffffffu, x, t);
        float* a = acc + jt * LD + lane;
#pragma unroll
        for (int c = 0; c < C; ++c) atomicAdd(a + 32 * c, xt * q[c]);
      }
    }
  }
  __syncthreads();
  float* out = part + (int64_t)chunk * g * LD;
  const int ng = min(GB, g - g0);
  for (int i = threadIdx.x; i < ng * LD; i += blockDim.x) out[(int64_t)g0 * LD + i] = acc[i];
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
template <typename ValT>
static cudaError_t col_stats_blocks_t(const int32_t* idx, const void* val, int64_t nnz, int32_t g, double* partial,
                                      int nparts, int part0, int count, cudaStream_t st, int num_sms) {
  if (count <= 0) return cudaSuccess;
  const ValT* v = static_cast<const ValT*>(val);
  const int32_t passes = std::max(1, (int32_t)(((int64_t)g + kStatsPassGenes - 1) / kStatsPassGenes));
  const int32_t pass_genes = (g + passes - 1) / passes;
  // one block per SM, of as few parts as spread them over all SMs
  const int sets = std::max(1, std::min(stats_sets(g), (count + num_sms - 1) / num_sms));
  const int ranges = sets >= kStatsOwn ? 1 : kStatsLeast / sets;
  const size_t smem = (size_t)sets * pass_genes * sizeof(double2);
  auto go = [&](auto kern) {
    if (smem > 48 * 1024)
      if (cudaError_t e = allow_smem(kern, smem); e != cudaSuccess) return e;
    note_launches(1);
    kern<<<(count + sets - 1) / sets, sets * ranges * 32, smem, st>>>(idx, v, nnz, g, pass_genes, ranges, nparts,
                                                                      part0, part0 + count, partial);
    return cudaGetLastError();
  };
  return ranges == 1 ? go(k_col_stats<ValT, false>) : go(k_col_stats<ValT, true>);
}

int64_t col_stats_block_begin(int64_t nnz, int nparts, int b) {
  const int64_t per = (nnz + nparts - 1) / nparts;
  return std::min(nnz, (int64_t)b * per);
}

cudaError_t launch_col_stats_blocks(int dtype, const int32_t* idx, const void* val, int64_t nnz, int32_t g,
                                    double* partial, int nparts, int part0, int count, cudaStream_t st,
                                    int num_sms) {
  switch (dtype) {
    case 0: return col_stats_blocks_t<float>(idx, val, nnz, g, partial, nparts, part0, count, st, num_sms);
    case 1: return col_stats_blocks_t<__nv_bfloat16>(idx, val, nnz, g, partial, nparts, part0, count, st, num_sms);
    default: return col_stats_blocks_t<__half>(idx, val, nnz, g, partial, nparts, part0, count, st, num_sms);
  }
}

cudaError_t launch_col_stats_reduce(const double* partial, int nparts, int32_t g, double* out, cudaStream_t st,
                                    int num_sms, int accumulate) {
  // a block per 32 sums, as many as there are (16 blocks, eight turns each, took 53 us at 2,000 genes, now 9)
  k_reduce_rows<double><<<grid_for(2 * g, 32, num_sms), 256, 0, st>>>(partial, nparts, 2 * (int64_t)g, out,
                                                                      accumulate);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_col_stats(int dtype, const int32_t* idx, const void* val, int64_t nnz,
                             int32_t g, double* partial, int nparts, double* out,
                             cudaStream_t st, int num_sms, int accumulate) {
  cudaError_t e = launch_col_stats_blocks(dtype, idx, val, nnz, g, partial, nparts, 0, nparts, st, num_sms);
  if (e != cudaSuccess) return e;
  return launch_col_stats_reduce(partial, nparts, g, out, st, num_sms, accumulate);
}

template <typename InT, typename OutT>
static cudaError_t transform_io(const int32_t* idx, const void* in, void* out, int64_t nnz, int32_t g, int mode,
                                const double* mu, const double* inv_std, const double* cshift, double clip,
                                cudaStream_t st, int num_sms) {
  auto go = [&](auto kern, size_t smem, int blocks_per_sm) {
    if (smem > 48 * 1024)
      if (cudaError_t e = allow_smem(kern, smem); e != cudaSuccess) return e;
    note_launches(1);
    kern<<<grid_for(nnz, 2048, num_sms, blocks_per_sm), 512, smem, st>>>(idx, static_cast<const InT*>(in),
                                                                         static_cast<OutT*>(out), nnz, g, mode, mu,
                                                                         inv_std, cshift, clip);
    return cudaGetLastError();
  };
  // the vectors in shared memory while two blocks of an SM can hold them
  const size_t smem = 3 * sizeof(double) * (size_t)g;
  if (mode != 0 && smem <= 100 * 1024)
    return go(k_transform_values<InT, OutT, true>, smem, (int)std::min<size_t>(4, 200 * 1024 / smem));
  return go(k_transform_values<InT, OutT, false>, 0, 4);
}

template <typename InT>
static cudaError_t transform_in(int out_dtype, const int32_t* idx, const void* in, void* out, int64_t nnz, int32_t g,
                                int mode, const double* mu, const double* inv_std, const double* cshift, double clip,
                                cudaStream_t st, int num_sms) {
  switch (out_dtype) {
    case 0: return transform_io<InT, float>(idx, in, out, nnz, g, mode, mu, inv_std, cshift, clip, st, num_sms);
    case 1:
      return transform_io<InT, __nv_bfloat16>(idx, in, out, nnz, g, mode, mu, inv_std, cshift, clip, st, num_sms);
    default: return transform_io<InT, __half>(idx, in, out, nnz, g, mode, mu, inv_std, cshift, clip, st, num_sms);
  }
}

cudaError_t launch_transform_values(int in_dtype, int out_dtype, const int32_t* idx, const void* in, void* out,
                                    int64_t nnz, int32_t g, int mode, const double* mu, const double* inv_std,
                                    const double* cshift, double clip, cudaStream_t st, int num_sms) {
  if (nnz == 0) return cudaSuccess;
  switch (in_dtype) {
    case 0: return transform_in<float>(out_dtype, idx, in, out, nnz, g, mode, mu, inv_std, cshift, clip, st, num_sms);
    case 1:
      return transform_in<__nv_bfloat16>(out_dtype, idx, in, out, nnz, g, mode, mu, inv_std, cshift, clip, st, num_sms);
    default: return transform_in<__half>(out_dtype, idx, in, out, nnz, g, mode, mu, inv_std, cshift, clip, st, num_sms);
  }
}

cudaError_t launch_row_block_ptr(const int64_t* indptr, const int32_t* idx, int64_t n, int nb,
                                 int gb, int32_t* rbp, cudaStream_t st, int num_sms) {
  if (n == 0) return cudaSuccess;
  note_launches(1);
  k_row_block_ptr<<<grid_for(n * 32, 256, num_sms, 8), 256, 0, st>>>(indptr, idx, n, nb, gb, rbp);
  return cudaGetLastError();
}

template <int C, typename ValT>
static cudaError_t spmm_t_c(const int64_t* indptr, const int32_t* idx, const void* val, int64_t n,
                            int32_t g, const int32_t* rbp, int nb, int nchunks,
                            int64_t rows_per_chunk, const float* Q, int ldq, float* part,
                            cudaStream_t st) {
  constexpr int GB = kTransposeGeneBlock;
  size_t smem = (size_t)GB * 32 * C * sizeof(float);
  auto kern = k_spmm_t<C, ValT, GB>;
  if (cudaError_t e = allow_smem(kern, smem); e != cudaSuccess) return e;
  dim3 grid(nchunks, nb);
  note_launches(1);
  kern<<<grid, 512, smem, st>>>(indptr, idx, static_cast<const ValT*>(val), n, g, rbp, nb,
                                rows_per_chunk, Q, ldq, part);
  return cudaGetLastError();
}

template <typename ValT>
static cudaError_t spmm_t_t(int ld, const int64_t* indptr, const int32_t* idx, const void* val,
                            int64_t n, int32_t g, const int32_t* rbp, int nb, int nchunks,
                            int64_t rpc, const float* Q, float* part, cudaStream_t st) {
  switch (ld) {
    case 32: return spmm_t_c<1, ValT>(indptr, idx, val, n, g, rbp, nb, nchunks, rpc, Q, ld, part, st);
    case 64: return spmm_t_c<2, ValT>(indptr, idx, val, n, g, rbp, nb, nchunks, rpc, Q, ld, part, st);
    case 96: return spmm_t_c<3, ValT>(indptr, idx, val, n, g, rbp, nb, nchunks, rpc, Q, ld, part, st);
    default: return spmm_t_c<4, ValT>(indptr, idx, val, n, g, rbp, nb, nchunks, rpc, Q, ld, part, st);
  }
}

cudaError_t launch_spmm_t(int dtype, int ld, const int64_t* indptr, const int32_t* idx,
                          const void* val, int64_t n, int32_t g, const int32_t* rbp, int nb,
                          int nchunks, int64_t rows_per_chunk, const float* Q, float* part,
                          cudaStream_t st) {
  switch (dtype) {
    case 0: return spmm_t_t<float>(ld, indptr, idx, val, n, g, rbp, nb, nchunks, rows_per_chunk, Q, part, st);
    case 1: return spmm_t_t<__nv_bfloat16>(ld, indptr, idx, val, n, g, rbp, nb, nchunks, rows_per_chunk, Q, part, st);
    default: return spmm_t_t<__half>(ld, indptr, idx, val, n, g, rbp, nb, nchunks, rows_per_chunk, Q, part, st);
  }
}

cudaError_t launch_reduce_rows_f32(const float* part, int nparts, int64_t len, double* out,
                                   int accumulate, cudaStream_t st, int num_sms) {
  note_launches(1);
  k_reduce_rows<float><<<grid_for(len, 32, num_sms), 256, 0, st>>>(part, nparts, len, out, accumulate);
  return cudaGetLastError();
}

cudaError_t launch_reduce_panel_f32(const float* part, int nparts, int64_t rows, int width, double* out, int ldo,
                                    cudaStream_t st, int num_sms) {
  const int64_t len = rows * width;
  note_launches(1);
  k_reduce_rows<float><<<grid_for(len, 32, num_sms), 256, 0, st>>>(part, nparts, len, out, 0, width, ldo);
  return cudaGetLastError();
}

cudaError_t launch_reduce_rows_f64(const double* part, int nparts, int64_t len, double* out,
                                   int accumulate, cudaStream_t st, int num_sms) {
  note_launches(1);
  k_reduce_rows<double><<<grid_for(len, 32, num_sms), 256, 0, st>>>(part, nparts, len, out, accumulate);
  return cudaGetLastError();
}

}  // namespace scx
