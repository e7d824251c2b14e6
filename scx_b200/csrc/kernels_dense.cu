// Dense-side kernels of the randomized PCA: tall Gram matrices (FP64
// accumulation), Cholesky + triangular inverse and the symmetric Jacobi
// eigensolver (single block, FP64), right-multiplications by small k x k
// factors, the Rayleigh-Ritz finish, embeddings and the seeded Gaussian test
// matrix.
//
// The small factorisations replace cuSOLVER potrf/trsm (scx-gpu/src/
// cusolver.rs:297-409) and the host faer thin SVD of B (scx-gpu/src/
// gpu_pca.rs:593-611): all of them stay on the device in FP64.
#include <algorithm>

#include "common.cuh"
#include "launch.h"

namespace scx {

// ---------------------------------------------------------------------------
// Gram partials in FP64.  Block b owns a contiguous row range; its warps take
// four rows at a time through the FP64 matrix instruction (8 x 8 outputs, four
// rows deep).  The instruction's two operands have the same layout for a Gram,
// lane l holding row l % 4 of one of the block's eight columns l / 4, so the
// four rows of all columns are LD / 8 registers per lane, loaded straight from
// memory, that serve every output tile on and above the diagonal as either
// operand.  Products of float inputs are exact in FP64; sums are FP64.
//
// Outputs on the CUDA cores are bound by the shared-memory reads of the rows
// (eight reads per ten FMAs and thread at ld 64: 178 us for 250,000 rows, 34 at
// the FP64 rate); here nothing is read twice.  Measured: 43 us for 250,000 rows
// at ld 64 (at 10,000 rows 6.9 against 11.2), 88 for 120,000 at ld 128 (137 before).
//
// A warp holds the tiles it owns in registers: all 36 at ld 64; at ld 96 and 128
// two and four warps share the same rows, warp w of W taking the tile rows i
// with i mod 2 W equal to w or 2 W - 1 - w, which gives each the same number of
// tiles.  The row groups of a block are added pairwise at the end.
// Column (i, m) of tile row i, lane row m is V (i / V) 8 + V m + i % V with
// V values per 16-byte load.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

constexpr int kGramWarps = 8;
template <int LD> constexpr int gram_split() { return LD <= 64 ? 1 : LD == 96 ? 2 : 4; }  // warps sharing rows
template <int LD> constexpr int gram_tiles() {  // tiles of one of them
  constexpr int NB = LD / 8;
  return NB * (NB + 1) / 2 / gram_split<LD>();
}
template <int LD> constexpr size_t gram_smem() {  // the block's sum; the row groups' tiles before it
  constexpr size_t sum = sizeof(double) * (LD * LD + LD);
  constexpr size_t tiles = sizeof(double) * ((size_t)kGramWarps / 2 * gram_tiles<LD>() * 64 + kGramWarps * LD);
  return sum > tiles ? sum : tiles;
}
// Whether warp `w` of W owns tile row i.
__host__ __device__ constexpr bool gram_owns(int i, int w, int W) { return i % (2 * W) == w || i % (2 * W) == 2 * W - 1 - w; }

// The block's barrier, met by its warps from different copies of gram_warp.
__device__ __forceinline__ void gram_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kGramWarps * 32) : "memory"); }

template <typename T, int LD, int SW>  // SW: which of the warps that share rows
__device__ __forceinline__ void gram_warp(const T* __restrict__ A, int64_t r0, int64_t r1, double* __restrict__ part,
                                          double* sm) {
  constexpr int NB = LD / 8, W = gram_split<LD>(), NT = gram_tiles<LD>(), G = kGramWarps / W;
  constexpr int V = 16 / (int)sizeof(T);  // values per 16-byte load
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, group = warp / W;
  const int kr = lane & 3, m = lane >> 2;
  double acc[NT][2];
#pragma unroll
  for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = 0.0;
  double csum[NB / W];
#pragma unroll
  for (int i = 0; i < NB / W; ++i) csum[i] = 0.0;
  T nx[NB];
  auto load = [&](int64_t r) {
#pragma unroll
    for (int p = 0; p < NB / V; ++p) {
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (r + kr < r1) v = *reinterpret_cast<const uint4*>(A + (r + kr) * LD + p * (8 * V) + V * m);
      *reinterpret_cast<uint4*>(nx + p * V) = v;
    }
  };
  load(r0 + 4 * group);
  for (int64_t r = r0 + 4 * group; r < r1; r += 4 * G) {
    double f[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) f[i] = (double)nx[i];
    load(r + 4 * G);
    int t = 0, s = 0;
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      if (!gram_owns(i, SW, W)) continue;
      csum[s++] += f[i];
#pragma unroll
      for (int j = i; j < NB; ++j) mma_f64(acc[t++], f[i], f[j]);
    }
  }
  // column sums: over the four row lanes, then over the groups in order
#pragma unroll
  for (int s = 0; s < NB / W; ++s) {
    csum[s] += __shfl_xor_sync(0xffffffffu, csum[s], 1);
    csum[s] += __shfl_xor_sync(0xffffffffu, csum[s], 2);
  }
  auto col = [&](int i, int mm) { return i / V * (8 * V) + V * mm + i % V; };
  // shared memory: tiles [G / 2 row groups][W][NT][32 lanes], then the sums
  double* sums = sm + (size_t)(G / 2) * W * NT * 64;  // [group][LD]
  {
    int s = 0;
#pragma unroll
    for (int i = 0; i < NB; ++i)
      if (gram_owns(i, SW, W)) {
        if (kr == 0) sums[group * LD + col(i, m)] = csum[s];
        ++s;
      }
  }
  // the upper half of the row groups hands its tiles to the lower half, until one is left
#pragma unroll
  for (int half = G / 2; half > 0; half /= 2) {
    double2* at = reinterpret_cast<double2*>(sm) + ((size_t)(group % half) * W + SW) * NT * 32 + lane;
    if (group >= half && group < 2 * half) {
#pragma unroll
      for (int t = 0; t < NT; ++t) at[t * 32] = make_double2(acc[t][0], acc[t][1]);
    }
    gram_barrier();
    if (group < half) {
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const double2 v = at[t * 32];
        acc[t][0] += v.x;
        acc[t][1] += v.y;
      }
    }
    gram_barrier();
  }
  double cs = 0.0;
  if (threadIdx.x < LD)
    for (int g = 0; g < G; ++g) cs += sums[g * LD + threadIdx.x];
  gram_barrier();  // the tiles and the sums are read
  if (group == 0) {
    int t = 0;
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      if (!gram_owns(i, SW, W)) continue;
#pragma unroll
      for (int j = i; j < NB; ++j) {
        const int a = col(i, m);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int b = col(j, 2 * kr + e);
          sm[a * LD + b] = acc[t][e];
          if (j != i) sm[b * LD + a] = acc[t][e];
        }
        ++t;
      }
    }
  }
  if (threadIdx.x < LD) sm[LD * LD + threadIdx.x] = cs;
  gram_barrier();
  for (int t = threadIdx.x; t < LD * LD + LD; t += kGramWarps * 32) part[t] = sm[t];
}

template <typename T, int LD>
__device__ __forceinline__ void gram_body(const T* __restrict__ A, int64_t n, double* __restrict__ part, int b,
                                          int nb) {
  extern __shared__ __align__(16) double gram_sm[];
  const int64_t per = (n + nb - 1) / nb;
  const int64_t r0 = min(n, (int64_t)b * per), r1 = min(n, r0 + per);
  double* out = part + (int64_t)b * (LD * LD + LD);
  // (the block's barriers are met by every warp in the same order, whatever its share)
  constexpr int W = gram_split<LD>();
  const int sw = (int)(threadIdx.x >> 5) % W;
  if (sw == 0) gram_warp<T, LD, 0>(A, r0, r1, out, gram_sm);
  if constexpr (W >= 2) {
    if (sw == 1) gram_warp<T, LD, 1>(A, r0, r1, out, gram_sm);
  }
  if constexpr (W >= 4) {
    if (sw == 2) gram_warp<T, LD, 2>(A, r0, r1, out, gram_sm);
    if (sw == 3) gram_warp<T, LD, 3>(A, r0, r1, out, gram_sm);
  }
}

template <typename T, int LD>
__global__ void __launch_bounds__(kGramWarps * 32, 1) k_gram(const T* __restrict__ A, int64_t n,
                                                             double* __restrict__ part) {
  gram_body<T, LD>(A, n, part, blockIdx.x, gridDim.x);
}

// One FP64 matrix per grid row y (batched segments): partials into the task's part.
template <int LD>
__global__ void __launch_bounds__(kGramWarps * 32, 1) k_gram_batch(const GramTask* __restrict__ tasks, int64_t n) {
  const GramTask t = tasks[blockIdx.y];
  gram_body<double, LD>(t.A, n, t.part, blockIdx.x, gridDim.x);
}

template <int LD, typename Kernel, typename... Args>
static cudaError_t gram_go(Kernel kern, dim3 grid, cudaStream_t st, Args... args) {
  constexpr size_t smem = gram_smem<LD>();
  if (smem > 48 * 1024)
    if (cudaError_t e = allow_smem(kern, smem); e != cudaSuccess) return e;
  note_launches(1);
  kern<<<grid, kGramWarps * 32, smem, st>>>(args...);
  return cudaGetLastError();
}

cudaError_t launch_gram_f64_batch(const GramTask* tasks, int ntasks, int64_t n, int ld, int nparts,
                                  cudaStream_t st, int num_sms) {
  if (ntasks <= 0) return cudaSuccess;
  const dim3 grid((unsigned)nparts, (unsigned)ntasks);
  cudaError_t e = cudaErrorInvalidValue;
  switch (ld) {
    case 32: e = gram_go<32>(k_gram_batch<32>, grid, st, tasks, n); break;
    case 64: e = gram_go<64>(k_gram_batch<64>, grid, st, tasks, n); break;
    case 96: e = gram_go<96>(k_gram_batch<96>, grid, st, tasks, n); break;
    case 128: e = gram_go<128>(k_gram_batch<128>, grid, st, tasks, n); break;
    default: break;
  }
  if (e != cudaSuccess) return e;
  return launch_reduce_rows_f64_batch(tasks, ntasks, nparts, (int64_t)ld * ld + ld, st, num_sms);
}

template <typename T>
static cudaError_t gram_t(const T* A, int64_t n, int ld, double* part, int nparts, cudaStream_t st) {
  if (ld > kMaxK) {
    if constexpr (sizeof(T) == 4) return launch_gram_wide_f32(reinterpret_cast<const float*>(A), n, ld, part, nparts, st);
    else return launch_gram_wide_f64(reinterpret_cast<const double*>(A), n, ld, part, nparts, st);
  }
  const dim3 grid((unsigned)nparts);
  switch (ld) {
    case 32: return gram_go<32>(k_gram<T, 32>, grid, st, A, n, part);
    case 64: return gram_go<64>(k_gram<T, 64>, grid, st, A, n, part);
    case 96: return gram_go<96>(k_gram<T, 96>, grid, st, A, n, part);
    default: return gram_go<128>(k_gram<T, 128>, grid, st, A, n, part);
  }
}

cudaError_t launch_gram_f32(const float* A, int64_t n, int ld, double* part, int nparts,
                            cudaStream_t st) {
  return gram_t<float>(A, n, ld, part, nparts, st);
}
cudaError_t launch_gram_f64(const double* A, int64_t n, int ld, double* part, int nparts,
                            cudaStream_t st) {
  return gram_t<double>(A, n, ld, part, nparts, st);
}

// ---------------------------------------------------------------------------
// Cholesky of the leading k x k block of G (ld x ld) and the inverse of its
// factor, one block of 256 threads.  A pivot j fails when its Schur complement
// d_j <= tau * G_jj (the column is numerically dependent on the previous ones)
// or is not finite.  With shift_on_fail the factorisation restarts once on
// G + s I, s = 10 tau max_j G_jj, which always succeeds on finite input.  With
// CLAMP (the eigensolver's factor) no pivot fails: one below 1e-15 of the
// largest diagonal, or 1e-300, is set there.
//
// Symmetric Gaussian elimination of the augmented matrix [A | I]: step j
// subtracts (A_ja / d_j) times row j from every row a > j, which turns A's
// upper triangle into D L^T and the identity into X = L^{-1} (unit lower
// triangular), where A = L D L^T.  Then R = D^{1/2} L^T and
// R^{-1} = X^T D^{-1/2}: R_jc = A_jc / sqrt(d_j), R^{-1}_ca = X_ac / sqrt(d_a).
// Every matrix entry lives in a register of its owner, thread (ty, tx) owning
// rows ty + 16 u and columns tx + 16 v; one register holds A_ac above the
// diagonal (c >= a) or X_ac below it.
//
// What bounds it is the chain of pivots: each needs a reciprocal and one
// multiply-add of the pivot before it.  One pivot per block barrier cost 1,300
// clocks (51 us at k = 60, 170 us at k = 110), so the rows go in panels of
// eight: a panel's rows are handed to a few warps that eliminate inside the
// panel without a barrier, one column per lane, and then all threads take the
// panel's eight steps at once on their entries.  Measured: 17 us at k = 60, 59 us at k = 110.
// ---------------------------------------------------------------------------
constexpr int kCholThreads = 256;
constexpr int kPanelRows = 8;

// 1 / x for normal x: the hardware's approximation and two Newton steps
// (y <- y (2 - x y), each doubling the correct bits).
__device__ __forceinline__ double rcp_fast(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}
// 1 / sqrt(x) for normal x > 0, in the same way (y <- y (3 - x y^2) / 2).
__device__ __forceinline__ double rsqrt_fast(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double h = 0.5 * x;
  y = fma(y, fma(-h * y, y, 0.5), y);
  return fma(y, fma(-h * y, y, 0.5), y);
}

template <int KP>
constexpr size_t chol_smem() {  // factored rows [KP][KP + 1]; a panel's rows and multipliers, X in its own columns
  return sizeof(double) * ((size_t)KP * (KP + 1) + 2 * kPanelRows * KP + (size_t)kPanelRows * (KP + 1));
}

// With `tasks` set (CholTask, or JacobiTask with CLAMP), block b factors the
// matrix of tasks[b] (many segments' factorisations in one launch, one block
// each) and the pointer arguments are ignored.
template <int KP, bool CLAMP>
__global__ void __launch_bounds__(kCholThreads) k_cholesky(const double* __restrict__ G, int k, int ld, double tau,
                                                           int shift_on_fail, double* __restrict__ R,
                                                           double* __restrict__ Rinv, float* __restrict__ Rinv_f,
                                                           int* __restrict__ status, const void* tasks) {
  if (tasks && CLAMP) {
    const JacobiTask t = static_cast<const JacobiTask*>(tasks)[blockIdx.x];
    G = t.C;
    R = t.evecs + (size_t)ld * ld;
    Rinv = R + (size_t)ld * ld;
  } else if (tasks) {
    const CholTask t = static_cast<const CholTask*>(tasks)[blockIdx.x];
    G = t.G;
    R = t.R;
    Rinv = t.Rinv;
    Rinv_f = t.Rinv_f;
    status = t.status;
  }
  constexpr int U = KP / 16, NT = kCholThreads, PR = kPanelRows, FS = KP + 1;
  extern __shared__ double chol_sm[];
  double* F = chol_sm;          // [KP][FS]: row j of D L^T (c >= j) and of X (c < j), once final
  double* P = F + KP * FS;      // [PR][KP]: the panel's rows as their owners left them
  double* M = P + PR * KP;      // [PR][KP]: multipliers A_ja / d_j
  double* T = M + PR * KP;      // [PR][FS]: X in the panel's own columns
  __shared__ double piv[KP], dg[KP];
  __shared__ double maxdiag_s;
  __shared__ int fail_s;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, warp = tid >> 5;
  for (int j = tid; j < k; j += NT) dg[j] = G[(int64_t)j * ld + j];
  __syncthreads();
  if (tid < 32) {
    double m = 0.0;
    for (int j = tid; j < k; j += 32) m = fmax(m, dg[j]);
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (tid == 0) maxdiag_s = m;
  }
  double shift = 0.0;
  for (int attempt = 0; attempt < 2; ++attempt) {
    double val[U][U];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int v = 0; v < U; ++v) {
        const int a = ty + 16 * u, c = tx + 16 * v;
        double x = 0.0;  // X starts as the identity; its unit diagonal is implicit
        if (c >= a && c < k) x = G[(int64_t)a * ld + c] + (a == c ? shift : 0.0);
        val[u][v] = x;
      }
    if (tid == 0) fail_s = -1;
    __syncthreads();
    const double floor_d = fmax(1e-15 * maxdiag_s, 1e-300);
    for (int j0 = 0; j0 < k; j0 += PR) {
      // the panel's rows, from their owners
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int a = ty + 16 * u;
        if ((unsigned)(a - j0) < (unsigned)PR) {
#pragma unroll
          for (int v = 0; v < U; ++v) P[(a - j0) * KP + tx + 16 * v] = val[u][v];
        }
      }
      __syncthreads();
      // elimination inside the panel, a column per lane: the panel's own columns
      // of X, every column outside the panel, the panel's own columns of A.  Each
      // lane repeats the 8 x 8 diagonal block's steps beside its column's, so
      // nothing is exchanged and the chain of a step is a reciprocal, a product
      // and a multiply-add.
      const int i = tid;
      if (warp < (KP + PR + 31) / 32) {
        int c = i - PR;
        if (c >= j0) c += PR;
        const bool xdiag = i < PR, adiag = i >= KP && i < KP + PR;
        if (xdiag) c = j0 + i;
        if (adiag) c = j0 + i - KP;
        const bool there = i < KP + PR;
        const int steps = min(PR, k - j0);
        double x[PR], D[PR][PR], di[PR], least[PR];
#pragma unroll
        for (int r = 0; r < PR; ++r) {
          x[r] = xdiag ? (r == i ? 1.0 : 0.0) : there ? P[r * KP + c] : 0.0;
#pragma unroll
          for (int q = r; q < PR; ++q) D[r][q] = P[r * KP + j0 + q];
          if (r >= steps) D[r][r] = 1.0;  // rows past the matrix: zero but for the pivot
          least[r] = CLAMP ? floor_d : attempt == 0 && r < steps ? fmax(tau * (dg[j0 + r] + shift), 0.0) : 0.0;
        }
        // No branch on a pivot: one that fails is noted, and what follows from it
        // is not used.  (Every lane of every warp sees the same pivots.)
        unsigned bad = 0;
#pragma unroll
        for (int r = 0; r < PR; ++r) {
          double d = D[r][r];
          if (CLAMP) d = d > floor_d ? d : floor_d;
          else if (!(d > least[r] && d < INFINITY)) bad |= 1u << r;
          di[r] = rcp_fast(d);
          D[r][r] = d;
#pragma unroll
          for (int q = r + 1; q < PR; ++q) {
            const double m = -(D[r][q] * di[r]);
#pragma unroll
            for (int s = q; s < PR; ++s) D[q][s] = fma(m, D[r][s], D[q][s]);
            x[q] = fma(m, x[r], x[q]);
          }
        }
        const int fail = bad ? j0 + __ffs(bad) - 1 : -1;
        if (tid == 0) {
#pragma unroll
          for (int r = 0; r < PR; ++r)
            if (r < steps) piv[j0 + r] = D[r][r];
        }
        if (fail >= 0) {
          if (tid == 0) fail_s = fail;
        } else if (xdiag) {
#pragma unroll
          for (int r = 0; r < PR; ++r) {
            T[r * FS + c] = x[r];
            if (r > i) F[(j0 + r) * FS + c] = x[r];
          }
        } else if (adiag) {
#pragma unroll
          for (int r = 0; r < PR; ++r)
            if (r <= i - KP) F[(j0 + r) * FS + c] = x[r];
        } else if (there) {
#pragma unroll
          for (int r = 0; r < PR; ++r) {
            F[(j0 + r) * FS + c] = x[r];
            M[r * KP + c] = x[r] * di[r];
          }
        }
      }
      __syncthreads();
      if (fail_s >= 0) break;
      // the panel's steps on the rows behind it: A's entries (c >= a), and X's
      // up to the panel's last column; four blocks of rows at a time
      const int pe = j0 + PR;
      if (pe < k) {
        const double* src[U];
#pragma unroll
        for (int v = 0; v < U; ++v) {
          const int c = tx + 16 * v;
          src[v] = (unsigned)(c - j0) < (unsigned)PR ? T + c : F + j0 * FS + c;
        }
#pragma unroll
        for (int ub = 0; ub < U; ub += 4) {
          if (16 * (ub + 4) <= pe) continue;
          double s[4][U] = {};
#pragma unroll
          for (int r = 0; r < PR; ++r) {
            double t[U];
#pragma unroll
            for (int v = 0; v < U; ++v) t[v] = src[v][r * FS];
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              if (16 * (ub + w + 1) <= pe) continue;
              const double m = M[r * KP + ty + 16 * (ub + w)];
#pragma unroll
              for (int v = 0; v < U; ++v) s[w][v] = fma(m, t[v], s[w][v]);
            }
          }
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            const int a = ty + 16 * (ub + w);
#pragma unroll
            for (int v = 0; v < U; ++v) {
              const int c = tx + 16 * v;
              if (a >= pe && (c >= a || c < pe)) val[ub + w][v] -= s[w][v];
            }
          }
        }
      }
    }
    __syncthreads();
    const int fail = fail_s;
    if (fail < 0) break;
    if (!shift_on_fail || attempt == 1) {
      if (tid == 0) status[0] = -(fail + 1);
      // Leave well-defined (identity) factors so downstream kernels stay finite.
      for (int t = tid; t < ld * ld; t += NT) {
        const int r = t / ld, c = t % ld;
        const double v = (r == c && r < k) ? 1.0 : 0.0;
        R[t] = v;
        Rinv[t] = v;
        Rinv_f[t] = (float)v;
      }
      return;
    }
    if (tid == 0) status[0] += 1;
    shift = 10.0 * tau * fmax(maxdiag_s, 1e-300);
    __syncthreads();
  }
  // 1 / sqrt(d_j), then R_jc = A_jc / sqrt(d_j) and R^{-1}_ca = X_ac / sqrt(d_a), c <= a
  if (tid < k) {
    const double d = piv[tid];
    dg[tid] = rsqrt_fast(d);
  }
  __syncthreads();
  for (int t = tid; t < ld * ld; t += NT) {
    const int r = t / ld, c = t - r * ld;
    double up = 0.0, inv = 0.0;
    if (c < k && r <= c) {
      up = r == c && CLAMP ? piv[r] * dg[r] : F[r * FS + c] * dg[r];
      inv = (r == c ? 1.0 : F[c * FS + r]) * dg[c];
    }
    R[t] = up;
    Rinv[t] = inv;
    if (!CLAMP) Rinv_f[t] = (float)inv;
  }
}

template <bool CLAMP>
static cudaError_t chol_go(const double* G, int k, int ld, double tau, int shift_on_fail, double* R, double* Rinv,
                           float* Rinv_f, int* status, const void* tasks, int nblocks, cudaStream_t st) {
  if (k > kMaxK || ld > kMaxK) return cudaErrorInvalidValue;
  note_launches(1);
  auto go = [&](auto kern, size_t smem) {
    if (cudaError_t e = allow_smem(kern, smem); e != cudaSuccess) return e;
    kern<<<nblocks, kCholThreads, smem, st>>>(G, k, ld, tau, shift_on_fail, R, Rinv, Rinv_f, status, tasks);
    return cudaGetLastError();
  };
  if (k <= 64) return go(k_cholesky<64, CLAMP>, chol_smem<64>());
  return go(k_cholesky<128, CLAMP>, chol_smem<128>());
}

cudaError_t launch_cholesky(const double* G, int k, int ld, double tau, int shift_on_fail,
                            double* R, double* Rinv, float* Rinv_f, int* status, cudaStream_t st) {
  if (ld > kMaxK) return launch_cholesky_wide(G, k, ld, tau, shift_on_fail, R, Rinv, Rinv_f, status, st);
  return chol_go<false>(G, k, ld, tau, shift_on_fail, R, Rinv, Rinv_f, status, nullptr, 1, st);
}

cudaError_t launch_cholesky_batch(const CholTask* tasks, int ntasks, int k, int ld, double tau, int shift_on_fail,
                                  cudaStream_t st) {
  if (ntasks <= 0) return cudaSuccess;
  return chol_go<false>(nullptr, k, ld, tau, shift_on_fail, nullptr, nullptr, nullptr, nullptr, tasks, ntasks, st);
}

// ---------------------------------------------------------------------------
// Tall x small: Out[i, :cnt] = In[i, :K] * M (K x cnt), 128-row tiles.
// M (zero-padded to OUTB columns) sits in shared memory; row tiles are
// double-buffered in shared memory by cp.async (16-byte copies, rows padded
// by 4 floats), so the next tile streams in while this one is multiplied.
// Thread (ty, tx) of the 16 x 16 grid computes rows ty + 16 i (i < 8) at
// columns 64 h + 4 tx + (0..3): per four k-steps it reads eight float4 of
// its rows (two distinct addresses per warp: broadcast) and 4 OUTB/64
// float4 of M, for 128 OUTB/64 FMAs.  A block loads a tile before it writes
// any of its rows, and only ever writes its own tiles, so Out may alias In.
// Optionally writes the 16-bit image of Out in the same pass: row stride
// 2 ldo, column 2 j = hi = round16(x), 2 j + 1 = round16(x - hi) (fmt 1 =
// bf16, 0 = f16).
// ---------------------------------------------------------------------------
constexpr int kTallRows = 128;

__device__ __forceinline__ void split16(float x, int fmt, uint16_t& h, uint16_t& l) {
  if (fmt) {
    const __nv_bfloat16 b = __float2bfloat16_rn(x);
    h = __bfloat16_as_ushort(b);
    l = __bfloat16_as_ushort(__float2bfloat16_rn(x - __bfloat162float(b)));
  } else {
    const __half b = __float2half_rn(x);
    h = __half_as_ushort(b);
    l = __half_as_ushort(__float2half_rn(x - __half2float(b)));
  }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// The matrices of one tall right-multiplication launch.  A task is one
// matrix: In (n x ldi, rows in tiles of 128), Out, the optional image, and M;
// tile0 numbers its first tile in the launch.
// TallOne: one matrix, block b takes the tiles b, b + nb, ...
// TallBatch: every matrix of a batch; block b takes a contiguous range of the
// launch's tiles, so it restages M only where its range crosses into the
// next matrix.
struct TallOne {
  TallTask t;
  int64_t n_tiles;
  __device__ int64_t first() const { return blockIdx.x; }
  __device__ int64_t next(int64_t tile) const { return tile + gridDim.x; }
  __device__ bool valid(int64_t tile) const { return tile < n_tiles; }
  __device__ int task_of(int64_t) const { return 0; }
  __device__ TallTask task(int) const { return t; }
};
struct TallBatch {
  const TallTask* tasks;
  int ntasks;
  int64_t begin, end;  // this block's tiles
  __device__ int64_t first() const { return begin; }
  __device__ int64_t next(int64_t tile) const { return tile + 1; }
  __device__ bool valid(int64_t tile) const { return tile < end; }
  __device__ int task_of(int64_t tile) const {  // the last task whose first tile is <= tile
    int lo = 0, hi = ntasks - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (tasks[mid].tile0 <= tile) lo = mid;
      else hi = mid - 1;
    }
    return lo;
  }
  __device__ TallTask task(int q) const { return tasks[q]; }
};
__device__ __forceinline__ TallBatch tall_batch(const TallTask* tasks, int ntasks, int64_t total_tiles) {
  return TallBatch{tasks, ntasks, (int64_t)blockIdx.x * total_tiles / gridDim.x,
                   (int64_t)(blockIdx.x + 1) * total_tiles / gridDim.x};
}

// NT threads, thread (ty, tx) of NT / 16 x 16 taking rows ty + NT / 16 i and
// four columns of every 64.  UPPER: M is upper triangular, so columns 64 h ..
// need its rows below 64 (h + 1) only.  At OUTB 128 one block fills an SM's
// shared memory and needs 16 warps to keep the FMAs fed (120,000 x 128 by
// 128 x 128: 256 threads 138 us; 512 threads 123, and 112 with an upper M).
template <int OUTB, int NT, bool UPPER, class Src>
__device__ __forceinline__ void tall_mm_body(const Src& src, int K, int ldi, int ldm, int cnt, int ldo, int fmt) {
  constexpr int H = OUTB / 64;
  constexpr int RS = NT / 16, RPT = kTallRows / RS;  // rows per thread
  extern __shared__ __align__(16) float sm_f[];
  const int KP = K + 4;
  float* Ms = sm_f;  // [K][OUTB]
  float* T0 = sm_f + K * OUTB;
  float* T1 = T0 + kTallRows * KP;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int k4 = K >> 2;
  const bool vec_out = ((cnt & 3) == 0) && ((ldo & 3) == 0);

  auto issue = [&](int64_t tile, float* T) {
    const TallTask tk = src.task(src.task_of(tile));
    const int64_t r0 = (tile - tk.tile0) * kTallRows;
    for (int t = threadIdx.x; t < kTallRows * k4; t += blockDim.x) {
      const int r = t / k4, c4 = t - r * k4;
      float* dst = T + r * KP + 4 * c4;
      if (r0 + r < tk.n) cp_async16(dst, tk.In + (r0 + r) * ldi + 4 * c4);
      else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };

  int cur = -1;  // the task whose M is staged
  int64_t tile = src.first();
  if (src.valid(tile)) issue(tile, T0);
  cp_async_commit();
  for (int it = 0; src.valid(tile); tile = src.next(tile), ++it) {
    float* T = (it & 1) ? T1 : T0;
    const int64_t next = src.next(tile);
    if (src.valid(next)) issue(next, (it & 1) ? T0 : T1);
    cp_async_commit();
    cp_async_wait1();  // this tile's copies are done (the next tile's may still run)
    const int q = src.task_of(tile);
    const TallTask tk = src.task(q);
    if (q != cur) {  // every thread finished with Ms at the previous tile's last barrier
      for (int t = threadIdx.x; t < K * OUTB; t += blockDim.x) {
        const int l = t / OUTB, o = t % OUTB;
        Ms[t] = o < cnt ? tk.M[l * ldm + o] : 0.f;
      }
      cur = q;
    }
    __syncthreads();
    float acc[RPT][4 * H];
#pragma unroll
    for (int i = 0; i < RPT; ++i)
#pragma unroll
      for (int o = 0; o < 4 * H; ++o) acc[i][o] = 0.f;
    auto terms = [&](int l0, int l1, auto first) {  // rows l0 .. l1 - 1 of M, its columns from 64 first on
      for (int l = l0; l < l1; l += 4) {
        float4 a[RPT];
#pragma unroll
        for (int i = 0; i < RPT; ++i) a[i] = *reinterpret_cast<const float4*>(T + (ty + RS * i) * KP + l);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
#pragma unroll
          for (int h = decltype(first)::value; h < H; ++h) {
            const float4 m = *reinterpret_cast<const float4*>(Ms + (l + u) * OUTB + 64 * h + 4 * tx);
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
              const float x = u == 0 ? a[i].x : u == 1 ? a[i].y : u == 2 ? a[i].z : a[i].w;
              acc[i][4 * h + 0] = fmaf(x, m.x, acc[i][4 * h + 0]);
              acc[i][4 * h + 1] = fmaf(x, m.y, acc[i][4 * h + 1]);
              acc[i][4 * h + 2] = fmaf(x, m.z, acc[i][4 * h + 2]);
              acc[i][4 * h + 3] = fmaf(x, m.w, acc[i][4 * h + 3]);
            }
          }
        }
      }
    };
    terms(0, UPPER && H == 2 ? 64 : K, std::integral_constant<int, 0>{});
    if constexpr (UPPER && H == 2) terms(64, K, std::integral_constant<int, 1>{});
    const int64_t r0 = (tile - tk.tile0) * kTallRows;
    float* Out = tk.Out;
    uint16_t* img = tk.img;
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int64_t row = r0 + ty + RS * i;
      if (row >= tk.n) continue;
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const int col = 64 * h + 4 * tx;
        if (col >= cnt) continue;
        float* out = Out + row * ldo + col;
        const float* v = &acc[i][4 * h];
        if (vec_out) {
          *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
          if (img) {
            uint16_t hh[4], ll[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) split16(v[j], fmt, hh[j], ll[j]);
            *reinterpret_cast<uint4*>(img + (row * ldo + col) * 2) =
                make_uint4(hh[0] | ((uint32_t)ll[0] << 16), hh[1] | ((uint32_t)ll[1] << 16),
                           hh[2] | ((uint32_t)ll[2] << 16), hh[3] | ((uint32_t)ll[3] << 16));
          }
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (col + j < cnt) {
              out[j] = v[j];
              if (img) split16(v[j], fmt, img[(row * ldo + col + j) * 2], img[(row * ldo + col + j) * 2 + 1]);
            }
        }
      }
    }
    __syncthreads();  // every thread is done with T (and Ms) before they are refilled
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int OUTB, int NT, bool UPPER>
__global__ void __launch_bounds__(NT, NT == 256 ? 2 : 1)
    k_tall_mm(const float* In, int64_t n, int K, int ldi, const float* __restrict__ M, int ldm, int cnt, float* Out,
              int ldo, uint16_t* __restrict__ img, int fmt) {
  tall_mm_body<OUTB, NT, UPPER>(TallOne{TallTask{In, Out, img, M, n, 0}, (n + kTallRows - 1) / kTallRows}, K, ldi,
                                ldm, cnt, ldo, fmt);
}

template <int OUTB>
__global__ void __launch_bounds__(256, 2) k_tall_mm_batch(const TallTask* __restrict__ tasks, int ntasks,
                                                          int64_t total_tiles, int K, int ldi, int ldm, int cnt,
                                                          int ldo, int fmt) {
  tall_mm_body<OUTB, 256, false>(tall_batch(tasks, ntasks, total_tiles), K, ldi, ldm, cnt, ldo, fmt);
}

// ---------------------------------------------------------------------------
// Y <- Y M at ld 64 for an upper-triangular M (the Cholesky inverse), with the
// optional 16-bit image: output column c takes only rows l <= c of M, half
// the FMAs of the full product.  Warp w computes the column groups w and
// 15 - w (4 columns each: 4 (w + 1) + 4 (16 - w) = 68 terms, the same for
// every warp), lane r the rows r + 32 i (i < 4) of a 128-row tile.  The tile
// is staged as in k_tall_mm (padded rows, cp.async double buffering, loaded
// whole before any of its rows is written, so Out may alias In).  The terms
// dropped are exact zeros, so the result equals the full product's.
// ---------------------------------------------------------------------------
template <class Src>
__device__ __forceinline__ void upper64_body(const Src& src, int fmt) {
  constexpr int K = 64, KP = K + 4;
  extern __shared__ __align__(16) float sm_u[];
  float* Ms = sm_u;                    // [K][K]
  float* T0 = sm_u + K * K;
  float* T1 = T0 + kTallRows * KP;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  auto issue = [&](int64_t tile, float* T) {
    const TallTask tk = src.task(src.task_of(tile));
    const int64_t r0 = (tile - tk.tile0) * kTallRows;
    for (int t = threadIdx.x; t < kTallRows * (K / 4); t += blockDim.x) {
      const int r = t / (K / 4), c4 = t - r * (K / 4);
      float* dst = T + r * KP + 4 * c4;
      if (r0 + r < tk.n) cp_async16(dst, tk.In + (r0 + r) * K + 4 * c4);
      else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  int cur = -1;  // the task whose M is staged
  int64_t tile = src.first();
  if (src.valid(tile)) issue(tile, T0);
  cp_async_commit();
  for (int it = 0; src.valid(tile); tile = src.next(tile), ++it) {
    float* T = (it & 1) ? T1 : T0;
    const int64_t next = src.next(tile);
    if (src.valid(next)) issue(next, (it & 1) ? T0 : T1);
    cp_async_commit();
    cp_async_wait1();
    const int q = src.task_of(tile);
    const TallTask tk = src.task(q);
    if (q != cur) {  // every thread finished with Ms at the previous tile's last barrier
      for (int t = threadIdx.x; t < K * K; t += blockDim.x) Ms[t] = tk.M[t];
      cur = q;
    }
    __syncthreads();
    const int64_t r0 = (tile - tk.tile0) * kTallRows, n = tk.n;
    float* Out = tk.Out;
    uint16_t* img = tk.img;
    float res[2][16];  // [column group][4 rows x 4 columns]
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int cg = h == 0 ? w : 15 - w;  // column group: columns 4 cg .. 4 cg + 3
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int o = 0; o < 4; ++o) acc[i][o] = 0.f;
      for (int l = 0; l < 4 * (cg + 1); l += 4) {
        float4 a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(T + (lane + 32 * i) * KP + l);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float4 m = *reinterpret_cast<const float4*>(Ms + (l + u) * K + 4 * cg);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float x = u == 0 ? a[i].x : u == 1 ? a[i].y : u == 2 ? a[i].z : a[i].w;
            acc[i][0] = fmaf(x, m.x, acc[i][0]);
            acc[i][1] = fmaf(x, m.y, acc[i][1]);
            acc[i][2] = fmaf(x, m.z, acc[i][2]);
            acc[i][3] = fmaf(x, m.w, acc[i][3]);
          }
        }
      }
      res[h][0] = acc[0][0]; res[h][1] = acc[0][1]; res[h][2] = acc[0][2]; res[h][3] = acc[0][3];
#pragma unroll
      for (int i = 1; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) res[h][4 * i + j] = acc[i][j];
    }
    // A lane holds rows of the tile, so storing from registers would put 32
    // rows (32 sectors) in every warp store.  The results go back into T
    // instead, and the tile leaves row-contiguous: each warp store covers two
    // whole 256-byte rows.
    __syncthreads();  // every warp is done reading T
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int cg = h == 0 ? w : 15 - w;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4*>(T + (lane + 32 * i) * KP + 4 * cg) =
            make_float4(res[h][4 * i], res[h][4 * i + 1], res[h][4 * i + 2], res[h][4 * i + 3]);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kTallRows * (K / 4) / 256; ++u) {
      const int f = threadIdx.x + 256 * u;
      const int r = f >> 4, c4 = f & 15;
      const int64_t row = r0 + r;
      if (row >= n) continue;
      const float4 v = *reinterpret_cast<const float4*>(T + r * KP + 4 * c4);
      *reinterpret_cast<float4*>(Out + row * K + 4 * c4) = v;
      if (img) {
        uint16_t hh[4], ll[4];
        split16(v.x, fmt, hh[0], ll[0]);
        split16(v.y, fmt, hh[1], ll[1]);
        split16(v.z, fmt, hh[2], ll[2]);
        split16(v.w, fmt, hh[3], ll[3]);
        *reinterpret_cast<uint4*>(img + (row * K + 4 * c4) * 2) =
            make_uint4(hh[0] | ((uint32_t)ll[0] << 16), hh[1] | ((uint32_t)ll[1] << 16),
                       hh[2] | ((uint32_t)ll[2] << 16), hh[3] | ((uint32_t)ll[3] << 16));
      }
    }
    __syncthreads();  // every thread is done with T before it is refilled
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

__global__ void __launch_bounds__(256, 2) k_tall_mm_upper64(const float* In, int64_t n,
                                                            const float* __restrict__ M, float* Out,
                                                            uint16_t* __restrict__ img, int fmt) {
  upper64_body(TallOne{TallTask{In, Out, img, M, n, 0}, (n + kTallRows - 1) / kTallRows}, fmt);
}

__global__ void __launch_bounds__(256, 2) k_tall_mm_upper64_batch(const TallTask* __restrict__ tasks, int ntasks,
                                                                  int64_t total_tiles, int fmt) {
  upper64_body(tall_batch(tasks, ntasks, total_tiles), fmt);
}

static cudaError_t tall_mm_upper64(const float* In, int64_t n, const float* M, float* Out, uint16_t* img, int fmt,
                                   cudaStream_t st, int num_sms) {
  if (n == 0) return cudaSuccess;
  const size_t smem = ((size_t)64 * 64 + 2 * (size_t)kTallRows * 68) * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(k_tall_mm_upper64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int grid = grid_for(n, kTallRows, num_sms, 2);
  note_launches(1);
  k_tall_mm_upper64<<<grid, 256, smem, st>>>(In, n, M, Out, img, fmt);
  return cudaGetLastError();
}

cudaError_t launch_apply_upper64_batch(const TallTask* tasks, int ntasks, int64_t total_tiles, int fmt,
                                       cudaStream_t st, int num_sms) {
  if (ntasks <= 0 || total_tiles <= 0) return cudaSuccess;
  const size_t smem = ((size_t)64 * 64 + 2 * (size_t)kTallRows * 68) * sizeof(float);
  if (cudaError_t e = allow_smem(k_tall_mm_upper64_batch, smem); e != cudaSuccess) return e;
  const int grid = (int)std::min<int64_t>(total_tiles, 2 * (int64_t)num_sms);
  note_launches(1);
  k_tall_mm_upper64_batch<<<grid, 256, smem, st>>>(tasks, ntasks, total_tiles, fmt);
  return cudaGetLastError();
}

cudaError_t launch_embed_batch(const TallTask* tasks, int ntasks, int64_t total_tiles, int ld, int nc,
                               cudaStream_t st, int num_sms) {
  if (ntasks <= 0 || total_tiles <= 0) return cudaSuccess;
  if (ld > 64 || nc > 64 || (ld & 3)) return cudaErrorInvalidValue;  // one 64-column panel, as launch_embed at ld 64
  const size_t smem = ((size_t)ld * 64 + 2 * (size_t)kTallRows * (ld + 4)) * sizeof(float);
  if (cudaError_t e = allow_smem(k_tall_mm_batch<64>, smem); e != cudaSuccess) return e;
  const int per_sm = (int)std::max<size_t>(1, std::min<size_t>(2, (220 * 1024) / smem));
  const int grid = (int)std::min<int64_t>(total_tiles, (int64_t)per_sm * num_sms);
  note_launches(1);
  k_tall_mm_batch<64><<<grid, 256, smem, st>>>(tasks, ntasks, total_tiles, ld, ld, nc, nc, nc, 0);
  return cudaGetLastError();
}

// upper: M is upper triangular (told apart at more than 64 columns only).
static cudaError_t tall_mm(const float* In, int64_t n, int K, int ldi, const float* M, int ldm, int cnt,
                           float* Out, int ldo, uint16_t* img, int fmt, cudaStream_t st,
                           int num_sms, bool upper = false) {
  if (n == 0) return cudaSuccess;
  if ((K & 3) || (ldi & 3)) return cudaErrorInvalidValue;
  const int outb = cnt <= 64 ? 64 : 128;
  const size_t smem = ((size_t)K * outb + 2 * (size_t)kTallRows * (K + 4)) * sizeof(float);
  const int per_sm = outb == 64 ? (int)std::max<size_t>(1, std::min<size_t>(2, (220 * 1024) / smem)) : 1;
  const int grid = grid_for(n, kTallRows, num_sms, per_sm);
  auto go = [&](auto kern, int threads) {
    if (cudaError_t e = allow_smem(kern, smem); e != cudaSuccess) return e;
    note_launches(1);
    kern<<<grid, threads, smem, st>>>(In, n, K, ldi, M, ldm, cnt, Out, ldo, img, fmt);
    return cudaGetLastError();
  };
  if (outb == 64) return go(k_tall_mm<64, 256, false>, 256);
  return upper ? go(k_tall_mm<128, 512, true>, 512) : go(k_tall_mm<128, 512, false>, 512);
}

cudaError_t launch_apply_right_f32(const float* In, int64_t n, int ld, const float* M, float* Out,
                                   cudaStream_t st, int num_sms) {
  if (ld > kMaxK) {
    // wider than one panel: in place for an upper-triangular M, else panel by panel into Out
    if (In == Out) return launch_apply_upper_wide(Out, n, ld, M, st, num_sms);
    for (int c0 = 0; c0 < ld; c0 += kPanel) {
      cudaError_t e = launch_tall_mm_wide(In, n, ld, ld, M, ld, c0, kPanel, Out, ld, st, num_sms);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  if (ld == 64) return tall_mm_upper64(In, n, M, Out, nullptr, 0, st, num_sms);
  return tall_mm(In, n, ld, ld, M, ld, ld, Out, ld, nullptr, 0, st, num_sms, true);
}

cudaError_t launch_apply_right_split(const float* In, int64_t n, int ld, const float* M, float* Out,
                                     uint16_t* img, int fmt, cudaStream_t st, int num_sms) {
  if (ld > kMaxK) return cudaErrorInvalidValue;  // the 16-bit image belongs to the tensor-core path (ld <= 128)
  if (ld == 64) return tall_mm_upper64(In, n, M, Out, img, fmt, st, num_sms);
  return tall_mm(In, n, ld, ld, M, ld, ld, Out, ld, img, fmt, st, num_sms, true);
}

// ---------------------------------------------------------------------------
// Gene-side FP64 ops: Z = (W - mu s^T) M for a g x LD matrix W and an LD x LD
// M (mu null: Z = W M; Z may be W), on the FP64 matrix instruction (8 x 8 x 4).
// A block of eight warps stages M once and then RB rows of W at a time; row
// strips and column ranges are dealt to the warps, and a warp keeps its tiles of
// Z in registers over the whole of l.  Rows of both staged matrices are LD + 4
// values apart, which puts the 4 x 8 values of one operand load into different
// banks.  At 64 matrices of 2,000 x 64 the FP64 pipe's floor is 29 us and the
// memory's 25; scalar FMAs, which read a shared value for every 1.6 of them,
// took 70 us, this takes 60: the chain of a block (M in, rows in, products,
// rows out) with three blocks an SM.  One matrix of 3,001 x 128: 24 -> 11 us,
// of 2,000 x 64: 5.1 -> 3.6.
// ---------------------------------------------------------------------------
// Rows per block step: 16 for one matrix (125 blocks at 2,000 genes, a
// latency-bound launch); 64 when a launch covers the segments of a batch
// (thousands of blocks: fewer, larger steps per staged M).
constexpr int kApplyRows = 16, kApplyRowsBatch = 64;

__host__ __device__ constexpr size_t center_apply_smem(int ld, int rb) {
  return ((size_t)ld + rb) * (ld + 4) * sizeof(double);
}

// Block b of nb (of one matrix's grid) takes the row blocks b, b + nb, ...
template <int LD, int RB>
__device__ __forceinline__ void center_apply_body(const double* W, int64_t g, const double* mu, const double* s,
                                                  const double* M, double* Z, int b, int nb) {
  constexpr int ST = LD + 4;
  constexpr int RS = RB / 16 == 1 ? 1 : 2;        // 8-row strips of a warp
  constexpr int NS = RB / (8 * RS);               // warps along the rows: 2 or 4
  constexpr int CT = LD / 8 / (8 / NS);           // 8-column tiles of a warp
  static_assert(NS * RS * 8 == RB && CT * 8 * (8 / NS) == LD, "eight warps cover the block's rows and columns");
  extern __shared__ double sm[];
  double* Ms = sm;               // [LD][ST]
  double* rows = sm + LD * ST;   // [RB][ST]
  {
    // every load of M in flight before the first shared store: one L2 round
    // trip per block instead of one per element the thread stages
    constexpr int PT = LD * LD / 256;  // elements per thread
    double mv[PT];
#pragma unroll
    for (int u = 0; u < PT; ++u) mv[u] = M[threadIdx.x + 256 * u];
#pragma unroll
    for (int u = 0; u < PT; ++u) {
      const int t = threadIdx.x + 256 * u;
      Ms[t / LD * ST + t % LD] = mv[u];
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kr = lane & 3, m = lane >> 2;
  const int r0 = warp % NS * (8 * RS), c0 = warp / NS * (8 * CT);
  for (int64_t j0 = (int64_t)b * RB; j0 < g; j0 += (int64_t)nb * RB) {
    __syncthreads();  // M staged; the previous block's rows consumed
    constexpr int RT = RB * LD / 256;  // row elements per thread
    double wv[RT];
#pragma unroll
    for (int u = 0; u < RT; ++u) {
      const int t = threadIdx.x + 256 * u;
      const int64_t j = j0 + t / LD;
      wv[u] = j < g ? W[j * LD + t % LD] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < RT; ++u) {
      const int t = threadIdx.x + 256 * u;
      const int r = t / LD, c = t % LD;
      const int64_t j = j0 + r;
      double v = wv[u];
      if (j < g && mu) v -= mu[j] * s[c];
      rows[r * ST + c] = v;
    }
    __syncthreads();
    double acc[RS][CT][2];
#pragma unroll
    for (int i = 0; i < RS; ++i)
#pragma unroll
      for (int v = 0; v < CT; ++v) acc[i][v][0] = acc[i][v][1] = 0.0;
#pragma unroll 4
    for (int l = 0; l < LD; l += 4) {
      double a[RS], bm[CT];
#pragma unroll
      for (int i = 0; i < RS; ++i) a[i] = rows[(r0 + 8 * i + m) * ST + l + kr];
#pragma unroll
      for (int v = 0; v < CT; ++v) bm[v] = Ms[(l + kr) * ST + c0 + 8 * v + m];
#pragma unroll
      for (int i = 0; i < RS; ++i)
#pragma unroll
        for (int v = 0; v < CT; ++v) mma_f64(acc[i][v], a[i], bm[v]);
    }
#pragma unroll
    for (int i = 0; i < RS; ++i) {
      const int64_t j = j0 + r0 + 8 * i + m;
      if (j < g)
#pragma unroll
        for (int v = 0; v < CT; ++v)
          *reinterpret_cast<double2*>(Z + j * LD + c0 + 8 * v + 2 * kr) = make_double2(acc[i][v][0], acc[i][v][1]);
    }
  }
}

template <int LD>
__global__ void __launch_bounds__(256) k_center_apply(const double* W, int64_t g, const double* __restrict__ mu,
                                                      const double* __restrict__ s, const double* __restrict__ M,
                                                      double* Z) {
  center_apply_body<LD, kApplyRows>(W, g, mu, s, M, Z, blockIdx.x, gridDim.x);
}

// One matrix per grid row y (batched segments).
template <int LD>
__global__ void __launch_bounds__(256, LD <= 64 ? 3 : 1) k_center_apply_batch(const ApplyTask* __restrict__ tasks, int64_t g) {
  const ApplyTask t = tasks[blockIdx.y];
  center_apply_body<LD, kApplyRowsBatch>(t.W, g, t.mu, t.s, t.M, t.Z, blockIdx.x, gridDim.x);
}

template <int LD>
static cudaError_t center_apply_t(const ApplyTask* tasks, int ntasks, const double* W, int64_t g, const double* mu,
                                  const double* s, const double* M, double* Z, cudaStream_t st) {
  if (g <= 0) return cudaSuccess;
  note_launches(1);
  if (tasks) {
    const size_t smem = center_apply_smem(LD, kApplyRowsBatch);
    if (cudaError_t e = allow_smem(k_center_apply_batch<LD>, smem); e != cudaSuccess) return e;
    // up to 16 blocks per matrix (two 64-row steps each at 2,000 genes), M
    // staged once per block; one wave of longer blocks took 67 us against 60
    const int64_t blocks = (g + kApplyRowsBatch - 1) / kApplyRowsBatch;
    const dim3 grid((unsigned)std::min<int64_t>(blocks, 16), (unsigned)ntasks);
    k_center_apply_batch<LD><<<grid, 256, smem, st>>>(tasks, g);
  } else {
    const size_t smem = center_apply_smem(LD, kApplyRows);
    const int64_t blocks = (g + kApplyRows - 1) / kApplyRows;
    if (cudaError_t e = allow_smem(k_center_apply<LD>, smem); e != cudaSuccess) return e;
    k_center_apply<LD><<<(unsigned)std::min<int64_t>(blocks, 160), 256, smem, st>>>(W, g, mu, s, M, Z);
  }
  return cudaGetLastError();
}

static cudaError_t center_apply_ld(const ApplyTask* tasks, int ntasks, const double* W, int64_t g, int ld,
                                   const double* mu, const double* s, const double* M, double* Z, cudaStream_t st) {
  switch (ld) {
    case 32: return center_apply_t<32>(tasks, ntasks, W, g, mu, s, M, Z, st);
    case 64: return center_apply_t<64>(tasks, ntasks, W, g, mu, s, M, Z, st);
    case 96: return center_apply_t<96>(tasks, ntasks, W, g, mu, s, M, Z, st);
    case 128: return center_apply_t<128>(tasks, ntasks, W, g, mu, s, M, Z, st);
    default: return cudaErrorInvalidValue;  // ld is a multiple of 32 up to kMaxK here
  }
}

cudaError_t launch_center_apply_batch(const ApplyTask* tasks, int ntasks, int64_t g, int ld, cudaStream_t st) {
  if (ld > kMaxK) return cudaErrorInvalidValue;
  if (ntasks <= 0) return cudaSuccess;
  return center_apply_ld(tasks, ntasks, nullptr, g, ld, nullptr, nullptr, nullptr, nullptr, st);
}

cudaError_t launch_center_apply(const double* W, int64_t g, int ld, const double* mu,
                                const double* s, const double* M, double* Z, cudaStream_t st) {
  if (ld > kMaxK) return launch_center_apply_wide(W, g, ld, mu, s, M, Z, st);
  return center_apply_ld(nullptr, 0, W, g, ld, mu, s, M, Z, st);
}

cudaError_t launch_apply_right_f64(double* A, int64_t g, int ld, const double* M, cudaStream_t st) {
  return launch_center_apply(A, g, ld, nullptr, nullptr, M, A, st);
}

__global__ void k_identity(double* __restrict__ M, int ld) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ld * ld; t += gridDim.x * blockDim.x)
    M[t] = t / ld == t % ld ? 1.0 : 0.0;
}

cudaError_t launch_identity(double* M, int ld, cudaStream_t st) {
  note_launches(1);
  k_identity<<<(ld * ld + 1023) / 1024, 256, 0, st>>>(M, ld);
  return cudaGetLastError();
}

__global__ void k_round_v(const double* __restrict__ A, int64_t g, int ld, float* __restrict__ Vf) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < g * ld;
       t += (int64_t)gridDim.x * blockDim.x)
    Vf[t] = (float)A[t];
}

__global__ void k_round_v_batch(const RoundTask* __restrict__ tasks, int64_t g, int ld) {
  const RoundTask tk = tasks[blockIdx.y];
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < g * ld;
       t += (int64_t)gridDim.x * blockDim.x)
    tk.Vf[t] = (float)tk.A[t];
}

// mc[c] = sum_j mu_j Vf[j][c], FP64 accumulation, one block per column.
__device__ __forceinline__ void mean_prefactor_body(const float* Vf, int64_t g, int ld, const double* mu,
                                                    float* mc, int c) {
  __shared__ double red[256];
  double acc = 0.0;
  if (mu)
    for (int64_t j = threadIdx.x; j < g; j += blockDim.x) acc += mu[j] * (double)Vf[j * ld + c];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) mc[c] = (float)red[0];
}

__global__ void k_mean_prefactor(const float* __restrict__ Vf, int64_t g, int ld,
                                 const double* __restrict__ mu, float* __restrict__ mc) {
  mean_prefactor_body(Vf, g, ld, mu, mc, blockIdx.x);
}

// The same sums for every segment of a batch, eight columns per block: row group
// r = 4 w + lane / 8 keeps, for its lane's column, the eight partial sums that
// the threads 8 r .. 8 r + 7 of k_mean_prefactor hold.  So rows are read a full
// 32-byte sector at a time (a block per column read 4 bytes of each: 64
// segments of 2,000 x 64 took 40 us, 13 us now) and the bits are the same.
__global__ void __launch_bounds__(256) k_mean_prefactor_batch(const RoundTask* __restrict__ tasks, int64_t g, int ld) {
  const RoundTask tk = tasks[blockIdx.y];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, c = blockIdx.x * 8 + (lane & 7);
  double acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.0;
  if (tk.mu)
    for (int64_t j0 = 8 * (4 * w + (lane >> 3)); j0 < g; j0 += 256)
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (j0 + i < g) acc[i] += tk.mu[j0 + i] * (double)tk.Vf[(j0 + i) * ld + c];
  __shared__ double red[4][8][32];
#pragma unroll
  for (int h = 4; h > 0; h >>= 1) {  // warps w and w + h
    if (w >= h && w < 2 * h)
#pragma unroll
      for (int i = 0; i < 8; ++i) red[w - h][i][lane] = acc[i];
    __syncthreads();
    if (w < h)
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += red[w][i][lane];
    __syncthreads();
  }
  if (w > 0) return;
#pragma unroll
  for (int o = 16; o >= 8; o >>= 1)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] += __shfl_down_sync(0xffffffffu, acc[i], o);
#pragma unroll
  for (int h = 4; h > 0; h >>= 1)
#pragma unroll
    for (int i = 0; i < h; ++i) acc[i] += acc[i + h];
  if (lane < 8) tk.mc[c] = (float)acc[0];
}

cudaError_t launch_round_v_batch(const RoundTask* tasks, int ntasks, int64_t g, int ld, cudaStream_t st) {
  if (ntasks <= 0) return cudaSuccess;
  note_launches(2);
  const int gx = (int)std::min<int64_t>((g * ld + 255) / 256, 64);
  k_round_v_batch<<<dim3((unsigned)gx, (unsigned)ntasks), 256, 0, st>>>(tasks, g, ld);
  k_mean_prefactor_batch<<<dim3((unsigned)(ld / 8), (unsigned)ntasks), 256, 0, st>>>(tasks, g, ld);
  return cudaGetLastError();
}

// A batch's per-segment results gathered into contiguous buffers, so the
// host takes them in three copies instead of four per segment: status[q] =
// the segment's three status words and its tensor-core error word, sigma[q]
// its k singular values, comps[q] its `count` component floats.
__global__ void k_gather_out(const OutTask* __restrict__ tasks, int k, int64_t count, int* __restrict__ status,
                             double* __restrict__ sigma, float* __restrict__ comps) {
  const int q = blockIdx.y;
  const OutTask t = tasks[q];
  if (blockIdx.x == 0) {
    if (threadIdx.x < 3) status[4 * q + threadIdx.x] = t.status[threadIdx.x];
    if (threadIdx.x == 3) status[4 * q + 3] = t.tc_err ? t.tc_err[0] : 0;
    for (int i = threadIdx.x; i < k; i += blockDim.x) sigma[(int64_t)q * k + i] = t.sigma[i];
  }
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < count; e += (int64_t)gridDim.x * blockDim.x)
    comps[(int64_t)q * count + e] = t.comps[e];
}

cudaError_t launch_gather_out(const OutTask* tasks, int ntasks, int k, int64_t count, int* status, double* sigma,
                              float* comps, cudaStream_t st) {
  if (ntasks <= 0) return cudaSuccess;
  note_launches(1);
  const int gx = (int)std::max<int64_t>(1, std::min<int64_t>((count + 255) / 256, 16));
  k_gather_out<<<dim3((unsigned)gx, (unsigned)ntasks), 256, 0, st>>>(tasks, k, count, status, sigma, comps);
  return cudaGetLastError();
}

// The four status words of every task set to zero (the start of a batch run).
__global__ void k_zero_status(const OutTask* __restrict__ tasks) {
  if (threadIdx.x < 4) tasks[blockIdx.x].status[threadIdx.x] = 0;
}

cudaError_t launch_zero_status(const OutTask* tasks, int ntasks, cudaStream_t st) {
  if (ntasks <= 0) return cudaSuccess;
  note_launches(1);
  k_zero_status<<<ntasks, 32, 0, st>>>(tasks);
  return cudaGetLastError();
}

// mc = mu^T Vf for every task (the Vf and mu of each; A unused).
cudaError_t launch_mean_prefactor_batch(const RoundTask* tasks, int ntasks, int64_t g, int ld, cudaStream_t st) {
  if (ntasks <= 0) return cudaSuccess;
  note_launches(1);
  k_mean_prefactor_batch<<<dim3((unsigned)(ld / 8), (unsigned)ntasks), 256, 0, st>>>(tasks, g, ld);
  return cudaGetLastError();
}

// tasks[q].Vf = src for q = 1 .. ntasks - 1 (count floats, a multiple of 4):
// one segment's test matrix handed to the others of a batch.
__global__ void k_broadcast_v(const float* __restrict__ src, int64_t count4, const RoundTask* __restrict__ tasks) {
  float4* dst = reinterpret_cast<float4*>(tasks[blockIdx.y + 1].Vf);
  const float4* s4 = reinterpret_cast<const float4*>(src);
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < count4; t += (int64_t)gridDim.x * blockDim.x)
    dst[t] = s4[t];
}

cudaError_t launch_broadcast_v(const float* src, int64_t count, const RoundTask* tasks, int ntasks,
                               cudaStream_t st) {
  if (ntasks <= 1 || count <= 0) return cudaSuccess;
  if (count & 3) return cudaErrorInvalidValue;
  note_launches(1);
  const int gx = (int)std::max<int64_t>(1, std::min<int64_t>((count / 4 + 255) / 256, 32));
  k_broadcast_v<<<dim3((unsigned)gx, (unsigned)(ntasks - 1)), 256, 0, st>>>(src, count / 4, tasks);
  return cudaGetLastError();
}

cudaError_t launch_mean_prefactor(const float* Vf, int64_t g, int ld, const double* mu, float* mc,
                                  cudaStream_t st) {
  note_launches(1);
  k_mean_prefactor<<<ld, 256, 0, st>>>(Vf, g, ld, mu, mc);
  return cudaGetLastError();
}

cudaError_t launch_round_v(const double* A, int64_t g, int ld, const double* mu, float* Vf,
                           float* mc, cudaStream_t st) {
  note_launches(1);
  k_round_v<<<(int)std::min<int64_t>((g * ld + 255) / 256, 1184), 256, 0, st>>>(A, g, ld, Vf);
  return launch_mean_prefactor(Vf, g, ld, mu, mc, st);
}

// ---------------------------------------------------------------------------
// Symmetric eigendecomposition of the k x k block of C (SPD up to rounding:
// C = B^T B) by one-sided (Hestenes) Jacobi on its Cholesky factor.
//   1. C = R^T R (FP64, right-looking, in shared memory; a pivot below
//      1e-300 or 1e-15 of the largest diagonal is clamped there -- those are
//      null directions of C, whose eigenvalues are zero to working accuracy).
//   2. Rotate pairs of columns of R from the right until all columns are
//      mutually orthogonal: R J_1 J_2 ... = U Sigma, V = J_1 J_2 ...; then
//      C = V Sigma^2 V^T, eigenvalue i = |column i|^2.
//   3. V is not accumulated rotation by rotation (that doubles the FP64
//      work of every round): it is recovered once as V = R0^{-1} (R0 V) by
//      back substitution against the Cholesky factor R0, and its columns are
//      renormalised.  Its error is about cond(R0) * 1e-16 = sqrt(cond(C)) *
//      1e-16.
// A round takes the kk/2 disjoint column pairs of a round-robin schedule;
// a half-warp owns one pair (a warp serves two pairs with the same shuffle
// instructions): the cross product p.q is a 16-lane partial reduced by
// shuffles, every lane of the half computes the same rotation, and the half
// rotates its two columns of R and of V.  Column norms are carried in closed
// form (a' = a - t c, b' = b + t c for the rotation that zeroes c) and
// recomputed at the start of every sweep.  Pairs are disjoint, so a round
// needs one block barrier.  Columns are stored contiguously (column-major,
// odd stride) so a column walk is conflict-free.  Stops after a sweep with no
// rotation (|p.q| <= 1e-15 |p| |q| for every pair, or |p.q| <= 1e-150), after
// a sweep whose largest rotation tangent is below 1e-4, or after 40 sweeps.
// Convergence is quadratic: the sweep after one whose largest tangent is t
// rotates by about t^2 / 4 at most (measured on power-iteration sketches of
// the NB synthetic at k = 40 and 60: 3e-2 -> 2e-5 -> 9e-11), so stopping at
// t < 1e-4 leaves every eigenvector within ~1e-9 of the next sweep's, below
// the FP32 resolution of the components and embeddings, and the eigenvalues
// (second order in the rotation) within ~1e-18.
// This form serves sketches wider than one panel (k > 128): R, and V after it,
// in the scratch that follows evecs.
template <int NR>  // column entries a lane holds in registers: kk <= 16 NR
__global__ void __launch_bounds__(1024) k_jacobi(const double* __restrict__ C, int k, int ld,
                                                 double* __restrict__ evals, double* __restrict__ evecs,
                                                 int* sweeps_out) {
  extern __shared__ __align__(16) double sm[];
  const int kk = (k + 1) & ~1;  // even number of columns; column k (if odd) is a zero dummy
  const int S = kk + 1;
  const int npair = kk / 2, m = kk - 1;
  double* V = evecs + (size_t)ld * ld;                   // [kk cols][S]: R0, then V
  double* R = V + (size_t)ld * (ld + 1);                 // [kk cols][S]: R[c * S + r]
  uint16_t* sched = reinterpret_cast<uint16_t*>(sm);     // [m][npair]: p | q << 8
  __shared__ double colnorm[kMaxKWide];
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int hl = lane & 15, half = lane >> 4;  // lane within the half-warp, which half
  const unsigned hmask = half ? 0xffff0000u : 0x0000ffffu;
  // R starts as the upper triangle of C (column-major)
  for (int t = tid; t < kk * S; t += nt) {
    const int c = t / S, r = t - c * S;
    R[t] = (r < k && c < k && r <= c) ? C[r * ld + c] : 0.0;
  }
  for (int t = tid; t < m * npair; t += nt) {
    const int round = t / npair, i = t - round * npair;
    int a, b;
    if (i == 0) { a = round; b = m; }
    else { a = (round + i) % m; b = (round - i + m) % m; }
    sched[t] = (uint16_t)(min(a, b) | (max(a, b) << 8));
  }
  __syncthreads();
  // ---- Cholesky in place (upper triangle, right-looking).  Every thread reads
  // pivot j; the diagonal entry itself is written one step later (by thread
  // 0), when nobody reads it any more. ----
  double dmax = 0.0;
  for (int j = 0; j < k; ++j) dmax = fmax(dmax, R[j * S + j]);
  double prev_diag = 0.0;
  for (int j = 0; j < k; ++j) {
    double d = R[j * S + j];
    if (!(d > 1e-15 * dmax) || !(d > 1e-300)) d = fmax(1e-15 * dmax, 1e-300);
    const double rd = rsqrt_nr(d);
    if (tid == 0 && j > 0) R[(j - 1) * S + (j - 1)] = prev_diag;
    prev_diag = d * rd;
    for (int c = j + 1 + tid; c < k; c += nt) R[c * S + j] *= rd;  // row j, right of the diagonal
    __syncthreads();
    // trailing update: R[a][c] -= R[j][a] R[j][c] for j < a <= c (column c by a
    // warp, row a by a lane)
    for (int c = j + 1 + warp; c < k; c += nw) {
      const double rjc = R[c * S + j];
      for (int a = j + 1 + lane; a <= c; a += 32) R[c * S + a] -= R[a * S + j] * rjc;
    }
    __syncthreads();
  }
  if (tid == 0 && k > 0) R[(k - 1) * S + (k - 1)] = prev_diag;
  __syncthreads();
  // R0, kept for the back substitution; a unit diagonal for the dummy column
  // (odd k) keeps it invertible
  for (int t = tid; t < kk * S; t += nt) V[t] = (k < kk && t == k * S + k) ? 1.0 : R[t];
  __syncthreads();
  // ---- one-sided Jacobi on the columns of R ----
  int sweep = 0;
  for (; sweep < 40; ++sweep) {
    // column norms from scratch once per sweep (a half-warp per column)
    for (int col = 2 * warp + half; col < kk; col += 2 * nw) {
      double a = 0.0;
      for (int r = hl; r < kk; r += 16) a = fma(R[col * S + r], R[col * S + r], a);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) a += __shfl_xor_sync(hmask, a, o);
      if (hl == 0) colnorm[col] = a;
    }
    __syncthreads();
    bool large = false;  // this thread's pairs turned by a tangent of 1e-4 or more
    for (int round = 0; round < m; ++round) {
      const uint16_t* pr = sched + round * npair;
      for (int i = 2 * warp + half; i < npair; i += 2 * nw) {
        const int p = pr[i] & 0xff, q = pr[i] >> 8;
        double* rp = R + p * S;
        double* rq = R + q * S;
        // the pair's columns stay in registers from the dot product to the
        // rotation: shared-memory traffic bounds a round, so each column is
        // read once and written once
        double xp[NR], xq[NR];
        double c = 0.0;
#pragma unroll
        for (int u = 0; u < NR; ++u) {
          const int r = hl + 16 * u;
          xp[u] = r < kk ? rp[r] : 0.0;
          xq[u] = r < kk ? rq[r] : 0.0;
          c = fma(xp[u], xq[u], c);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) c += __shfl_xor_sync(hmask, c, o);
        const double a = colnorm[p], b = colnorm[q];
        if (!(fabs(c) > 1e-150 && c * c > 1e-30 * a * b)) continue;  // uniform over the half-warp
        // t = tan of the angle that zeroes p.q: the smaller root of
        // t^2 + 2 zeta t - 1 = 0, zeta = (b - a) / 2c, written as
        // 2c sgn(tau) / (|tau| + sqrt(tau^2 + 4c^2)) with tau = b - a.  The
        // angle only sets how much of p.q a rotation removes, so t is formed
        // in FP32 (inputs scaled by a power of two into range); the rotation
        // itself stays exactly orthogonal in FP64: cs = 1 / sqrt(1 + t^2),
        // sn = t cs.  Near convergence |t| is tiny and its FP32 relative error
        // leaves a residual below 1e-7 |p.q|, cleared by the next sweep.
        const double sc = pow2_int(-exponent_of(a + b));
        const float tf = (float)((b - a) * sc), cf = (float)(2.0 * c * sc);
        const float den = fabsf(tf) + sqrtf(fmaf(tf, tf, cf * cf));
        const double t = (double)(__fdividef(tf >= 0.f ? cf : -cf, den));
        if (t == 0.0) continue;  // below FP32 resolution: nothing to rotate
        const double cs = rsqrt_nr(fma(t, t, 1.0)), sn = t * cs;
#pragma unroll
        for (int u = 0; u < NR; ++u) {
          const int r = hl + 16 * u;
          if (r < kk) {
            rp[r] = cs * xp[u] - sn * xq[u];
            rq[r] = sn * xp[u] + cs * xq[u];
          }
        }
        if (hl == 0) {
          const double cc = cs * cs, ss = sn * sn, x2 = 2.0 * cs * sn * c;
          colnorm[p] = fma(cc, a, fma(ss, b, -x2));
          colnorm[q] = fma(ss, a, fma(cc, b, x2));
        }
        large |= !(fabs(t) < 1e-4);
      }
      __syncthreads();
    }
    if (!__syncthreads_or(large)) break;  // no rotation, or none of 1e-4
  }
  // eigenvalues: squared column norms of R0 V
  for (int col = 2 * warp + half; col < kk; col += 2 * nw) {
    double a = 0.0;
    for (int r = hl; r < kk; r += 16) a = fma(R[col * S + r], R[col * S + r], a);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) a += __shfl_xor_sync(hmask, a, o);
    if (hl == 0) colnorm[col] = a;
  }
  // V = R0^{-1} (R0 V): back substitution, one column per thread, then unit columns
  __syncthreads();
  for (int c = tid; c < kk; c += nt) {
    double* rc = R + c * S;  // column c of R0 V, overwritten by column c of V
    for (int r = kk - 1; r >= 0; --r) {
      double x = rc[r];
      for (int j = r + 1; j < kk; ++j) x = fma(-V[j * S + r], rc[j], x);
      rc[r] = x * rcp_nr(V[r * S + r]);
    }
  }
  __syncthreads();
  // unit eigenvector columns (the squared norms of R0 V's columns, the
  // eigenvalues, were taken before the back substitution)
  for (int i = warp; i < kk; i += nw) {
    double a = 0.0;
    for (int r = lane; r < kk; r += 32) a = fma(R[i * S + r], R[i * S + r], a);
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    a = __shfl_sync(0xffffffffu, a, 0);
    const double inv = a > 0.0 ? rsqrt_nr(a) : 0.0;
    for (int r = lane; r < kk; r += 32) R[i * S + r] *= inv;
  }
  __syncthreads();
  for (int i = tid; i < k; i += nt) {
    const double v = colnorm[i];
    int rank = 0;
    for (int j = 0; j < k; ++j) {
      const double w = colnorm[j];
      if (w > v || (w == v && j < i)) ++rank;
    }
    evals[rank] = v;
    for (int r = 0; r < ld; ++r) evecs[r * ld + rank] = (r < k) ? R[i * S + r] : 0.0;
  }
  for (int t = tid; t < ld * ld; t += nt) {
    const int c = t % ld;
    if (c >= k) evecs[t] = 0.0;
  }
  if (tid == 0 && sweeps_out) *sweeps_out = sweep;
}

// ---------------------------------------------------------------------------
// The same for k <= 128: one-sided Jacobi on the columns of the factor R0 that
// k_cholesky<., true> left in global memory with its inverse (the rotations,
// their order, the angle and the stopping rule are those of k_jacobi).  R0 sits
// in shared memory column by column; eight lanes own a pair and read a column
// 16 bytes per lane (eight lanes cover 128 consecutive bytes: no conflicts for
// any pair).
//
// A round is a chain: columns in, a dot product, the angle, the rotation,
// columns out, a barrier.  A half-warp per pair took 2,600 clocks for it at
// k = 60: the largest tangent went through a 64-bit shared-memory maximum by
// every pair, which serialised them (a lane keeps its own now, and the block
// votes once per sweep), and at k = 110 both columns of every pair through
// shared memory were more than its bandwidth hid.  Of the round-robin's two
// columns of a pair one can stay in its group's registers for half a sweep, so
// only the other moves.  Eight lanes need one shuffle stage less than sixteen
// and half the warps, so the angle's instructions are issued for four pairs at
// once; the pair of a round is kept by counting instead of a table; square
// roots and reciprocals are the hardware's approximations, with steps to
// double precision where the rotation has to be orthogonal.  V = R0^{-1} (R0 V)
// is a product with the stored inverse instead of a back substitution per
// column.  A round now takes 1,300 clocks at k = 60, bound by the latency of
// the chain.  Measured, factor included: 454 -> 295 us at k = 60,
// 228 -> 162 at k = 40, 1,861 -> 977 at k = 110.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int NQ>  // 16-byte pieces of a column per lane: kk <= 16 NQ
__global__ void __launch_bounds__(NQ <= 4 ? 256 : 512) k_jacobi8(int k, int ld, double* evals, double* evecs, int* sweeps_out,
                                                 const JacobiTask* __restrict__ tasks) {
  if (tasks) {
    const JacobiTask t = tasks[blockIdx.x];
    evals = t.evals;
    evecs = t.evecs;
    sweeps_out = t.sweeps;
  }
  // the scratch behind evecs: R0, then R0^{-1}
  double* R0 = evecs + (size_t)ld * ld;
  const double* R0inv = R0 + (size_t)ld * ld;
  constexpr int H = 16 * NQ;  // rows held (zero past k)
  constexpr int S = H + 2;    // column stride: even, so every column starts on 16 bytes
  extern __shared__ __align__(16) double sm[];
  double* R = sm;  // [kk][S]
  __shared__ double colnorm[kMaxK], inv_norm[kMaxK];
  __shared__ int rank_of[kMaxK];
  const int kk = (k + 1) & ~1;  // even number of columns; column k (if odd) is a zero dummy
  const int npair = kk / 2, m = kk - 1;
  const int tid = threadIdx.x, nt = blockDim.x, l = tid & 7, group = tid >> 3, ngroup = nt >> 3;
  for (int t = tid; t < kk * S; t += nt) R[t] = 0.0;
  __syncthreads();
#pragma unroll 8
  for (int t = tid; t < k * ld; t += nt) {
    const int r = t / ld, c = t - r * ld;
    const double x = R0[t];
    if (r <= c && c < k) R[c * S + r] = x;
  }
  __syncthreads();
  auto column = [&](double (&x)[2 * NQ], int c) {
#pragma unroll
    for (int u = 0; u < NQ; ++u)
      *reinterpret_cast<double2*>(x + 2 * u) = *reinterpret_cast<const double2*>(R + c * S + 16 * u + 2 * l);
  };
  auto dot8 = [&](const double (&x)[2 * NQ], const double (&y)[2 * NQ]) {
    double a = 0.0, b = 0.0;
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
      a = fma(x[2 * u], y[2 * u], a);
      b = fma(x[2 * u + 1], y[2 * u + 1], b);
    }
    a += b;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
  };
  auto put_back = [&](const double (&x)[2 * NQ], int c) {
#pragma unroll
    for (int u = 0; u < NQ; ++u)
      *reinterpret_cast<double2*>(R + c * S + 16 * u + 2 * l) = make_double2(x[2 * u], x[2 * u + 1]);
  };
  auto norms = [&]() {
    for (int c0 = 0; c0 < kk; c0 += ngroup) {  // whole warps: a group past the columns repeats the last one
      const int c = min(c0 + group, kk - 1);
      double x[2 * NQ];
      column(x, c);
      const double a = dot8(x, x);
      if (l == 0) colnorm[c] = a;
    }
  };
  const bool active = group < npair;  // a group past the pairs shadows pair 0 and writes nothing
  int sweep = 0;
  for (; sweep < 40; ++sweep) {
    norms();  // from scratch once per sweep
    __syncthreads();
    bool large = false;  // this lane's pair turned by a tangent of 1e-4 or more
    // Pair i of round t: columns (t + i) mod m and (t - i) mod m, and t and m for
    // i = 0.  A group keeps the first of them, xa, in registers while i counts
    // down from its start to 0; only the second moves through shared memory.
    // After i = 0 column t goes back and the group takes column t + npair, the
    // second column of the round's last pair.
    int i = active ? group : 0, ca = i, cb = i ? m - i : 0;
    bool take = true;
    double xa[2 * NQ];
    for (int round = 0; round < m; ++round) {
      const int other = i == 0 ? m : cb;
      double xb[2 * NQ];
      if (take) column(xa, ca);
      column(xb, other);
      const double na = colnorm[ca], nb = colnorm[other];
      // what the angle needs of the norms, while the dot product is on its way
      const double sc = pow2_int(-exponent_of(na + nb));
      const float tf = (float)((ca < other ? nb - na : na - nb) * sc);
      const double least = 1e-30 * na * nb, sc2 = 2.0 * sc;
      const double c = dot8(xa, xb);
      if (active && fabs(c) > 1e-150 && c * c > least) {  // uniform over the pair's lanes
        // t = tan of the angle that zeroes p.q (p the lower column), in single
        // precision from inputs scaled by a power of two into range (k_jacobi);
        // below its resolution t is 0 and the rotation the identity
        const float cf = (float)(c * sc2);
        const float den = fabsf(tf) + sqrt_approx(fmaf(tf, tf, cf * cf));
        const float ts = __fdividef(tf >= 0.f ? cf : -cf, den);
        // cs = 1 / sqrt(1 + t^2) to double precision: a single-precision seed y
        // and one step y (1 + e / 2 + 3 e^2 / 8), e = 1 - (1 + t^2) y^2
        const double t = (double)ts, y = (double)rsqrt_approx(fmaf(ts, ts, 1.f));
        const double e = fma(-fma(t, t, 1.0), y * y, 1.0);
        const double cs = fma(y * e, fma(0.375, e, 0.5), y), sn = ca < other ? t * cs : -t * cs;
#pragma unroll
        for (int u = 0; u < NQ; ++u) {
          double2 z;
          z.x = sn * xa[2 * u] + cs * xb[2 * u];
          z.y = sn * xa[2 * u + 1] + cs * xb[2 * u + 1];
          xa[2 * u] = cs * xa[2 * u] - sn * xb[2 * u];
          xa[2 * u + 1] = cs * xa[2 * u + 1] - sn * xb[2 * u + 1];
          *reinterpret_cast<double2*>(R + other * S + 16 * u + 2 * l) = z;
        }
        if (l == 0) {
          const double cc = cs * cs, ss = sn * sn, x2 = 2.0 * cs * sn * c;
          colnorm[ca] = fma(cc, na, fma(ss, nb, -x2));
          colnorm[other] = fma(ss, na, fma(cc, nb, x2));
        }
        large |= !(fabsf(ts) < 1e-4f);
      }
      take = i == 0;
      if (take) {
        if (active) put_back(xa, ca);
        i = npair - 1;
        cb = ca + 2 - npair;
        if (cb < 0) cb += m;
        ca += npair;
        if (ca >= m) ca -= m;
      } else {
        --i;
        cb += 2;
        if (cb >= m) cb -= m;
      }
      __syncthreads();
    }
    if (active && !take) put_back(xa, ca);
    __syncthreads();
    if (!__syncthreads_or(large)) break;
  }
  // eigenvalues: squared column norms of R0 V; V = R0^{-1} (R0 V), then unit columns
  norms();
  // R0^{-1}'s upper triangle, row by row, behind R
  double* Ri = R + (size_t)kk * S;
  auto row_at = [&](int r) { return Ri + r * k - r * (r + 1) / 2; };  // row_at(r)[j], j >= r
#pragma unroll 8
  for (int t = tid; t < k * ld; t += nt) {
    const int r = t / ld, j = t - r * ld;
    const double x = R0inv[t];
    if (j >= r && j < k) row_at(r)[j] = x;
  }
  __syncthreads();
  // four rows by four columns of V per thread, before scaling: behind both
  // where they fit, else over R0
  double* W = NQ <= 4 ? Ri + k * (k + 1) / 2 : R0;
  const int t4 = (k + 3) / 4;
  for (int t = tid; t < t4 * t4; t += nt) {
    const int r0 = t / t4 * 4, c0 = t % t4;  // columns c0 + t4 f: neighbours in neighbouring lanes
    double acc[4][4] = {};
    const double* ri[4];
    const double* cj[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      ri[e] = row_at(min(r0 + e, k - 1));
      cj[e] = R + min(c0 + t4 * e, k - 1) * S;
    }
    for (int j = r0; j < k; ++j) {
      double x[4], y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        x[e] = j >= r0 + e ? ri[e][j] : 0.0;
        y[e] = cj[e][j];
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int f = 0; f < 4; ++f) acc[e][f] = fma(x[e], y[f], acc[e][f]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int f = 0; f < 4; ++f)
        if (r0 + e < k && c0 + t4 * f < k) W[(r0 + e) * ld + c0 + t4 * f] = acc[e][f];
  }
  __syncthreads();
  // column c's length and rank, eight lanes per column
  for (int c0 = 0; c0 < k; c0 += ngroup) {
    const int c = min(c0 + group, k - 1);
    const double v = colnorm[c];
    double a = 0.0;
    int rank = 0;
    for (int r = l; r < k; r += 8) {
      const double w = W[r * ld + c], o = colnorm[r];
      a = fma(w, w, a);
      if (o > v || (o == v && r < c)) ++rank;
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      rank += __shfl_xor_sync(0xffffffffu, rank, o);
    }
    if (l == 0) {
      inv_norm[c] = a > 0.0 ? rsqrt_nr(a) : 0.0;
      rank_of[c] = rank;
      evals[rank] = v;
    }
  }
  __syncthreads();
  for (int t = tid; t < ld * ld; t += nt) {
    const int r = t / ld, c = t - r * ld;
    if (r < k && c < k) evecs[r * ld + rank_of[c]] = W[t] * inv_norm[c];
    else evecs[t] = 0.0;
  }
  if (tid == 0 && sweeps_out) *sweeps_out = sweep;
}

static cudaError_t jacobi_go(const double* C, int k, int ld, double* evals, double* evecs, int* sweeps,
                             const JacobiTask* tasks, int nblocks, cudaStream_t st) {
  const int kk = (k + 1) & ~1;
  auto go = [&](auto kern, int threads, size_t smem, auto... args) {
    if (cudaError_t e = allow_smem(kern, smem); e != cudaSuccess) return e;
    note_launches(1);
    kern<<<nblocks, threads, smem, st>>>(args...);
    return cudaGetLastError();
  };
  if (k <= kMaxK) {
    // C = R0^T R0 and R0^{-1} into the scratch behind evecs (the plan allocates
    // ld * ld + 2 ld (ld + 1) doubles there), then the rotations
    double* R0 = tasks ? nullptr : evecs + (size_t)ld * ld;
    cudaError_t e = chol_go<true>(C, k, ld, 0.0, 0, R0, tasks ? nullptr : R0 + (size_t)ld * ld, nullptr, nullptr,
                                  tasks, nblocks, st);
    if (e != cudaSuccess) return e;
    const int threads = (kk / 2 * 8 + 31) / 32 * 32;
    auto smem = [&](int nq) {
      return sizeof(double) * ((size_t)kk * (16 * nq + 2) + (size_t)k * (k + 1) / 2 + (nq <= 4 ? (size_t)k * ld : 0));
    };
    if (kk <= 64) return go(k_jacobi8<4>, threads, smem(4), k, ld, evals, evecs, sweeps, tasks);
    return go(k_jacobi8<8>, threads, smem(8), k, ld, evals, evecs, sweeps, tasks);
  }
  if (kk > 256) return cudaErrorInvalidValue;  // the schedule packs a column pair into 8 + 8 bits
  const size_t sched = ((size_t)(kk - 1) * (kk / 2) + 3) / 4 * sizeof(double);
  const int warps = std::min(32, std::max(1, (kk / 2 + 1) / 2));  // one half-warp per column pair
  return go(k_jacobi<16>, 32 * warps, sched, C, k, ld, evals, evecs, sweeps);
}

cudaError_t launch_jacobi_eig(const double* C, int k, int ld, double* evals, double* evecs,
                              int* sweeps, cudaStream_t st) {
  return jacobi_go(C, k, ld, evals, evecs, sweeps, nullptr, 1, st);
}

cudaError_t launch_jacobi_eig_batch(const JacobiTask* tasks, int ntasks, int k, int ld, cudaStream_t st) {
  if (ntasks <= 0) return cudaSuccess;
  return jacobi_go(nullptr, k, ld, nullptr, nullptr, nullptr, tasks, ntasks, st);
}

// ---------------------------------------------------------------------------
// Rayleigh-Ritz finish: sigma, the components and M_emb from B (g x k, in
// Z), the eigenpairs of B^T B and R2^{-1}.
// ---------------------------------------------------------------------------
// Sketches wider than one panel (ld > 128), one matrix: components c0 .. c0 +
// ncc - 1 of nc per launch (E's columns staged in shared memory).  Block b of
// nb takes the rows l = b, b + nb, ... of M_emb and the genes j = b, b + nb,
// ... of the components, its 128 threads spread over (row, component) pairs.
// Each output is one FMA chain in index order.
__global__ void __launch_bounds__(128) k_ritz_finish(const double* __restrict__ B, int64_t g, int ld, int k,
                                                     int nc, int c0, int ncc, const double* __restrict__ evals,
                                                     const double* __restrict__ E,
                                                     const double* __restrict__ Rinv2, double* __restrict__ sigma,
                                                     float* __restrict__ comps, float* __restrict__ M_emb) {
  const int b = blockIdx.x, nb = gridDim.x;
  extern __shared__ double sm[];
  double* Es = sm;              // [ld][ncc]: columns c0 .. c0 + ncc - 1 of E
  double* sg = sm + ld * ncc;   // [ncc]
  for (int t = threadIdx.x; t < ld * ncc; t += blockDim.x) {
    const int l = t / ncc, c = t - l * ncc;
    Es[t] = E[l * ld + c0 + c];
  }
  for (int c = threadIdx.x; c < ncc; c += blockDim.x) sg[c] = sqrt(fmax(evals[c0 + c], 0.0));
  __syncthreads();
  if (b == 0 && c0 == 0)
    for (int c = threadIdx.x; c < k; c += blockDim.x) sigma[c] = sqrt(fmax(evals[c], 0.0));
  // M_emb row l = Rinv2[l, :] E[:, :nc] diag(sigma)
  const int64_t rows_m = b < ld ? (ld - 1 - b) / nb + 1 : 0;
  for (int64_t t = threadIdx.x; t < rows_m * ncc; t += blockDim.x) {
    const int l = b + (int)(t / ncc) * nb, c = (int)(t % ncc);
    double acc = 0.0;
    for (int m = 0; m < ld; ++m) acc = fma(Rinv2[l * ld + m], Es[m * ncc + c], acc);
    M_emb[l * nc + c0 + c] = (float)(acc * sg[c]);
  }
  // components[c][j] = (B E)[j][c] / sigma_c
  const int64_t rows_g = b < g ? (g - 1 - b) / nb + 1 : 0;
  for (int64_t t = threadIdx.x; t < rows_g * ncc; t += blockDim.x) {
    const int64_t j = b + (t / ncc) * nb;
    const int c = (int)(t % ncc);
    double acc = 0.0;
    for (int l = 0; l < k; ++l) acc = fma(B[j * ld + l], Es[l * ncc + c], acc);
    comps[(int64_t)(c0 + c) * g + j] = sg[c] > 0.0 ? (float)(acc / sg[c]) : 0.f;
  }
}

// The same at ld <= 128, where E's columns fit beside the rows: both products
// on the FP64 matrix instruction.  A block stages E (zero past row k and column
// nc) and takes strips of 32 rows at a time, first those of M_emb, then the
// genes of the components; a warp owns eight rows of a strip and half of the
// columns.  Scalar FMAs read E from shared memory once per FMA and a row of B
// through a broadcast load: 2,000 genes, k = 60, 50 components 20 us, 8 now;
// 64 segments with k = 40 and 30 components 164 -> 58; 3,001 genes, k = 110,
// 100 components 72 -> 23.
constexpr int kRitzRows = 32;

template <int LD>
__device__ __forceinline__ void ritz_mma_body(const double* __restrict__ B, int64_t g, int k, int nc,
                                              const double* __restrict__ evals, const double* __restrict__ E,
                                              const double* __restrict__ Rinv2, double* __restrict__ sigma,
                                              float* __restrict__ comps, float* __restrict__ M_emb, int b, int nb) {
  constexpr int ST = LD + 4, CT = LD / 16;  // 8-column tiles of a warp
  extern __shared__ double sm[];
  double* Es = sm;              // [LD][ST]
  double* rows = sm + LD * ST;  // [kRitzRows][ST]
  __shared__ double sg[LD];
  for (int t = threadIdx.x; t < LD * LD; t += 256) {
    const int l = t / LD, c = t % LD;
    Es[l * ST + c] = l < k && c < nc ? E[t] : 0.0;
  }
  for (int c = threadIdx.x; c < LD; c += 256) sg[c] = c < k ? sqrt(fmax(evals[c], 0.0)) : 0.0;
  __syncthreads();
  if (b == 0)
    for (int c = threadIdx.x; c < k; c += 256) sigma[c] = sg[c];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kr = lane & 3, m = lane >> 2;
  const int r0 = warp % 4 * 8, c0 = warp / 4 * (8 * CT);
  constexpr int emb_strips = LD / kRitzRows;
  const int64_t strips = emb_strips + (g + kRitzRows - 1) / kRitzRows;
  for (int64_t strip = b; strip < strips; strip += nb) {
    const bool emb = strip < emb_strips;
    const int64_t j0 = (emb ? strip : strip - emb_strips) * kRitzRows, jn = emb ? LD : g;
    const double* from = emb ? Rinv2 : B;
    __syncthreads();  // the previous strip's rows consumed
    constexpr int RT = kRitzRows * LD / 256;
    double v[RT];
#pragma unroll
    for (int u = 0; u < RT; ++u) {
      const int t = threadIdx.x + 256 * u;
      const int64_t j = j0 + t / LD;
      v[u] = j < jn && t % LD < k ? from[j * LD + t % LD] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < RT; ++u) {
      const int t = threadIdx.x + 256 * u;
      rows[t / LD * ST + t % LD] = v[u];
    }
    __syncthreads();
    if (c0 >= nc) continue;
    double acc[CT][2];
#pragma unroll
    for (int f = 0; f < CT; ++f) acc[f][0] = acc[f][1] = 0.0;
#pragma unroll 4
    for (int l = 0; l < LD; l += 4) {
      const double a = rows[(r0 + m) * ST + l + kr];
#pragma unroll
      for (int f = 0; f < CT; ++f) mma_f64(acc[f], a, Es[(l + kr) * ST + c0 + 8 * f + m]);
    }
    const int64_t j = j0 + r0 + m;
    if (j >= jn) continue;
#pragma unroll
    for (int f = 0; f < CT; ++f)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = c0 + 8 * f + 2 * kr + e;
        if (c >= nc) continue;
        if (emb)
          M_emb[j * nc + c] = (float)(acc[f][e] * sg[c]);
        else
          comps[(int64_t)c * g + j] = sg[c] > 0.0 ? (float)(acc[f][e] / sg[c]) : 0.f;
      }
  }
}

__host__ __device__ constexpr size_t ritz_mma_smem(int ld) {
  return (size_t)(ld + kRitzRows) * (ld + 4) * sizeof(double);
}

// One matrix, or with `tasks` one segment of a batch per grid row y.
template <int LD>
__global__ void __launch_bounds__(256) k_ritz_mma(const RitzTask* __restrict__ tasks, RitzTask one, int64_t g, int k,
                                                  int nc) {
  const RitzTask t = tasks ? tasks[blockIdx.y] : one;
  ritz_mma_body<LD>(t.B, g, k, nc, t.evals, t.evecs, t.Rinv2, t.sigma, t.comps, t.M_emb, blockIdx.x, gridDim.x);
}

template <int LD>
static cudaError_t ritz_mma_go(const RitzTask* tasks, int ntasks, const RitzTask& one, int64_t g, int k, int nc,
                               cudaStream_t st, int num_sms) {
  constexpr size_t smem = ritz_mma_smem(LD);
  if (cudaError_t e = allow_smem(k_ritz_mma<LD>, smem); e != cudaSuccess) return e;
  // one matrix: a strip per block, as many blocks as SMs; a batch: a few strips per staged E
  const int64_t strips = LD / kRitzRows + (g + kRitzRows - 1) / kRitzRows;
  const dim3 grid((unsigned)std::min<int64_t>(strips, tasks ? 16 : num_sms), (unsigned)(tasks ? ntasks : 1));
  note_launches(1);
  k_ritz_mma<LD><<<grid, 256, smem, st>>>(tasks, one, g, k, nc);
  return cudaGetLastError();
}

static cudaError_t ritz_mma(const RitzTask* tasks, int ntasks, const RitzTask& one, int64_t g, int ld, int k, int nc,
                            cudaStream_t st, int num_sms) {
  switch (ld) {
    case 32: return ritz_mma_go<32>(tasks, ntasks, one, g, k, nc, st, num_sms);
    case 64: return ritz_mma_go<64>(tasks, ntasks, one, g, k, nc, st, num_sms);
    case 96: return ritz_mma_go<96>(tasks, ntasks, one, g, k, nc, st, num_sms);
    case 128: return ritz_mma_go<128>(tasks, ntasks, one, g, k, nc, st, num_sms);
    default: return cudaErrorInvalidValue;
  }
}

// Components staged per launch, and the launch's shared bytes.
static int ritz_cols(int ld, int nc, size_t* smem) {
  constexpr size_t kStage = 160 * 1024;  // shared bytes for the staged columns of E
  const int ncc = (int)std::max<size_t>(1, std::min<size_t>(nc, kStage / ((size_t)(ld + 1) * sizeof(double))));
  *smem = (size_t)(ld * ncc + ncc) * sizeof(double);
  return ncc;
}

cudaError_t launch_ritz_finish(const double* B, int64_t g, int ld, int k, int nc,
                               const double* evals, const double* evecs, const double* Rinv2,
                               double* sigma, float* components, float* M_emb, cudaStream_t st, int num_sms) {
  if (ld <= kMaxK)
    return ritz_mma(nullptr, 0, RitzTask{B, evals, evecs, Rinv2, sigma, components, M_emb}, g, ld, k, nc, st,
                    num_sms);
  size_t smem = 0;
  const int ncc = ritz_cols(ld, nc, &smem);
  if (cudaError_t e = allow_smem(k_ritz_finish, smem); e != cudaSuccess) return e;
  // Few blocks: each stages E once and then takes a run of genes.
  const int grid = (int)std::max<int64_t>(std::min<int64_t>(g, 296), std::min<int64_t>(ld, 296));
  for (int c0 = 0; c0 < nc; c0 += ncc) {
    note_launches(1);
    k_ritz_finish<<<grid, 128, smem, st>>>(B, g, ld, k, nc, c0, std::min(ncc, nc - c0), evals, evecs, Rinv2,
                                           sigma, components, M_emb);
  }
  return cudaGetLastError();
}

cudaError_t launch_ritz_finish_batch(const RitzTask* tasks, int ntasks, int64_t g, int ld, int k, int nc,
                                     cudaStream_t st) {
  if (ntasks <= 0) return cudaSuccess;
  return ritz_mma(tasks, ntasks, RitzTask{}, g, ld, k, nc, st, 0);
}

// Embeddings U = Q M_emb (n x nc row-major).
cudaError_t launch_embed(const float* Q, int64_t n, int ld, int k, const float* M_emb, int nc,
                         float* U, cudaStream_t st, int num_sms) {
  (void)k;  // rows k..ld-1 of M_emb are zero
  if (ld > kMaxK) {
    for (int c0 = 0; c0 < nc; c0 += kPanel) {
      cudaError_t e = launch_tall_mm_wide(Q, n, ld, ld, M_emb, nc, c0, std::min(kPanel, nc - c0), U, nc, st,
                                          num_sms);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  return tall_mm(Q, n, ld, ld, M_emb, nc, nc, U, nc, nullptr, 0, st, num_sms);
}

// ---------------------------------------------------------------------------
// Seeded Gaussian: Philox4x32-10 (Salmon et al., SC'11) + Box-Muller in FP64.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void philox4x32_10(uint32_t c[4], uint32_t k0, uint32_t k1) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    uint32_t hi0 = __umulhi(M0, c[0]), lo0 = M0 * c[0];
    uint32_t hi1 = __umulhi(M1, c[2]), lo1 = M1 * c[2];
    uint32_t n0 = hi1 ^ c[1] ^ k0, n1 = lo1, n2 = hi0 ^ c[3] ^ k1, n3 = lo0;
    c[0] = n0; c[1] = n1; c[2] = n2; c[3] = n3;
    k0 += W0;
    k1 += W1;
  }
}

__global__ void k_gaussian(uint64_t seed, int64_t n_rows, int64_t n_cols, float* __restrict__ out,
                           int ld_pad) {
  const int64_t total = n_rows * n_cols;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    uint64_t p = (uint64_t)e >> 1;
    uint32_t c[4] = {(uint32_t)p, (uint32_t)(p >> 32), 0u, 0u};
    philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
    uint64_t a = (((uint64_t)c[0] << 32) | c[1]) >> 11;
    uint64_t b = (((uint64_t)c[2] << 32) | c[3]) >> 11;
    double u1 = ((double)a + 0.5) * 0x1.0p-53;
    double u2 = ((double)b + 0.5) * 0x1.0p-53;
    double r = sqrt(-2.0 * log(u1));
    double ang = 2.0 * 3.141592653589793 * u2;
    double z = (e & 1) ? r * sin(ang) : r * cos(ang);
    if (ld_pad > 0) {
      int64_t i = e % n_rows, j = e / n_rows;
      out[i * ld_pad + j] = (float)z;
    } else {
      out[e] = (float)z;
    }
  }
}

cudaError_t launch_gaussian(uint64_t seed, int64_t n_rows, int64_t n_cols, float* out, int ld_pad,
                            cudaStream_t st, int num_sms) {
  int64_t total = n_rows * n_cols;
  if (total == 0) return cudaSuccess;
  note_launches(1);
  k_gaussian<<<grid_for(total, 256, num_sms), 256, 0, st>>>(seed, n_rows, n_cols, out, ld_pad);
  return cudaGetLastError();
}

__global__ void k_colmajor_to_padded(const float* __restrict__ in, int64_t n_rows, int64_t n_cols,
                                     int ld, float* __restrict__ out) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_rows * ld;
       t += (int64_t)gridDim.x * blockDim.x) {
    int64_t i = t / ld, j = t % ld;
    out[t] = j < n_cols ? in[j * n_rows + i] : 0.f;
  }
}

cudaError_t launch_colmajor_to_padded(const float* in, int64_t n_rows, int64_t n_cols, int ld,
                                      float* out, cudaStream_t st, int num_sms) {
  if (n_rows == 0) return cudaSuccess;
  note_launches(1);
  k_colmajor_to_padded<<<grid_for(n_rows * ld, 256, num_sms), 256, 0, st>>>(in, n_rows, n_cols, ld, out);
  return cudaGetLastError();
}

}  // namespace scx
