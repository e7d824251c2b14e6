// CUDA-core SpMM pair with FP32 products and a fixed summation order (the
// strict FP32 path, and the CUDA-core path of 16-bit values when the tensor
// cores cannot take a matrix).  Both kernels read their dense operand from
// shared memory and accumulate in registers; neither uses floating-point
// atomics, so every result is bit-identical from run to run.
//
//   forward    Y = P V - 1 mc^T   (CSR rows, V staged in gene chunks)
//   transposed W_part = P^T Q     (chunk-CSC copy, Q staged one row chunk at a time)
//
// Restate spmm_forward_row (scx-accel/src/pca/cpu.rs:1500-1523) with the mean
// correction of forward_mean_prefactor (scx-gpu/src/gpu_pca.rs:218-237), and
// spmm_transpose_block (scx-accel/src/pca/cpu.rs:1282-1328) with the output-
// partitioned reduction of spmm_transpose_into (cpu.rs:1330-1389).
//
// Layouts (device memory):
//   CSR       : int64 indptr[n+1], int32 idx[nnz], values[nnz], rows sorted by gene
//   V         : float [n_vars][ld] gene-major;  Y, Q: float [n_obs][ld] cell-major
//   chunk CSC : for row chunk t (geo.rows rows, entries indptr[t T] .. indptr[(t+1) T]),
//               the same entries reordered by (slot, row): row[p] = row within the
//               chunk (uint16), cval[p] = value; tptr[t (g + 1) + s] = offset of slot
//               s's first entry from indptr[t T].  Slots are the genes in decreasing
//               order of stored entries (gene2slot / slot2gene), so neighbouring
//               slots have lists of about the same length.
//   partial   : float [ranges][n_vars][ld], summed in range order by k_reduce_rows
//
// What bounds the pair, and the layout that follows.  An entry costs one row of
// the dense operand out of shared memory, ld x 4 bytes: 2 clocks of an SM's
// 128 bytes per clock at ld 64, 323 us for 47M entries on 148 SMs.  Everything
// else has to hide under that.  So
//   * a block owns a SLICE of 64 or 32 columns and keeps a table of dense rows
//     of that slice, as many as shared memory holds (800 or 1,600), so a list
//     is long, a barrier rare, and one block per SM stages a table a few times
//     per product;
//   * four lanes walk one LIST (a cell's entries inside the table's genes, or a
//     gene's entries inside the table's cells) straight from global memory,
//     eight entries per 32-byte load of indices and of values (the lanes read
//     the same address: a whole sector, so nothing depends on what little L1
//     is left staying there), two steps loaded ahead.  Nothing is exchanged
//     between lanes: no shuffles, ballots or barriers in the walk.  The load
//     delivers a copy of the entry to every lane, which the same pipe pays
//     for: four lanes with 16 columns each cost half of eight lanes with 8;
//   * a lane reads its columns 16 bytes at a time, and the two lists that share
//     a wavefront take the 64-byte halves of a line in opposite order, so no
//     read conflicts;
//   * the eight lists of a warp have about the same length (cells ordered by
//     length in the kernel, genes by slot), and the warps of a block take
//     groups of eight lists in that order.
// With 64 columns the entries are read once and a step has half the overhead
// per column; with 32 there are twice as many blocks per range, so a range is
// twice as long, its partial half the traffic, and a table holds twice the
// rows.  Measured (forward / transposed / sum of partials, us): 250,000 cells
// 554 / 512 / 14 with 64 columns, 569 / 586 / 9 with 32; 50,000 cells 136 / 124
// / 14 and 137 / 134 / 8; 10,000 cells 53 / 48 / 13 and 49 / 44 / 8.  The line
// lies at 256 cells per SM.
// Against the layout before (a 128-row dense window per block, entries
// broadcast with shuffles, 14.6 instructions per entry): 1,304 / 923 us at
// 250,000 x 2,000 (47M entries), 370 / 200 at 50,000, 167 / 62 at 10,000.
#include <algorithm>

#include "common.cuh"
#include "launch.h"

namespace scx {

namespace {

constexpr int kThreads = 512;      // threads of a product block (one block per SM)
constexpr int kLanes = 4;          // lanes that walk a list together
constexpr int kLists = kThreads / kLanes;
constexpr int kRowBlock = 4096;    // cells a forward block orders and walks at a time
constexpr int kBuckets = 256;      // length classes of that order
constexpr size_t kSmemMax = 231424;  // 227 KB less the static variables' share
// forward: the cells' order (uint16) and their cursors (uint32), the length classes
constexpr size_t kFwdSmemFixed = kRowBlock * 2 + kRowBlock * 4 + kBuckets * 4;
// Columns a block holds: 64 where the panel is a multiple of 64 and there are
// cells enough, else 32.
int slice_cols(int ld, int64_t n, int num_sms) {
  return ld % 64 == 0 && n >= (int64_t)256 * num_sms ? 64 : 32;
}
// rows of the table (one more, all zeros, follows them)
constexpr int fwd_table_rows(int cols) { return (int)((kSmemMax - kFwdSmemFixed) / (cols * 4)) - 1; }
constexpr int rmat_table_rows(int cols) { return (int)(kSmemMax / (cols * 4)) - 1; }

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;\n" ::: "memory");
}

// Stage `rows` rows of one slice (row stride lds floats) with the block, and
// the row of zeros behind them.
template <int NV>
__device__ __forceinline__ void stage_table(float* tab, const float* src, int rows, int lds) {
  constexpr int Q = kLanes * NV;  // 16-byte pieces per row
  for (int o = threadIdx.x; o < rows * Q; o += kThreads) {
    const int r = o / Q, q = o % Q;
    cp_async16(tab + r * (4 * Q) + 4 * q, src + (int64_t)r * lds + 4 * q);
  }
  if (threadIdx.x < 4 * Q) tab[rows * (4 * Q) + threadIdx.x] = 0.f;
  cp_async_wait_all();
}

// Eight consecutive list entries, their position a multiple of eight: whole
// 32-byte sectors of an int32 or FP32 array, in one 256-bit load.
template <typename T>
struct Oct {
  alignas(32) T v[8];
};

__device__ __forceinline__ void load_oct(Oct<float>& d, const float* p) {
  asm("ld.global.nc.L2::256B.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(d.v[0]), "=f"(d.v[1]), "=f"(d.v[2]), "=f"(d.v[3]), "=f"(d.v[4]), "=f"(d.v[5]), "=f"(d.v[6]), "=f"(d.v[7])
      : "l"(p));
}
__device__ __forceinline__ void load_oct(Oct<int32_t>& d, const int32_t* p) {
  asm("ld.global.nc.L2::256B.v8.s32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(d.v[0]), "=r"(d.v[1]), "=r"(d.v[2]), "=r"(d.v[3]), "=r"(d.v[4]), "=r"(d.v[5]), "=r"(d.v[6]), "=r"(d.v[7])
      : "l"(p));
}
template <typename T>  // 16-bit types
__device__ __forceinline__ void load_oct(Oct<T>& d, const T* p) {
  static_assert(sizeof(T) == 2, "16-bit entries");
  *reinterpret_cast<uint4*>(d.v) = __ldg(reinterpret_cast<const uint4*>(p));
}

// VEC: the array allows the aligned vector load; positions at or past `lim`
// (the array's length) are not read.
template <bool VEC, typename T>
__device__ __forceinline__ void load_oct(Oct<T>& d, const T* a, int64_t p, int64_t lim) {
  if (VEC && p + 8 <= lim) {
    load_oct(d, a + p);
  } else {
#pragma unroll
    for (int u = 0; u < 8; ++u) d.v[u] = p + u < lim ? a[p + u] : T();
  }
}

__device__ __forceinline__ float4 lds128(unsigned addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}

// acc += sum over the entries [s, e) of val[p] * table row (idx[p] - j0), in
// position order; with LIMIT it stops at the first entry whose row is not in
// the table (idx[p] >= j0 + rows; the list is sorted).  Returns where it
// stopped.  `tab` is the shared address of the lane's first piece of row 0.
// Entries of a step that are not the list's count as zeros and read the row of
// zeros behind the table, so a step is the same instructions for a full and for
// a ragged one and the lists of a warp stay together.  (Their values are cleared
// too: a neighbouring list's may be an infinity, where a finite value does not
// fit the 16-bit working type.  Indices are validated when the plan is built;
// one that is out of range reads that row as well.)
template <bool VEC, bool LIMIT, int NV, typename IdxT, typename ValT>
__device__ __forceinline__ int64_t walk(float (&acc)[4 * NV], const IdxT* __restrict__ idx,
                                        const ValT* __restrict__ val, int64_t s, int64_t e, int64_t lim, int j0,
                                        int rows, unsigned tab) {
  if (s >= e) return e;
  int64_t p = s & ~int64_t(7);
  unsigned valid = 0xffu << (int)(s - p);
  Oct<IdxT> j1, j2;  // the next two steps' entries
  Oct<ValT> x1, x2;
  load_oct<VEC>(j1, idx, p, lim);
  load_oct<VEC>(x1, val, p, lim);
  if (p + 8 < e) {
    load_oct<VEC>(j2, idx, p + 8, lim);
    load_oct<VEC>(x2, val, p + 8, lim);
  }
  while (true) {
    Oct<IdxT> cj = j1;
    Oct<ValT> cx = x1;
    j1 = j2;
    x1 = x2;
    const int64_t left = e - p;  // entries from the step's first position to the list's end
    if (left > 16) {
      load_oct<VEC>(j2, idx, p + 16, lim);
      load_oct<VEC>(x2, val, p + 16, lim);
    } else if (left < 8) {
      valid &= (1u << (int)left) - 1u;
    }
    bool stop = false;
    // (past the list's end the last entry is another list's and says nothing)
    if (LIMIT && (left < 8 || (int)cj.v[7] >= j0 + rows)) {
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if ((int)cj.v[u] >= j0 + rows && (valid >> u & 1)) {
          valid &= (1u << u) - 1u;
          stop = true;
        }
    }
    if (valid != 0xffu) {
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (!(valid >> u & 1)) {
          cj.v[u] = (IdxT)(j0 + rows);
          cx.v[u] = from_f32<ValT>(0.f);
        }
    }
#pragma unroll
    for (int half = 0; half < 8; half += 4) {
      if (LIMIT || (valid >> half & 0xfu)) {
#pragma unroll
        for (int u = half; u < half + 4; ++u) {
          const unsigned r = tab + min((unsigned)((int)cj.v[u] - j0), (unsigned)rows) * (64 * NV);
          const float x = to_f32(cx.v[u]);
#pragma unroll
          for (int h = 0; h < NV; ++h) {
            const float4 v = lds128((h & 1 ? r ^ 64u : r) + (h >> 1) * 128);
            acc[4 * h + 0] = fmaf(x, v.x, acc[4 * h + 0]);
            acc[4 * h + 1] = fmaf(x, v.y, acc[4 * h + 1]);
            acc[4 * h + 2] = fmaf(x, v.z, acc[4 * h + 2]);
            acc[4 * h + 3] = fmaf(x, v.w, acc[4 * h + 3]);
          }
        }
      }
    }
    if (LIMIT && stop) return max(s, p + 32 - __clz(valid));  // past the last entry taken
    if (left <= 8) return e;
    p += 8;
    valid = 0xffu;
  }
}

// A lane's columns of a row: piece h is 4 floats at 16 ((h & ~1) + ((h ^ list) & 1)) + 4 l.
// Lists of odd and even number in the block take the two 64-byte pieces of a
// 128-byte line in opposite order, so the two lists of a shared-memory
// wavefront (8 lanes) never meet in a bank.
__device__ __forceinline__ int piece_col(int h, int odd) { return 16 * ((h & ~1) + ((h & 1) ^ odd)); }

template <int NV>
__device__ __forceinline__ void load_cols(float (&a)[4 * NV], const float* src, int odd) {
#pragma unroll
  for (int h = 0; h < NV; ++h)
    *reinterpret_cast<float4*>(a + 4 * h) = *reinterpret_cast<const float4*>(src + piece_col(h, odd));
}
template <int NV>
__device__ __forceinline__ void store_cols(float* dst, const float (&a)[4 * NV], int odd) {
#pragma unroll
  for (int h = 0; h < NV; ++h)
    *reinterpret_cast<float4*>(dst + piece_col(h, odd)) =
        make_float4(a[4 * h], a[4 * h + 1], a[4 * h + 2], a[4 * h + 3]);
}

}  // namespace

// ---------------------------------------------------------------------------
// Stored entries per gene.  Each block counts its share in shared memory and
// adds its counts to the global ones (integers: the order does not matter).
// Matrices with more genes than a block's counters go to global memory directly.
// (100,000 x 2,000, 18M entries: 26 us, against 606 us with one global
// atomic per entry, which a few frequent genes serialise.)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(512) k_gene_counts(const int32_t* __restrict__ idx, int64_t nnz, int32_t g,
                                                     int32_t* __restrict__ counts) {
  extern __shared__ int32_t hist[];
  for (int j = threadIdx.x; j < g; j += blockDim.x) hist[j] = 0;
  __syncthreads();
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < nnz; p += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t j = (uint32_t)__ldg(idx + p);
    if (j < (uint32_t)g) atomicAdd(hist + j, 1);  // a streamed shard is counted before its flags are read
  }
  __syncthreads();
  for (int j = threadIdx.x; j < g; j += blockDim.x) {
    const int32_t c = hist[j];
    if (c) atomicAdd(counts + j, c);
  }
}

__global__ void k_gene_counts_global(const int32_t* __restrict__ idx, int64_t nnz, int32_t g,
                                     int32_t* __restrict__ counts) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < nnz; p += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t j = (uint32_t)__ldg(idx + p);
    if (j < (uint32_t)g) atomicAdd(counts + j, 1);
  }
}

// Slots: genes in decreasing order of stored entries, ties by gene.  One warp
// per gene counts the genes in front of it, so the order needs no host round
// trip (2,000 genes: a few us, against two copies, a synchronisation and a
// host sort).
__global__ void __launch_bounds__(256) k_rank_genes(const int32_t* __restrict__ counts, int32_t g,
                                                    int32_t* __restrict__ gene2slot, int32_t* __restrict__ slot2gene) {
  const int lane = threadIdx.x & 31;
  const int32_t j = (int32_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (j >= g) return;
  const int32_t mine = __ldg(counts + j);
  int32_t before = 0;
  for (int32_t i = lane; i < g; i += 32) {
    const int32_t c = __ldg(counts + i);
    before += (c > mine || (c == mine && i < j)) ? 1 : 0;
  }
  before = (int32_t)__reduce_add_sync(0xffffffffu, (unsigned)before);
  if (lane == 0) {
    gene2slot[j] = before;
    slot2gene[before] = j;
  }
}

// ---------------------------------------------------------------------------
// Chunk-CSC build, one block per row chunk (once per plan).  Counting sort of
// the chunk's entries by slot that keeps row order inside a slot: warp w takes
// the w-th run of consecutive rows, counts its entries per slot in shared
// memory, the block turns the counts into each warp's first position in every
// slot, and each warp then places its rows in order.  Few and long chunks are
// built by `splits` blocks each, a run of rows a block: a first launch
// (PASS 1) leaves each warp's counts in `first`, k_chunk_sums turns them into
// its first place in every slot's list and k_chunk_scan the lists' lengths into
// the slots' pointers, and a second launch (PASS 2) places.  Within one 32-entry
// step two lanes can name the same gene only across a duplicate; the step is
// cut into runs of strictly increasing gene, applied in lane order, which
// keeps the placement (and so the later summation order) deterministic.
// The scattered stores bound it (each entry writes a part of two sectors: at
// 100,000 x 2,000 the 115 MB copy causes 835 MB of DRAM writes); up to 16 warps
// share a chunk and load four steps ahead.  10,000 x 2,000: 74 us against
// 836 us for one warp per 128-row tile, 100,000: 723 against 1,171 us.
// ---------------------------------------------------------------------------
template <typename ValT, int PASS>  // 0: a block does all of its chunk
__global__ void __launch_bounds__(512) k_chunk_csc(const int64_t* __restrict__ indptr, const int32_t* __restrict__ idx,
                                                   const ValT* __restrict__ val, int64_t n, int chunk_rows, int splits,
                                                   const int32_t* __restrict__ gene2slot, int32_t g, bool map_in_smem,
                                                   int32_t* __restrict__ first, int32_t* __restrict__ tptr,
                                                   uint16_t* __restrict__ row, ValT* __restrict__ cval) {
  extern __shared__ int32_t cur_all[];  // [warps][g], then gene2slot
  __shared__ int32_t warp_sum[16];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int64_t t = PASS == 0 ? blockIdx.x : blockIdx.x / splits;
  const int64_t c0 = t * chunk_rows, c1 = min(n, c0 + chunk_rows);
  // the block's rows b0 .. b1 - 1, of which the warp's are r0 .. r1 - 1
  const int per_block = PASS == 0 ? chunk_rows : (chunk_rows + splits - 1) / splits;
  const int64_t b0 = PASS == 0 ? c0 : min(c1, c0 + (int64_t)(blockIdx.x % splits) * per_block);
  const int64_t b1 = min(c1, b0 + per_block);
  const int per_warp = (int)((b1 - b0 + warps - 1) / warps);
  const int64_t r0 = min(b1, b0 + (int64_t)w * per_warp), r1 = min(b1, r0 + per_warp);
  const int64_t base = indptr[c0];
  int32_t* cur = cur_all + (int64_t)w * g;
  const int32_t* map = gene2slot;
  if (map_in_smem) {
    int32_t* m = cur_all + (int64_t)warps * g;
    for (int j = threadIdx.x; j < g; j += blockDim.x) m[j] = gene2slot[j];
    map = m;
  }
  const int nc = warps * g;
  if (PASS < 2) {
    for (int j = threadIdx.x; j < nc; j += blockDim.x) cur_all[j] = 0;
    __syncthreads();
    // counts (integer atomics: the counts do not depend on the order)
    const int64_t b = indptr[r0], e = indptr[r1];
#pragma unroll 4
    for (int64_t p = b + lane; p < e; p += 32) atomicAdd(&cur[map[__ldg(idx + p)]], 1);
    __syncthreads();
  }
  if (PASS == 0) {
    // exclusive scan over (slot, warp): thread i owns a run of slots
    const int per = (g + (int)blockDim.x - 1) / (int)blockDim.x;
    const int j0 = min(g, (int)threadIdx.x * per), j1 = min(g, j0 + per);
    int32_t sum = 0;
    for (int j = j0; j < j1; ++j)
      for (int u = 0; u < warps; ++u) sum += cur_all[(int64_t)u * g + j];
    int32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) warp_sum[w] = incl;
    __syncthreads();
    int32_t run = incl - sum;
    for (int u = 0; u < w; ++u) run += warp_sum[u];
    for (int j = j0; j < j1; ++j) {
      tptr[t * (g + 1) + j] = run;
      for (int u = 0; u < warps; ++u) {
        const int32_t c = cur_all[(int64_t)u * g + j];
        cur_all[(int64_t)u * g + j] = run;
        run += c;
      }
    }
    if (threadIdx.x == 0) tptr[t * (g + 1) + g] = (int32_t)(indptr[c1] - base);
  } else {
    int32_t* mine = first + (int64_t)blockIdx.x * nc;
    if (PASS == 1) {
      for (int j = threadIdx.x; j < nc; j += blockDim.x) mine[j] = cur_all[j];
      return;
    }
    for (int j = threadIdx.x; j < nc; j += blockDim.x) cur_all[j] = mine[j] + __ldg(tptr + t * (g + 1) + j % g);
  }
  __syncthreads();
  // placement, rows in order
  const unsigned lanemask_le = 0xffffffffu >> (31 - lane);
  if (r0 >= r1) return;
  // the steps (32 entries of one row) are loaded kAhead steps before they are placed
  constexpr int kAhead = 4;
  int32_t sj[kAhead];
  ValT sx[kAhead];
  int sr[kAhead];  // row within the chunk, -1 past the last step
  int64_t r = r0, b = indptr[r0], e = indptr[r0 + 1];
  auto fetch = [&](int u) {
    while (b >= e && ++r < r1) {  // the next row with entries
      b = e;
      e = indptr[r + 1];
    }
    sr[u] = r < r1 ? (int)(r - c0) : -1;
    const bool ok = r < r1 && b + lane < e;
    sj[u] = ok ? __ldg(idx + b + lane) : -1;
    sx[u] = ok ? val[b + lane] : ValT();
    b += 32;
    if (b > e) b = e;
  };
#pragma unroll
  for (int u = 0; u < kAhead; ++u) fetch(u);
  while (sr[0] >= 0) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int32_t j = sj[u];
      const ValT x = sx[u];
      const int rl = sr[u];
      fetch(u);
      const bool ok = j >= 0;
      const int32_t jl = __shfl_up_sync(0xffffffffu, j, 1);
      const unsigned starts = __ballot_sync(0xffffffffu, lane > 0 && ok && j <= jl);
      const int my_run = __popc(starts & lanemask_le);
      const int runs = __popc(starts) + 1;
      const int32_t slot = ok ? map[j] : 0;
      for (int rr = 0; rr < runs; ++rr) {
        if (ok && my_run == rr) {
          const int32_t q = cur[slot];
          cur[slot] = q + 1;
          row[base + q] = (uint16_t)rl;
          cval[base + q] = x;
        }
        __syncwarp();
      }
    }
  }
}

// first[chunk][share][slot]: a share's (a warp's) counts become its first place in
// each slot's list; the lists' lengths go to tptr.
__global__ void __launch_bounds__(256) k_chunk_sums(int shares, int32_t g, int32_t* __restrict__ first,
                                                    int32_t* __restrict__ tptr) {
  const int j = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (j >= g) return;
  int32_t* f = first + (int64_t)blockIdx.y * shares * g + j;
  int32_t run = 0;
#pragma unroll 8
  for (int u = 0; u < shares; ++u) {
    const int32_t c = f[(int64_t)u * g];
    f[(int64_t)u * g] = run;
    run += c;
  }
  tptr[(int64_t)blockIdx.y * (g + 1) + j] = run;
}

// A chunk's list lengths become its pointers, in place; one block per chunk.
__global__ void __launch_bounds__(1024) k_chunk_scan(int32_t g, int32_t* __restrict__ tptr) {
  __shared__ int32_t warp_sum[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int32_t* tp = tptr + (int64_t)blockIdx.x * (g + 1);
  int32_t base = 0;
  for (int j0 = 0; j0 < g; j0 += 1024) {
    const int j = j0 + (int)threadIdx.x;
    const int32_t c = j < g ? tp[j] : 0;
    int32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) warp_sum[w] = incl;
    __syncthreads();
    int32_t before = 0, total = 0;
    for (int u = 0; u < 32; ++u) {
      if (u < w) before += warp_sum[u];
      total += warp_sum[u];
    }
    if (j < g) tp[j] = base + before + incl - c;
    base += total;
    __syncthreads();  // the warps' sums are read
  }
  if (threadIdx.x == 0) tp[g] = base;
}

// ---------------------------------------------------------------------------
// Forward product.  Block (slice, range) owns 64 or 32 columns (16 NV) of a
// contiguous range of cells, kRowBlock of them at a time, and takes the genes in chunks of
// `table_rows`: V's chunk is staged, every cell's entries inside the chunk are
// walked, and the sums go to Y (read back by the same lanes for the next
// chunk; the entries are added in row order whatever the chunks).  The cells
// are ordered by length (a counting sort over kBuckets classes): the order
// only decides which lanes take which cell, not any result.  A walk stops at
// the first gene past the chunk (rows are sorted); where it stopped is kept in
// shared memory for the next chunk.
// ---------------------------------------------------------------------------
template <bool VEC, int NV, typename ValT>
__global__ void __launch_bounds__(kThreads, 1)
    k_fwd_strict(const int64_t* __restrict__ indptr, const int32_t* __restrict__ idx, const ValT* __restrict__ val,
                 int64_t n, int32_t g, int nslice, int64_t rows_per_range, int table_rows,
                 const float* __restrict__ V, const float* __restrict__ mc, float* Y, int lds) {
  extern __shared__ __align__(128) char smem[];
  float* tab = reinterpret_cast<float*>(smem);
  uint32_t* cursor = reinterpret_cast<uint32_t*>(smem + (size_t)(table_rows + 1) * (64 * NV));
  int32_t* bucket = reinterpret_cast<int32_t*>(cursor + kRowBlock);
  uint16_t* order = reinterpret_cast<uint16_t*>(bucket + kBuckets);
  __shared__ int32_t longest;
  const int tid = threadIdx.x, lane = tid & 31, l = tid % kLanes, list = tid / kLanes, odd = list & 1;
  const int slice = blockIdx.x % nslice;
  const int64_t range = blockIdx.x / nslice;
  const int64_t r0 = range * rows_per_range, r1 = min(n, r0 + rows_per_range);
  const int nch = (g + table_rows - 1) / table_rows;
  const int64_t lim = indptr[n];
  const int col = slice * (16 * NV) + 4 * l;
  const unsigned tab_lane = (unsigned)__cvta_generic_to_shared(smem) + 16 * l + 64 * odd;
  float m[4 * NV] = {};
  if (mc) load_cols<NV>(m, mc + col, odd);
  for (int64_t rb = r0; rb < r1; rb += kRowBlock) {
    const int rows = (int)min((int64_t)kRowBlock, r1 - rb);
    // order the cells by decreasing number of entries
    if (tid == 0) longest = 1;
    for (int b = tid; b < kBuckets; b += kThreads) bucket[b] = 0;
    __syncthreads();
    for (int i = tid; i < rows; i += kThreads) {
      const int64_t len = indptr[rb + i + 1] - indptr[rb + i];
      cursor[i] = (uint32_t)min(len, (int64_t)INT32_MAX);
      atomicMax(&longest, (int)cursor[i]);
    }
    __syncthreads();
    const float scale = (float)(kBuckets - 1) / (float)longest;
    auto bucket_of = [&](int i) { return kBuckets - 1 - min(kBuckets - 1, (int)((float)cursor[i] * scale)); };
    for (int i = tid; i < rows; i += kThreads) atomicAdd(&bucket[bucket_of(i)], 1);
    __syncthreads();
    if (tid < 32) {  // exclusive scan of the classes
      int32_t run = 0;
      for (int b = lane; b < kBuckets; b += 32) {
        const int32_t c = bucket[b];
        int32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += y;
        }
        bucket[b] = run + incl - c;
        run += __shfl_sync(0xffffffffu, incl, 31);
      }
    }
    __syncthreads();
    for (int i = tid; i < rows; i += kThreads) order[atomicAdd(&bucket[bucket_of(i)], 1)] = (uint16_t)i;
    __syncthreads();
    for (int i = tid; i < rows; i += kThreads) cursor[i] = 0;
    for (int ch = 0; ch < nch; ++ch) {
      const int g0 = ch * table_rows, g1 = min((int)g, g0 + table_rows);
      const bool last = ch + 1 == nch;
      if (ch > 0 || nch > 1 || rb == r0) {  // one chunk: the table stays
        __syncthreads();                    // everyone is done with the table
        stage_table<NV>(tab, V + (int64_t)g0 * lds + slice * (16 * NV), g1 - g0, lds);
      }
      __syncthreads();
      int64_t nbase = 0, nend = 0;  // the next cell's bounds, read one cell ahead
      if (list < rows) {
        nbase = indptr[rb + order[list]];
        nend = indptr[rb + order[list] + 1];
      }
      for (int i = list; i < rows; i += kLists) {
        const int rl = order[i];
        const int64_t row = rb + rl;
        const int64_t base = nbase, s = base + cursor[rl], e = nend;
        if (i + kLists < rows) {
          nbase = indptr[rb + order[i + kLists]];
          nend = indptr[rb + order[i + kLists] + 1];
        }
        float* y = Y + row * lds + col;
        float acc[4 * NV] = {};
        if (ch > 0) load_cols<NV>(acc, y, odd);
        const int64_t stop = walk<VEC, true, NV>(acc, idx, val, s, e, lim, g0, g1 - g0, tab_lane);
        if (last) {
#pragma unroll
          for (int c = 0; c < 4 * NV; ++c) acc[c] -= m[c];
        } else if (l == 0) {  // read next after the block's barrier
          cursor[rl] = (uint32_t)(stop - base);
        }
        store_cols<NV>(y, acc, odd);
      }
    }
    __syncthreads();  // the order and the cursors are rewritten
  }
}

// ---------------------------------------------------------------------------
// Transposed product.  Block (slice, range) owns 64 or 32 columns (16 NV) of
// the row chunks of one contiguous range; for each chunk it stages Q's rows and
// walks every slot's list, a warp taking eight neighbouring slots.  The sums go
// to the range's partial (read back by the same lanes for the next chunk).
// Entries are added in (chunk, row) order.  gridDim.y blocks share the slots of
// a range (strict_geometry).
// ---------------------------------------------------------------------------
template <int NV, typename ValT>
__global__ void __launch_bounds__(kThreads, 1)
    k_rmat_strict(const int64_t* __restrict__ indptr, const int32_t* __restrict__ tptr,
                  const uint16_t* __restrict__ row, const ValT* __restrict__ cval, int64_t n, int32_t g,
                  const int32_t* __restrict__ slot2gene, int chunk_rows, int64_t n_chunks, int chunks_per_range,
                  int nslice, const float* __restrict__ Q, int lds, float* part, int ldp) {
  extern __shared__ __align__(128) char smem[];
  float* tab = reinterpret_cast<float*>(smem);
  const int tid = threadIdx.x, l = tid % kLanes, list = tid / kLanes, odd = list & 1;
  const unsigned tab_lane = (unsigned)__cvta_generic_to_shared(smem) + 16 * l + 64 * odd;
  const int slice = blockIdx.x % nslice;
  const int64_t range = blockIdx.x / nslice;
  const int64_t t0 = range * chunks_per_range, t1 = min(n_chunks, t0 + chunks_per_range);
  // the block's slots: eight neighbours a warp, the blocks' eights in turn
  const int s0 = (list / 8 * (int)gridDim.y + (int)blockIdx.y) * 8 + list % 8, step = (int)gridDim.y * kLists;
  float* out = part + range * g * ldp + slice * (16 * NV) + 4 * l;
  for (int64_t t = t0; t < t1; ++t) {
    const int64_t r0 = t * chunk_rows;
    const int rows = (int)min((int64_t)chunk_rows, n - r0);
    __syncthreads();  // everyone is done with the table
    stage_table<NV>(tab, Q + r0 * lds + slice * (16 * NV), rows, lds);
    __syncthreads();
    const int64_t base = indptr[r0], lim = indptr[r0 + rows];
    const int32_t* tp = tptr + t * (g + 1);
    int nb = 0, ne = 0, ng = 0;  // the next list's bounds and gene, read one list ahead
    if (s0 < g) {
      nb = __ldg(tp + s0);
      ne = __ldg(tp + s0 + 1);
      ng = __ldg(slot2gene + s0);
    }
    for (int s = s0; s < g; s += step) {
      const int64_t b = base + nb, e = base + ne;
      float* w = out + (int64_t)ng * ldp;
      if (s + step < g) {
        nb = __ldg(tp + s + step);
        ne = __ldg(tp + s + step + 1);
        ng = __ldg(slot2gene + s + step);
      }
      if (t > t0 && b >= e) continue;
      float acc[4 * NV] = {};
      if (t > t0) load_cols<NV>(acc, w, odd);
      walk<true, false, NV>(acc, row, cval, b, e, lim, 0, rows, tab_lane);
      store_cols<NV>(w, acc, odd);
    }
  }
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------

// The transposed product's row chunks: the ranges of all slices, with `parts`
// blocks each, fill the SMs once; a range is a whole number of equal chunks that
// fit the table, and a chunk has at least 64 rows (below that a list is shorter
// than its set-up).
//
// Every range writes a partial of all genes and every list costs a load's
// latency, so with many genes and few cells (fewer than 256 per SM) the SMs are
// filled by parts rather than by ranges: a part per 2,048 genes (with fewer the
// most frequent genes' lists set a block's time), and as many as give a chunk
// 128 rows while a part keeps 256 genes.  Product and sum of partials with one
// block a range, with this, and in the 128-row layout before (us): 2,000 x
// 30,000, k = 60 528, 137, 202; 5,000 x 10,000, k = 30 190, 86, 139; 10,000 x
// 30,000, k = 110 653, 335, 760; 300 x 20,000, k = 30 the call 379, 93, 104.
// Where this leaves one part (10,000 x 2,000, k = 60: 67 us) nothing changes.
//
// Long chunks are built by as many blocks as fill the SMs once: from 256 rows on,
// or 64 where the genes leave room for at most 12 warps a block.  A plan of 2,000 x
// 30,000 takes 5.9 ms (one block a 64-row chunk 8.8, 23.7 before), of 10,000 x
// 30,000 4.0 (3.9, 10.9).  g = 0 (a streamed shard, whose copy is built for every
// product): one block a range and a chunk.
StrictGeometry strict_geometry(int64_t n, int64_t g, int ld, int num_sms) {
  StrictGeometry geo;
  geo.cols = slice_cols(ld, n, num_sms);
  const int nslice = ld / geo.cols, table_rows = rmat_table_rows(geo.cols);
  const int64_t want = std::max<int64_t>(1, num_sms / nslice);
  int64_t parts = 1;
  if (n < (int64_t)256 * num_sms) {  // (g = 0: one part)
    const int64_t longer = std::min<int64_t>((128 * want + n - 1) / n, g / 256);
    const int64_t fewest = (n + table_rows - 1) / table_rows;  // ranges of one chunk
    parts = std::max<int64_t>(1, std::min<int64_t>(std::max<int64_t>(g / 2048, longer), want / fewest));
  }
  const int64_t ranges = std::max<int64_t>(1, want / parts);
  const int64_t per = std::max<int64_t>(64, (n + ranges - 1) / ranges);
  const int64_t m = (per + table_rows - 1) / table_rows;
  geo.rows = (int)((per + m - 1) / m);
  geo.chunks = (n + geo.rows - 1) / geo.rows;
  geo.per_range = (int)m;
  geo.ranges = (int)((geo.chunks + m - 1) / m);
  // the last ones: ranges of at least 64 rows may be fewer still
  geo.parts = (int)std::max<int64_t>(1, std::min<int64_t>(want / geo.ranges, (g + kLists - 1) / kLists));
  if (parts > 1 && geo.rows >= (g > 4096 ? 64 : 256))
    geo.splits = (int)std::max<int64_t>(1, std::min<int64_t>(geo.rows / 32, num_sms / geo.chunks));
  return geo;
}

// One warp's slot counters of the chunk-CSC build have to fit shared memory.
bool strict_csc_fits(int64_t g) { return g <= kStrictMaxGenes; }

cudaError_t launch_gene_counts(const int32_t* idx, int64_t nnz, int32_t g, int32_t* counts, cudaStream_t st,
                               int num_sms) {
  if (nnz == 0) return cudaSuccess;
  note_launches(1);
  const size_t smem = sizeof(int32_t) * (size_t)g;
  if (smem <= 100 * 1024) {  // two blocks per SM
    if (smem > 48 * 1024)
      if (cudaError_t e = allow_smem(k_gene_counts, smem); e != cudaSuccess) return e;
    k_gene_counts<<<grid_for(nnz, 8192, num_sms, 2), 512, smem, st>>>(idx, nnz, g, counts);
  } else {
    k_gene_counts_global<<<grid_for(nnz, 256, num_sms), 256, 0, st>>>(idx, nnz, g, counts);
  }
  return cudaGetLastError();
}

cudaError_t launch_rank_genes(const int32_t* counts, int32_t g, int32_t* gene2slot, int32_t* slot2gene,
                              cudaStream_t st) {
  note_launches(1);
  k_rank_genes<<<(unsigned)(((int64_t)g + 7) / 8), 256, 0, st>>>(counts, g, gene2slot, slot2gene);
  return cudaGetLastError();
}

// Warps of a block of the build: as many as have room for their counters.
static int csc_warps(const StrictGeometry& geo, int64_t g) {
  const int most = (int)std::min<int64_t>(16, kStrictMaxGenes / g);
  return std::max(1, std::min(most, ((geo.rows + geo.splits - 1) / geo.splits + 3) / 4));
}

template <typename ValT>
static cudaError_t chunk_csc_t(const int64_t* indptr, const int32_t* idx, const void* val, int64_t n,
                               const StrictGeometry& geo, const int32_t* gene2slot, int32_t g, int32_t* first,
                               int32_t* tptr, uint16_t* row, void* cval, cudaStream_t st) {
  if (!strict_csc_fits(g)) return cudaErrorInvalidValue;
  const int splits = geo.splits, warps = csc_warps(geo, g);
  const size_t per_warp = sizeof(int32_t) * (size_t)g;
  // the slot map beside the counters where it fits (a gather per entry from L1
  // costs a tag lookup per line it touches)
  const bool map_in_smem = per_warp * (warps + 1) <= kStatsSmemMax;
  const size_t smem = per_warp * (warps + (map_in_smem ? 1 : 0));
  auto go = [&](auto kern) {
    if (smem > 48 * 1024)
      if (cudaError_t e = allow_smem(kern, smem); e != cudaSuccess) return e;
    note_launches(1);
    kern<<<(unsigned)(geo.chunks * splits), warps * 32, smem, st>>>(indptr, idx, static_cast<const ValT*>(val), n,
                                                                    geo.rows, splits, gene2slot, g, map_in_smem, first,
                                                                    tptr, row, static_cast<ValT*>(cval));
    return cudaGetLastError();
  };
  if (splits == 1) return go(k_chunk_csc<ValT, 0>);
  if (cudaError_t e = go(k_chunk_csc<ValT, 1>); e != cudaSuccess) return e;
  note_launches(2);
  k_chunk_sums<<<dim3((unsigned)((g + 255) / 256), (unsigned)geo.chunks), 256, 0, st>>>(splits * warps, g, first, tptr);
  k_chunk_scan<<<(unsigned)geo.chunks, 1024, 0, st>>>(g, tptr);
  if (cudaError_t e = cudaGetLastError(); e != cudaSuccess) return e;
  return go(k_chunk_csc<ValT, 2>);
}

size_t chunk_csc_scratch(const StrictGeometry& geo, int64_t g) {
  return geo.splits == 1 ? 0 : sizeof(int32_t) * (size_t)geo.chunks * geo.splits * csc_warps(geo, g) * g;
}

cudaError_t launch_chunk_csc(int dtype, const int64_t* indptr, const int32_t* idx, const void* val, int64_t n,
                             const StrictGeometry& geo, const int32_t* gene2slot, int32_t g, int32_t* scratch,
                             int32_t* tptr, uint16_t* row, void* cval, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  switch (dtype) {
    case 0: return chunk_csc_t<float>(indptr, idx, val, n, geo, gene2slot, g, scratch, tptr, row, cval, st);
    case 1: return chunk_csc_t<__nv_bfloat16>(indptr, idx, val, n, geo, gene2slot, g, scratch, tptr, row, cval, st);
    default: return chunk_csc_t<__half>(indptr, idx, val, n, geo, gene2slot, g, scratch, tptr, row, cval, st);
  }
}

template <typename ValT>
static cudaError_t fwd_strict_t(int ld, const int64_t* indptr, const int32_t* idx, const void* val, int64_t n,
                                int32_t g, const float* V, const float* mc, float* Y, int lds, cudaStream_t st,
                                int num_sms) {
  const int cols = slice_cols(ld, n, num_sms), nslice = ld / cols;
  const int nch = (g + fwd_table_rows(cols) - 1) / fwd_table_rows(cols);
  const int table_rows = (g + nch - 1) / nch;
  const size_t smem = (size_t)(table_rows + 1) * cols * 4 + kFwdSmemFixed;
  const int64_t want = std::max<int64_t>(1, num_sms / nslice);
  const int64_t per = std::max<int64_t>((n + want - 1) / want, 1);
  const int64_t ranges = (n + per - 1) / per;
  // a caller's matrix may sit at any element: vector loads need both arrays
  // aligned to eight elements (100,000 x 2,000, 25M entries, a product with its
  // copies: 0.36 ms, 0.44 where they are not; 0.76 for either in the layout before)
  const bool vec = (reinterpret_cast<uintptr_t>(idx) & 31) == 0 &&
                   (reinterpret_cast<uintptr_t>(val) & (8 * sizeof(ValT) - 1)) == 0;
  auto go = [&](auto kern) {
    if (cudaError_t e = allow_smem(kern, smem); e != cudaSuccess) return e;
    kern<<<(unsigned)(ranges * nslice), kThreads, smem, st>>>(indptr, idx, static_cast<const ValT*>(val), n, g,
                                                              nslice, per, table_rows, V, mc, Y, lds);
    note_launches(1);
    return cudaGetLastError();
  };
  if (cols == 64) return vec ? go(k_fwd_strict<true, 4, ValT>) : go(k_fwd_strict<false, 4, ValT>);
  return vec ? go(k_fwd_strict<true, 2, ValT>) : go(k_fwd_strict<false, 2, ValT>);
}

cudaError_t launch_fwd_strict(int dtype, int ld, const int64_t* indptr, const int32_t* idx, const void* val,
                              int64_t n, int32_t g, const float* V, const float* mc, float* Y, cudaStream_t st,
                              int num_sms, int lds) {
  if (n == 0) return cudaSuccess;
  if (lds == 0) lds = ld;
  if (lds < ld || (lds & 3) || ld % 32 || ld > kMaxK) return cudaErrorInvalidValue;
  switch (dtype) {
    case 0: return fwd_strict_t<float>(ld, indptr, idx, val, n, g, V, mc, Y, lds, st, num_sms);
    case 1: return fwd_strict_t<__nv_bfloat16>(ld, indptr, idx, val, n, g, V, mc, Y, lds, st, num_sms);
    default: return fwd_strict_t<__half>(ld, indptr, idx, val, n, g, V, mc, Y, lds, st, num_sms);
  }
}

template <typename ValT>
static cudaError_t rmat_strict_t(int ld, const int64_t* indptr, const int32_t* tptr, const uint16_t* row,
                                 const void* cval, int64_t n, int32_t g, const int32_t* slot2gene,
                                 const StrictGeometry& geo, const float* Q, int lds, float* part, cudaStream_t st) {
  const int cols = geo.cols, nslice = ld / cols;
  const size_t smem = (size_t)(geo.rows + 1) * cols * 4;
  auto go = [&](auto kern) {
    if (cudaError_t e = allow_smem(kern, smem); e != cudaSuccess) return e;
    kern<<<dim3((unsigned)(geo.ranges * nslice), (unsigned)geo.parts), kThreads, smem, st>>>(
        indptr, tptr, row, static_cast<const ValT*>(cval), n, g, slot2gene, geo.rows, geo.chunks, geo.per_range, nslice,
        Q, lds, part, ld);
    note_launches(1);
    return cudaGetLastError();
  };
  return cols == 64 ? go(k_rmat_strict<4, ValT>) : go(k_rmat_strict<2, ValT>);
}

cudaError_t launch_rmat_strict(int dtype, int ld, const int64_t* indptr, const int32_t* tptr, const uint16_t* row,
                               const void* cval, int64_t n, int32_t g, const int32_t* slot2gene,
                               const StrictGeometry& geo, const float* Q, float* part, cudaStream_t st, int lds) {
  if (lds == 0) lds = ld;
  if (lds < ld || (lds & 3) || ld % 32 || ld > kMaxK) return cudaErrorInvalidValue;
  switch (dtype) {
    case 0: return rmat_strict_t<float>(ld, indptr, tptr, row, cval, n, g, slot2gene, geo, Q, lds, part, st);
    case 1: return rmat_strict_t<__nv_bfloat16>(ld, indptr, tptr, row, cval, n, g, slot2gene, geo, Q, lds, part, st);
    default: return rmat_strict_t<__half>(ld, indptr, tptr, row, cval, n, g, slot2gene, geo, Q, lds, part, st);
  }
}

}  // namespace scx
