// KKT error evaluation of a given LP point without any device allocation.
//
// Computes, for (x, y, reduced costs) of an LP held in device memory in the user's CSR order, the
// same quantities the solver reports for its own solution (the reference's
// convergence_information_t::compute_convergence_information, cpp/src/pdlp/termination_strategy/
// convergence_information.cu:327-489, restated by term_kernel in kernels.cuh):
//   l2 primal residual  |A x - clamp(A x, lc, uc)|_2
//   l2 dual residual    |c - A^T y - rc|_2
//   primal / dual objective, gap, and the three relative errors.
//
// Who needs it: callers that must check a candidate point while they may not allocate device
// memory — a process whose memory pool is already fully reserved by a larger solve or by another
// framework's caching allocator (where a foreign cudaMalloc fails or fragments the pool), and
// latency-bound loops (heuristics testing many candidate points) where cudaMalloc / cudaFree would
// add an implicit device synchronisation on every call.  The solver's own evaluation builds a
// relabelled matrix layout and per-solve buffers; this variant reads the user's CSR directly and
// keeps its scratch in fixed-size device globals instead (g_na):
//   aty           A^T y accumulator, kNaMaxCols doubles (4 MiB): bounds num_variables; must be zero
//                 before the row pass (cleared on every call);
//   partials      per-block partial sums of the two passes, written in full before they are read;
//   bad, arrived  count of malformed entries (column indices outside [0, n), rows whose offsets
//                 decrease or start below 0), and the blocks of the column pass that have
//                 finished; zero before the row pass (cleared on every call).
// Because the scratch is one static copy per device, calls that overlap in time on the same
// device (different streams or host threads without ordering between them) race on it and give
// wrong results; callers must order them.  A^T y is accumulated with double-precision atomics, so
// the dual residual and the quantities derived from it may differ in the last bits between calls.
// The scratch belongs to this library's device code, which the CUDA runtime loads on a device at
// the first call that needs it (lazily, by default): that first call is when the static arrays take
// their device memory.
#include <math_constants.h>

#include <algorithm>
#include <cstddef>
#include <cstdio>

#include <cuopt_b200.h>

#include "common.cuh"

namespace cuopt_b200 {
namespace {

constexpr int kBlock     = 256;
constexpr int kNaMaxCols = 1 << 19;  // 524,288 columns
constexpr int kNaBlocks  = 1184;     // 148 SMs x 8 resident blocks of 256 threads
constexpr int kNaRowRed  = 3;        // row pass: |r_p|^2, dual row term, |b|^2
constexpr int kNaColRed  = 4;        // column pass: |r_d|^2, c.x, rc.x, |c|^2
// Small LPs run in one cluster of kNaClusterBlocks blocks: one launch in place of a memset and two
// kernels.  The line is drawn on m n, which bounds the non-zeros (the host does not know them), and on
// n / m, because few long rows leave most of the eight SMs idle.  One cluster / kernels / the memset
// and three kernels of one warp per row that these replaced, us: 300 x 873 with 2 400 entries 10.5 /
// 12.7 / 21.9, dense 29 / 23 / 36; 4096 x 64 with 32 768 17.7 / 20.8 / 28.8; dense 512 x 512 28 / 25 /
// 36; beyond the line 64 x 4096 with 65 536 37 / 19 / 34, dense 1000 x 1000 68 / 44 / 57.
constexpr int kNaClusterBlocks   = 8;
constexpr int kNaClusterThreads  = 1024;
constexpr int64_t kNaClusterArea = 1 << 18;
constexpr int kNaClusterAspect   = 32;

struct na_globals {
  unsigned bad, arrived;  // the clear of a call covers these and the first n entries of aty
  double aty[kNaMaxCols];
  double partials[kNaBlocks * (kNaRowRed + kNaColRed)];
};
static __device__ __align__(256) na_globals g_na;

struct na_problem {
  int m, n;
  const int* off;
  const int* idx;
  const double* val;
  const double *c, *lo, *up, *x, *y, *rc;
  double sgn, offset;
  double* out;
};

__device__ __forceinline__ double fin0(double v) { return isfinite(v) ? v : 0.0; }

// Block sum of K per-thread values (fixed order); thread q < K writes partials[block * K + q].
template <int K, int THREADS>
__device__ __forceinline__ void block_sum_store(const double (&v)[K], double* partials, int block)
{
  constexpr int W = THREADS / kWarp;
  __shared__ double sm[W][K];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const double w = warp_sum(v[q]);
    if (lane == 0) sm[warp][q] = w;
  }
  __syncthreads();
  if (threadIdx.x < K) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < W; ++w) t += sm[w][threadIdx.x];
    partials[(size_t)block * K + threadIdx.x] = t;
  }
}

// Entries b + first, b + first + STRIDE, ... of one row: this lane's part of A x, and the scatter of
// yi A[i, :] into the A^T y accumulator.  Four at a time, so that their loads, then their gathers, are
// in flight together.  The count left is signed, the position is not: neither wraps near 2^31 entries.
template <int STRIDE>
__device__ __forceinline__ double na_row_part(const na_problem& p, int b, int e, int first, double yi)
{
  double ax = 0.0;
  unsigned k = (unsigned)b + first;
  for (int left = e - b - first; left > 0; left -= 4 * STRIDE, k += 4 * STRIDE) {
    int j[4];
    double a[4], xj[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) j[q] = q * STRIDE < left ? p.idx[k + q * STRIDE] : -1;
#pragma unroll
    for (int q = 0; q < 4; ++q) a[q] = q * STRIDE < left ? p.val[k + q * STRIDE] : 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) xj[q] = (unsigned)j[q] < (unsigned)p.n ? p.x[j[q]] : 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if ((unsigned)j[q] < (unsigned)p.n) {
        ax += a[q] * xj[q];
        atomicAdd(g_na.aty + j[q], a[q] * yi);
      } else if (q * STRIDE < left) {
        atomicAdd(&g_na.bad, 1u);
      }
    }
  }
  return ax;
}

// G lanes per constraint row: A x and the row's residual / dual-objective / |b| terms, and the
// scatter of y_i A[i, :] into the A^T y accumulator.  Bound by the L1 request rate (one gather and
// one reduction per non-zero), so rows shorter than a warp share one: with a whole warp per row of
// 20 non-zeros 12 of 32 lanes issued nothing.  A row of more than kNaLongRounds rounds of its G lanes
// is left to the whole warp, which takes such rows of its groups one after another: the longest row
// sets the time of the pass (one of 50 000 entries among 20 000 rows of 8: 1 730 us on 4 lanes, 227 us
// on the warp).
constexpr int kNaLongRounds = 8;
template <int G>
__device__ __forceinline__ void na_rows(const na_problem& p, int warp0, int nwarps,
                                        double (&r)[kNaRowRed])
{
  constexpr int kRows = kWarp / G;  // rows per warp
  const int lane = threadIdx.x & 31, sub = lane & (G - 1), grp = lane / G;
  for (int i0 = warp0 * kRows; i0 < p.m; i0 += nwarps * kRows) {
    const int i = i0 + grp;
    bool live   = i < p.m;
    int b = 0, e = 0;
    double yi = 0.0, l = 0.0, u = 0.0;
    if (live) {
      b  = p.off[i];
      e  = p.off[i + 1];
      yi = p.y[i];
      l  = p.lo[i];
      u  = p.up[i];
      if (b < 0 || e < b) {  // malformed offsets: counted, the row is skipped
        if (sub == 0) atomicAdd(&g_na.bad, 1u);
        live = false;
        b = e = 0;
      }
    }
    const bool longer = G < kWarp && e - b > kNaLongRounds * 4 * G;
    double ax         = longer ? 0.0 : na_row_part<G>(p, b, e, sub, yi);
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) ax += __shfl_xor_sync(0xffffffffu, ax, o);
    if constexpr (G < kWarp) {
      for (unsigned left = __ballot_sync(0xffffffffu, longer && sub == 0); left; left &= left - 1) {
        const int from  = __ffs(left) - 1;
        const int lb    = __shfl_sync(0xffffffffu, b, from), le = __shfl_sync(0xffffffffu, e, from);
        const double ly = __shfl_sync(0xffffffffu, yi, from);
        const double t  = warp_sum(na_row_part<kWarp>(p, lb, le, lane, ly));
        if (lane == from) ax = t;
      }
    }
    if (sub == 0 && live) {
      const double rp   = ax - fmax(l, fmin(ax, u));
      const double yint = p.sgn * yi;  // the dual in minimisation form
      r[0] += rp * rp;
      r[1] += fmax(yint, 0.0) * fin0(l) + fmin(yint, 0.0) * fin0(u);
      r[2] += ((isfinite(l) && l != u) ? l * l : 0.0) + (isfinite(u) ? u * u : 0.0);
    }
  }
}

// The row pass of block `block` of `nblocks`; the lanes per row follow the mean row length.  A block
// takes neighbouring rows; in the one cluster, short rows are dealt to the blocks (300 x 873 with 2 400
// entries: 12.6 -> 10.5 us), but long ones then meet in their atomics (dense: 29 -> 41 us).
template <int THREADS>
__device__ __forceinline__ void na_row_pass(const na_problem& p, int block, int nblocks)
{
  constexpr int W      = THREADS / kWarp;
  double r[kNaRowRed]  = {};
  const int warp       = threadIdx.x >> 5;
  const int mean       = p.off[p.m] / p.m;
  const int neighbours = block * W + warp;
  const int dealt      = THREADS == kNaClusterThreads ? warp * nblocks + block : neighbours;
  if (mean <= 12)
    na_rows<4>(p, dealt, nblocks * W, r);
  else if (mean <= 48)
    na_rows<8>(p, dealt, nblocks * W, r);
  else
    na_rows<32>(p, neighbours, nblocks * W, r);
  block_sum_store<kNaRowRed, THREADS>(r, g_na.partials, block);
}

// Thread per variable: dual residual and objective terms.
template <int THREADS>
__device__ __forceinline__ void na_col_pass(const na_problem& p, int block, int nblocks)
{
  double r[kNaColRed] = {};
  for (int j = block * THREADS + threadIdx.x; j < p.n; j += nblocks * THREADS) {
    const double cj = p.c[j], xj = p.x[j], sj = p.rc[j];
    const double rd = (cj - __ldcg(g_na.aty + j)) - sj;
    r[0] += rd * rd;
    r[1] += cj * xj;
    r[2] += sj * xj;
    r[3] += cj * cj;
  }
  block_sum_store<kNaColRed, THREADS>(r, g_na.partials + kNaBlocks * kNaRowRed, block);
}

// One block: ordered, compensated sums over the block partials (a warp for each quantity), then
// the reported quantities.  The partials come from other blocks of the launch: read through L2.
__device__ __forceinline__ void na_finish(const na_problem& p, int row_blocks, int col_blocks)
{
  __shared__ double tot[kNaRowRed + kNaColRed];
  const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (q < kNaRowRed + kNaColRed) {
    const bool row_q   = q < kNaRowRed;
    const int K        = row_q ? kNaRowRed : kNaColRed;
    const int nb       = row_q ? row_blocks : col_blocks;
    const double* base = g_na.partials + (row_q ? q : kNaBlocks * kNaRowRed + q - kNaRowRed);
    ksum acc;
#pragma unroll 4
    for (int b = lane; b < nb; b += kWarp) acc.add(__ldcg(base + (size_t)b * K));
    const double t = warp_sum(acc.value());
    if (lane == 0) tot[q] = t;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double rp2 = tot[0], drow = tot[1], b2 = tot[2];
    const double rd2 = tot[3], cx = tot[4], sx = tot[5], c2 = tot[6];
    const double l2p = sqrt(rp2), l2d = sqrt(rd2);
    const double primal = cx + p.offset;
    const double dual   = p.sgn * (drow + p.sgn * sx) + p.offset;
    const double gap    = fabs(primal - dual);
    const unsigned bad  = __ldcg(&g_na.bad);
    const double vals[8] = {l2p, l2d, primal, dual, gap, l2p / (1.0 + sqrt(b2)),
                            l2d / (1.0 + sqrt(c2)), gap / (1.0 + fabs(primal) + fabs(dual))};
    for (int k = 0; k < 8; ++k) p.out[k] = bad ? CUDART_NAN : vals[k];
    p.out[8] = (double)bad;
  }
}

__global__ void __launch_bounds__(kBlock) na_rows_kernel(const na_problem p)
{
  na_row_pass<kBlock>(p, (int)blockIdx.x, (int)gridDim.x);
}

// The column pass; the block that finishes last forms the results.
__global__ void __launch_bounds__(kBlock) na_cols_kernel(const na_problem p, int row_blocks)
{
  na_col_pass<kBlock>(p, (int)blockIdx.x, (int)gridDim.x);
  __shared__ int last;
  __syncthreads();  // threads 0 .. kNaColRed - 1 wrote the block's partials
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&g_na.arrived, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  na_finish(p, row_blocks, (int)gridDim.x);
}

// The whole evaluation in one cluster: clear, row pass, column pass, results, a cluster barrier
// (hardware, no polling) between them.
__device__ __forceinline__ void na_cluster_barrier()
{
  __threadfence();
  asm volatile(
    "barrier.cluster.arrive.release;\n"
    "barrier.cluster.wait.acquire;\n" ::
      : "memory");
}
__global__ void __cluster_dims__(kNaClusterBlocks, 1, 1) __launch_bounds__(kNaClusterThreads)
  na_small_kernel(const na_problem p)
{
  const int block = (int)blockIdx.x;
  for (int j = block * kNaClusterThreads + threadIdx.x; j < p.n;
       j += kNaClusterBlocks * kNaClusterThreads)
    g_na.aty[j] = 0.0;
  if (block == 0 && threadIdx.x == 0) g_na.bad = 0;
  na_cluster_barrier();
  na_row_pass<kNaClusterThreads>(p, block, kNaClusterBlocks);
  na_cluster_barrier();
  na_col_pass<kNaClusterThreads>(p, block, kNaClusterBlocks);
  na_cluster_barrier();
  if (block == 0) na_finish(p, kNaClusterBlocks, kNaClusterBlocks);
}

}  // namespace
}  // namespace cuopt_b200

extern "C" cuopt_int_t cuOptComputeKKTErrorsNoAlloc(
  cuopt_int_t m, cuopt_int_t n, cuopt_int_t sense, cuopt_float_t offset, const cuopt_float_t* d_c,
  const cuopt_int_t* d_off, const cuopt_int_t* d_idx, const cuopt_float_t* d_val,
  const cuopt_float_t* d_lo, const cuopt_float_t* d_up, const cuopt_float_t* d_x,
  const cuopt_float_t* d_y, const cuopt_float_t* d_rc, void* stream, cuopt_float_t* d_out)
{
  using namespace cuopt_b200;
  if (!d_c || !d_off || !d_idx || !d_val || !d_lo || !d_up || !d_x || !d_y || !d_rc || !d_out)
    return CUOPT_INVALID_ARGUMENT;
  if (m <= 0 || n <= 0) return CUOPT_INVALID_ARGUMENT;
  if (sense != CUOPT_MINIMIZE && sense != CUOPT_MAXIMIZE) return CUOPT_INVALID_ARGUMENT;
  if (n > kNaMaxCols) {
    std::fprintf(stderr,
                 "cuOptComputeKKTErrorsNoAlloc: num_variables = %d exceeds the static scratch "
                 "capacity of %d variables\n",
                 (int)n, kNaMaxCols);
    return CUOPT_INVALID_ARGUMENT;
  }
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  const double sgn      = sense == CUOPT_MAXIMIZE ? -1.0 : 1.0;
  const na_problem p{m, n, d_off, d_idx, d_val, d_c, d_lo, d_up, d_x, d_y, d_rc, sgn, offset, d_out};
  if ((int64_t)m * n <= kNaClusterArea && n <= (int64_t)kNaClusterAspect * m) {
    na_small_kernel<<<kNaClusterBlocks, kNaClusterThreads, 0, st>>>(p);
  } else {
    // The scratch's address is looked up on every call (a host query that allocates nothing), so
    // that a device reset or a new primary context, after which the module is loaded again at a
    // new address, never leaves a stale one behind.
    void* scratch = nullptr;
    if (cudaGetSymbolAddress(&scratch, g_na) != cudaSuccess) {
      std::fprintf(stderr, "cuOptComputeKKTErrorsNoAlloc: scratch lookup failed\n");
      return CUOPT_RUNTIME_ERROR;
    }
    if (cudaMemsetAsync(scratch, 0, offsetof(na_globals, aty) + (size_t)n * sizeof(double), st) !=
        cudaSuccess)
      return CUOPT_RUNTIME_ERROR;
    const int row_blocks = std::min(kNaBlocks, ceil_div(m, kBlock / kWarp));
    const int col_blocks = std::min(kNaBlocks, ceil_div(n, kBlock));
    na_rows_kernel<<<row_blocks, kBlock, 0, st>>>(p);
    na_cols_kernel<<<col_blocks, kBlock, 0, st>>>(p, row_blocks);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    std::fprintf(stderr, "cuOptComputeKKTErrorsNoAlloc: %s\n", cudaGetErrorString(e));
    return CUOPT_RUNTIME_ERROR;
  }
  return CUOPT_SUCCESS;
}
