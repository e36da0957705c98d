// sm_100a kernels of the PDLP path.
//
// Every matrix sweep is one launch of `sell_map_kernel`: warps either walk one long row (CSR,
// lanes stride along the row) or one 32-row slice of the sliced-ELL part (lane t owns row t and
// reads element k at base + 32k + t, so each warp load is one contiguous segment).  The row's dot
// product is handed to an epilogue functor that performs the PDHG projection / reflection /
// Halpern step (or a termination / fixed-point-error term) for that row, so x, y and the reflected
// iterate cross HBM once per sweep.  Epilogues may also contribute to up to four block-level sums
// that are reduced deterministically (fixed tree, then one ordered pass over blocks).
#pragma once

#include <type_traits>

#include "common.cuh"

namespace cuopt_b200 {

constexpr int kBlock         = 256;
constexpr int kWarpsPerBlock = kBlock / kWarp;

template <typename T>
struct dev_sell {
  int rows;
  int n_long;
  int n_slices;
  const int64_t* long_off;
  const int64_t* slice_off;
  const int* idx;
  const T* val;
  // Optional work lists (block-diagonal batches with finished instances): when set, a sweep visits
  // only the listed long rows / slices, work_long / work_slices of them.
  const int* long_list  = nullptr;
  const int* slice_list = nullptr;
  int work_long         = 0;
  int work_slices       = 0;
  int n_wide            = 0;  // the first n_wide long rows are taken by kWideStrands warps each
  B200_HD int long_count() const { return long_list ? work_long : n_long; }
  B200_HD int wide_count() const { return long_list ? 0 : n_wide; }
  B200_HD int slice_count() const { return slice_list ? work_slices : n_slices; }
};

B200_HD inline int long_blocks(int n_long, int wpb = kWarpsPerBlock) { return ceil_div(n_long, wpb); }
// Grid of the kernels that take every long row with one warp (setup, climbers).
template <typename T>
inline int sell_grid(const dev_sell<T>& a, int wpb = kWarpsPerBlock)
{
  const int g = long_blocks(a.long_count(), wpb) + ceil_div(a.slice_count(), wpb);
  return g > 0 ? g : 1;  // an empty work list still launches one (idle) block
}
// Wide rows: a row of a few thousand elements on one warp is a chain of some 150 dependent load
// rounds, which a sweep waits for when the rest of it is done (20k x 60k LP, Zipf rows up to 5000
// long: 38 of 50 us an iteration).  So rows longer than kWideRow elements (a sixteenth of such a
// chain) are cut into kWideStrands strands, lane l of strand s taking elements 256 t + 32 s + l,
// whose sums are added in strand order: by the 8 warps of a block (or half block of 16 warps), or by
// one warp (where a block has fewer, in the cluster-resident form, in batches and for climbers).  Every
// form of the sweeps adds them in the same order, so iterates do not depend on the form.
constexpr int kWideStrands = 8;
B200_HD inline int wide_blocks(int n_wide, int wpb = kWarpsPerBlock)
{
  return wpb >= kWideStrands ? ceil_div(n_wide, wpb / kWideStrands) : ceil_div(n_wide, wpb);
}
// Blocks of a sweep (sell_map_block) before its slices, and all of them.
template <typename T>
B200_HD inline int row_blocks(const dev_sell<T>& a, int wpb = kWarpsPerBlock)
{
  return wide_blocks(a.wide_count(), wpb) + long_blocks(a.long_count() - a.wide_count(), wpb);
}
template <typename T>
B200_HD inline int sweep_grid(const dev_sell<T>& a, int wpb = kWarpsPerBlock)
{
  const int g = row_blocks(a, wpb) + ceil_div(a.slice_count(), wpb);
  return g > 0 ? g : 1;
}

// Scalars that change between iterations live on the device so captured graphs stay valid.
struct pdlp_scalars {
  double tau;      // primal step  = eta / omega
  double sigma;    // dual step    = eta * omega
  double eta;      // step size
  double omega;    // primal weight
  long long t0;    // iterations since the last restart, at the start of the next step
};

__device__ __forceinline__ double halpern_weight(const pdlp_scalars* st, int it_off)
{
  const double t = (double)(st->t0 + it_off);
  return (t + 1.0) / (t + 2.0);
}

// The Halpern step w v + (1 - w) anchor, rounded the same way in every form of the iterations (left
// to the compiler, which of the two products was fused depended on the kernel).  The fused step of y
// takes the other product than the one of x: these are the roundings that the graphs' kernels always
// had, and a mixed-precision solve of a million rows shows a difference in the last bit.
__device__ __forceinline__ double halpern_mix(double w, double v, double anchor)
{
  return fma(w, v, (1.0 - w) * anchor);
}
__device__ __forceinline__ double halpern_mix_y(double w, double v, double anchor)
{
  return fma(1.0 - w, anchor, w * v);
}

template <int K>
struct red_t {
  double v[K > 0 ? K : 1];
};

// Block reduction of K doubles (sums, or maxima when MAX); threads 0..K-1 write
// partials[slot * K + r].
template <int K, bool MAX = false>
__device__ __forceinline__ void block_reduce_store(red_t<K>& r, double* partials, int slot)
{
  if constexpr (K > 0) {
    __shared__ double sm[kWarpsPerBlock][K];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < K; ++q) {
      double v = MAX ? warp_max(r.v[q]) : warp_sum(r.v[q]);
      if (lane == 0) sm[warp][q] = v;
    }
    __syncthreads();
    if (threadIdx.x < K) {
      double s = MAX ? sm[0][threadIdx.x] : 0.0;
#pragma unroll
      for (int w = 0; w < kWarpsPerBlock; ++w)
        s = MAX ? fmax(s, sm[w][threadIdx.x]) : s + sm[w][threadIdx.x];
      partials[(size_t)slot * K + threadIdx.x] = s;
    }
  }
}
template <int K, bool MAX = false>
__device__ __forceinline__ void block_reduce_store(red_t<K>& r, double* partials)
{
  block_reduce_store<K, MAX>(r, partials, (int)blockIdx.x);
}

// Epilogues may declare `static constexpr bool kMaxRed = true`: their block values are then
// combined by maxima instead of sums.
template <class E, class = void>
struct has_max_red : std::false_type {};
template <class E>
struct has_max_red<E, std::void_t<decltype(E::kMaxRed)>> : std::bool_constant<E::kMaxRed> {};

// out[q] = sum over blocks of partials[b*K+q], summed by one block (ordered, compensated).  L2: the
// partials were written by other blocks of the same launch, so they are read through L2.
template <int K, bool L2 = false>
__device__ __forceinline__ void ordered_block_sum(const double* partials, int nblocks, double* out)
{
  __shared__ double sm[kBlock];
  for (int q = 0; q < K; ++q) {
    ksum acc;
    for (int b = threadIdx.x; b < nblocks; b += kBlock) {
      const double* p = partials + (size_t)b * K + q;
      acc.add(L2 ? __ldcg(p) : *p);
    }
    sm[threadIdx.x] = acc.value();
    __syncthreads();
    for (int s = kBlock / 2; s > 0; s >>= 1) {
      if (threadIdx.x < s) sm[threadIdx.x] += sm[threadIdx.x + s];
      __syncthreads();
    }
    if (threadIdx.x == 0) out[q] = sm[0];
    __syncthreads();
  }
}
template <int K>
__global__ void __launch_bounds__(kBlock) finalize_sum_kernel(const double* partials, int nblocks,
                                                              double* out)
{
  ordered_block_sum<K>(partials, nblocks, out);
}

// p[0 .. n) = v.
static __global__ void fill_kernel(double* p, int n, double v)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = v;
}

// out[q] = max over blocks of partials[b*K+q] (single block).
template <int K>
__global__ void __launch_bounds__(kBlock) finalize_max_kernel(const double* partials, int nblocks,
                                                              double* out)
{
  __shared__ double sm[kBlock];
  for (int q = 0; q < K; ++q) {
    double v = -INFINITY;
    for (int b = threadIdx.x; b < nblocks; b += kBlock) v = fmax(v, partials[(size_t)b * K + q]);
    sm[threadIdx.x] = v;
    __syncthreads();
    for (int s = kBlock / 2; s > 0; s >>= 1) {
      if (threadIdx.x < s) sm[threadIdx.x] = fmax(sm[threadIdx.x], sm[threadIdx.x + s]);
      __syncthreads();
    }
    if (threadIdx.x == 0) out[q] = sm[0];
    __syncthreads();
  }
}

// 4 consecutive values of one lane chunk (16-byte aligned), streamed with evict-first loads.
__device__ __forceinline__ void load_chunk(const float* p, double (&v)[4])
{
  const float4 t = __ldcs(reinterpret_cast<const float4*>(p));
  v[0]           = t.x;
  v[1]           = t.y;
  v[2]           = t.z;
  v[3]           = t.w;
}
__device__ __forceinline__ void load_chunk(const double* p, double (&v)[4])
{
  const double2 a = __ldcs(reinterpret_cast<const double2*>(p));
  const double2 b = __ldcs(reinterpret_cast<const double2*>(p) + 1);
  v[0]            = a.x;
  v[1]            = a.y;
  v[2]            = b.x;
  v[3]            = b.y;
}
__device__ __forceinline__ int4 load_idx_chunk(const int* p)
{
  return __ldcs(reinterpret_cast<const int4*>(p));
}

// Epilogues of block-diagonal batches may declare `bool skip_range(int r0, int r1)`: true when
// rows r0..r1 belong only to finished instances, so a warp can skip their dot products.
template <class E, class = void>
struct has_skip_range : std::false_type {};
template <class E>
struct has_skip_range<E, std::void_t<decltype(&E::skip_range)>> : std::true_type {};

template <class Epi>
__device__ __forceinline__ bool skip_rows(const Epi& epi, int r0, int r1)
{
  if constexpr (has_skip_range<Epi>::value)
    return epi.skip_range(r0, r1);
  else
    return false;
}

// Generic fused sweep: acc_r = sum_k A[r,k] * g[idx[r,k]], then epi(r, acc_r, pre, red).
// The epilogue's per-row operands (`pre`) are loaded before the matrix loop so their memory latency
// overlaps the gathers.  Sliced rows are read in 4-element lane chunks, two chunks in flight.
// `vb` is the block's index in the sweep's grid (blockIdx.x, or a virtual index in a persistent
// kernel that walks the grid).
// Gathered-vector loads.  A kernel that writes the gathered vector itself (the persistent
// iterations below) reads it through L2 (ld.global.cg), which its grid barrier keeps coherent;
// every other sweep uses plain loads of the restrict-qualified vector, which no sweep writes
// (an explicit __ldg measured slower on the mixed-precision primal sweep: 73.1 against 69.9 us on
// the 1M x 2M LP).
template <bool COH, typename T>
__device__ __forceinline__ T gather_load(const T* __restrict__ g, int i)
{
  if constexpr (COH)
    return __ldcg(g + i);
  else
    return g[i];
}

// Sum over elements k = first, first + STRIDE, ... below `end` of a row, in that order: U of them
// are loaded at a time (also the last, incomplete batch), so a row is a chain of ceil(count / U)
// rounds of two dependent loads and not of one per element left over.
template <int U, int STRIDE, bool COH, typename TM, typename TG>
__device__ __forceinline__ double strided_product(const dev_sell<TM>& A, const TG* __restrict__ g,
                                                  int64_t first, int64_t end)
{
  double acc = 0.0;
  for (int64_t k = first; k < end; k += U * STRIDE) {
    const int left = (int)(end - k);
    int x[U];
    TM v[U];
    TG w[U];
#pragma unroll
    for (int q = 0; q < U; ++q) x[q] = q * STRIDE < left ? ld_stream(A.idx + k + q * STRIDE) : 0;
#pragma unroll
    for (int q = 0; q < U; ++q)
      if (q * STRIDE < left) v[q] = ld_stream(A.val + k + q * STRIDE);
#pragma unroll
    for (int q = 0; q < U; ++q)
      if (q * STRIDE < left) w[q] = gather_load<COH>(g, x[q]);
#pragma unroll
    for (int q = 0; q < U; ++q)
      if (q * STRIDE < left) acc += (double)v[q] * (double)w[q];
  }
  return acc;
}
// The strands of a wide row: this warp's, and all of them on one warp.
template <bool COH, typename TM, typename TG>
__device__ __forceinline__ double wide_strand(const dev_sell<TM>& A, const TG* __restrict__ g,
                                              int64_t b, int64_t e, int strand)
{
  return warp_sum(strided_product<4, kWideStrands * kWarp, COH>(
    A, g, b + strand * kWarp + (threadIdx.x & 31), e));
}
template <class Load>
__device__ __forceinline__ double wide_row_by_warp(int len, Load&& term)
{
  double acc[kWideStrands];
#pragma unroll
  for (int q = 0; q < kWideStrands; ++q) acc[q] = 0.0;
  for (int k = threadIdx.x & 31; k < len; k += kWideStrands * kWarp)
#pragma unroll
    for (int q = 0; q < kWideStrands; ++q)
      if (k + q * kWarp < len) term(k + q * kWarp, acc[q]);
  double sum = 0.0;
#pragma unroll
  for (int q = 0; q < kWideStrands; ++q) sum += warp_sum(acc[q]);
  return sum;
}
// Barrier of one group (0 or 1) of kWideStrands warps of the block.  The barriers are named by
// constants: with a register, the compiler reserves all 16 for the block.
__device__ __forceinline__ void wide_barrier(int group)
{
  if (group == 0)
    asm volatile("bar.sync 1, %0;" ::"n"(kWideStrands* kWarp) : "memory");
  else
    asm volatile("bar.sync 2, %0;" ::"n"(kWideStrands* kWarp) : "memory");
}

// WPB: warps (rows or slices) per block.  Only the grouping of warps into blocks depends on it,
// not any row's arithmetic; sweeps with block reductions (kRed > 0) use kWarpsPerBlock.
template <typename TM, typename TG, class Epi, bool COH = false, int WPB = kWarpsPerBlock>
__device__ __forceinline__ void sell_map_block(const dev_sell<TM>& A, const TG* __restrict__ g,
                                               const Epi& epi, double* partials, int vb)
{
  constexpr int K = Epi::kRed;
  static_assert(K == 0 || WPB == kWarpsPerBlock, "block reductions assume kWarpsPerBlock warps");
  red_t<K> red;
#pragma unroll
  for (int q = 0; q < (K > 0 ? K : 1); ++q) red.v[q] = 0.0;
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) & (WPB - 1);
  const int wb   = wide_blocks(A.wide_count(), WPB);
  const int lb   = row_blocks(A, WPB);
  if (vb < wb) {
    if constexpr (WPB >= kWideStrands) {
      __shared__ double strands[2][kWideStrands];
      static_assert(WPB <= 2 * kWideStrands, "two groups of strands");
      const int group = threadIdx.x / (kWideStrands * kWarp), strand = warp & (kWideStrands - 1);
      const int row   = vb * (WPB / kWideStrands) + warp / kWideStrands;
      if (row < A.wide_count()) {
        const auto pre = epi.load(row);
        const double t = wide_strand<COH>(A, g, A.long_off[row], A.long_off[row + 1], strand);
        wide_barrier(group);  // the sums of the group's row before have been read
        if (lane == 0) strands[group][strand] = t;
        wide_barrier(group);
        if (strand == 0 && lane == 0) {
          double acc = 0.0;
#pragma unroll
          for (int q = 0; q < kWideStrands; ++q) acc += strands[group][q];
          epi(row, acc, pre, red);
        }
      }
    } else {
      const int row = vb * WPB + warp;
      if (row < A.wide_count()) {
        const auto pre  = epi.load(row);
        const int64_t b = A.long_off[row];
        const double acc =
          wide_row_by_warp((int)(A.long_off[row + 1] - b), [&](int k, double& a) {
            a += (double)ld_stream(A.val + b + k) *
                 (double)gather_load<COH>(g, ld_stream(A.idx + b + k));
          });
        if (lane == 0) epi(row, acc, pre, red);
      }
    }
  } else if (vb < lb) {
    const int q   = A.wide_count() + (vb - wb) * WPB + warp;
    const int row = q < A.long_count() ? (A.long_list ? A.long_list[q] : q) : 0;
    if (q < A.long_count() && !skip_rows(epi, row, row)) {
      const auto pre  = epi.load(row);
      const int64_t b = A.long_off[row], e = A.long_off[row + 1];
      double acc = 0.0;
      // In batches the wide rows are not the first ones: one warp takes each, strand after strand.
      if (has_skip_range<Epi>::value && e - b > kWideRow)
        for (int q = 0; q < kWideStrands; ++q) acc += wide_strand<COH>(A, g, b, e, q);
      else
        acc = warp_sum(strided_product<4, kWarp, COH>(A, g, b + lane, e));
      if (lane == 0) epi(row, acc, pre, red);
    }
  } else {
    const int q = (vb - lb) * WPB + warp;
    const int s = q < A.slice_count() ? (A.slice_list ? A.slice_list[q] : q) : 0;
    if (q < A.slice_count() &&
        !skip_rows(epi, A.n_long + s * kWarp, min(A.n_long + s * kWarp + kWarp, A.rows) - 1)) {
      const int row      = A.n_long + s * kWarp + lane;
      const bool valid   = row < A.rows;
      const auto pre     = epi.load(valid ? row : A.rows - 1);
      const int64_t base = A.slice_off[s];
      const int nchunk   = (int)((A.slice_off[s + 1] - base) >> 7);  // 32 lanes x 4 elements
      const TM* v        = A.val + base + lane * kChunk;
      const int* ix      = A.idx + base + lane * kChunk;
      double acc         = 0.0;
      // Two chunks at a time; the indices of the next two are loaded while these are gathered, so a
      // round waits for its gathers alone.
      int4 i0 = make_int4(0, 0, 0, 0), i1 = i0;
      if (nchunk > 0) i0 = load_idx_chunk(ix);
      if (nchunk > 1) i1 = load_idx_chunk(ix + 32 * kChunk);
      int q = 0;
      for (; q + 2 <= nchunk; q += 2) {
        double v0[4], v1[4];
        load_chunk(v, v0);
        load_chunk(v + 32 * kChunk, v1);
        const TG g0 = gather_load<COH>(g, i0.x), g1 = gather_load<COH>(g, i0.y);
        const TG g2 = gather_load<COH>(g, i0.z), g3 = gather_load<COH>(g, i0.w);
        const TG g4 = gather_load<COH>(g, i1.x), g5 = gather_load<COH>(g, i1.y);
        const TG g6 = gather_load<COH>(g, i1.z), g7 = gather_load<COH>(g, i1.w);
        v += 64 * kChunk;
        ix += 64 * kChunk;
        if (q + 2 < nchunk) i0 = load_idx_chunk(ix);
        if (q + 3 < nchunk) i1 = load_idx_chunk(ix + 32 * kChunk);
        acc += v0[0] * (double)g0;
        acc += v0[1] * (double)g1;
        acc += v0[2] * (double)g2;
        acc += v0[3] * (double)g3;
        acc += v1[0] * (double)g4;
        acc += v1[1] * (double)g5;
        acc += v1[2] * (double)g6;
        acc += v1[3] * (double)g7;
      }
      if (q < nchunk) {
        double v0[4];
        load_chunk(v, v0);
        const TG g0 = gather_load<COH>(g, i0.x), g1 = gather_load<COH>(g, i0.y);
        const TG g2 = gather_load<COH>(g, i0.z), g3 = gather_load<COH>(g, i0.w);
        acc += v0[0] * (double)g0;
        acc += v0[1] * (double)g1;
        acc += v0[2] * (double)g2;
        acc += v0[3] * (double)g3;
      }
      if (valid) epi(row, acc, pre, red);
    }
  }
  block_reduce_store<K, has_max_red<Epi>::value>(red, partials, vb);
}

// Resident blocks of 256 threads the sweeps are compiled for: 5 an SM with FP32 matrices (48
// registers), 3 with FP64 (80).  FP64, 1M x 2M LP with 16M non-zeros, primal + dual sweep: 86.4 + 81.1
// us at 4 blocks (64 registers), 86.5 + 78.9 at 3, 95.2 + 86.9 left alone; 400k x 1M: 45.1 + 45.8, 45.0
// + 43.2, 48.3 + 47.0.  FP32, 1M x 2M: 71.8 + 73.3 at 5, 74.4 + 73.1 at 4.
// Batches, whose gathers hit L1, want the warps instead: 4 in FP64 (512 LPs with 51.6M non-zeros,
// primal sweep 215 us, 231 at 3).
template <typename TM, class Epi>
constexpr int kSweepBlocks = sizeof(TM) == 4 ? 5 : has_skip_range<Epi>::value ? 4 : 3;
template <typename TM, typename TG, class Epi>
__global__ void __launch_bounds__(kBlock, kSweepBlocks<TM, Epi>) sell_map_kernel(const dev_sell<TM> A,
                                                          const TG* __restrict__ g, Epi epi,
                                                          double* partials)
{
  sell_map_block(A, g, epi, partials, (int)blockIdx.x);
}

// Blocks vb0, vb0 + 1, ... of a sweep's grid only (measurement of one row-length class: the
// long rows are blocks [0, long_blocks), the slices the rest).
template <typename TM, typename TG, class Epi>
__global__ void __launch_bounds__(kBlock, kSweepBlocks<TM, Epi>) sell_map_range_kernel(const dev_sell<TM> A,
                                                                const TG* __restrict__ g, Epi epi,
                                                                double* partials, int vb0)
{
  sell_map_block(A, g, epi, partials, vb0 + (int)blockIdx.x);
}

// The same sweep with WPB warps per block (the plain sweeps' block shape is autotuned).
template <typename TM, typename TG, class Epi, int WPB>
__global__ void __launch_bounds__(WPB * kWarp, kSweepBlocks<TM, Epi> * kWarpsPerBlock / WPB)
  sell_map_wpb_kernel(const dev_sell<TM> A, const TG* __restrict__ g, Epi epi, double* partials)
{
  sell_map_block<TM, TG, Epi, false, WPB>(A, g, epi, partials, (int)blockIdx.x);
}

// Launches sell_map_wpb_kernel with wpb (4, 8 or 16) warps per block.
template <typename TM, typename TG, class Epi>
void launch_sell_wpb(int wpb, const dev_sell<TM>& A, const TG* g, const Epi& epi,
                     double* partials, cudaStream_t s)
{
  const int grid = sweep_grid(A, wpb);
  switch (wpb) {
    case 4:
      sell_map_wpb_kernel<TM, TG, Epi, 4><<<grid, 4 * kWarp, 0, s>>>(A, g, epi, partials);
      break;
    case 16:
      sell_map_wpb_kernel<TM, TG, Epi, 16><<<grid, 16 * kWarp, 0, s>>>(A, g, epi, partials);
      break;
    default:
      sell_map_kernel<TM, TG, Epi><<<grid, kBlock, 0, s>>>(A, g, epi, partials);
  }
}

// ---------------------------------------------------------------------------------------------
// Persistent plain iterations: one cooperative launch runs L primal / dual sweep pairs with a
// grid-wide barrier after each sweep, instead of 2L kernel nodes of a CUDA graph.  Block b takes
// the sweep's virtual blocks b, b + gridDim.x, ... in both sweeps of every iteration, so each row's
// own iterates are read back by the thread that wrote them; the gathered vectors, written by other
// blocks, are read through L2.
//
// Every wait is bounded: a barrier that is not reached before the launch's deadline (read from
// %globaltimer) or within kBarrierPolls polls stores a status in the control block and every block
// returns; the host reads the status at its next synchronisation and fails the solve.

struct persist_ctl {
  unsigned arrivals;  // barrier arrivals of the current launch (zeroed before each launch)
  int status;         // 0, or kBarrierTimedOut / kBarrierPollLimit
};
constexpr int kBarrierTimedOut  = 1;
constexpr int kBarrierPollLimit = 2;
constexpr unsigned kBarrierPolls = 1u << 24;
// Deadline of one persistent launch of the solvers (at most 255 iterations): far above any
// legitimate run, it only bounds a launch whose grid barrier could not complete.
constexpr unsigned long long kPersistBudgetNs = 30ull * 1000 * 1000 * 1000;

__device__ __forceinline__ unsigned long long global_ns()
{
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p)
{
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_gpu_add(unsigned* p, unsigned v)
{
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_relaxed_gpu(const int* p)
{
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Arrive and wait until `target` arrivals have been counted.  Returns false (uniformly across
// the block) when the wait gave up or another block's wait already had.  The block's writes reach
// thread 0 through the block barrier; its arrival is a release at GPU scope (cumulative over
// them), and the poll that sees the last arrival an acquire, after which the block barrier hands
// the other blocks' writes on to every thread.
__device__ __forceinline__ bool persist_barrier(persist_ctl* c, unsigned target,
                                                unsigned long long deadline)
{
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    red_release_gpu_add(&c->arrivals, 1u);
    int st = 0;
    for (unsigned polls = 0;; ++polls) {
      if (ld_acquire_gpu(&c->arrivals) >= target) break;
      if ((st = ld_relaxed_gpu(&c->status)) != 0) break;
      if (polls >= kBarrierPolls) {
        st = kBarrierPollLimit;
        atomicCAS(&c->status, 0, st);
        break;
      }
      if ((polls & 15) == 15 && global_ns() > deadline) {
        st = kBarrierTimedOut;
        atomicCAS(&c->status, 0, st);
        break;
      }
    }
    ok = st == 0;
  }
  __syncthreads();
  return ok;
}

// Block 0's closing step of a persistent launch (after the last barrier): the iteration counter
// of the one LP, or of every active instance of a batch, moves on by L.
struct advance_one {
  pdlp_scalars* st;
  __device__ void operator()(int steps) const
  {
    if (threadIdx.x == 0) st->t0 += steps;
  }
};
struct advance_active {
  pdlp_scalars* sc;
  const int* active;
  int count;
  __device__ void operator()(int steps) const
  {
    for (int b = threadIdx.x; b < count; b += blockDim.x)
      if (active[b]) sc[b].t0 += steps;
  }
};

template <typename TX, class PE, class DE, class ADV>
__global__ void __launch_bounds__(kBlock, 3)
  persistent_plain_kernel(const dev_sell<TX> AT, const dev_sell<TX> A, const TX* y, const TX* xbar,
                          PE pe, DE de, ADV adv, int L, int grid_p, int grid_d, persist_ctl* ctl,
                          unsigned long long budget_ns)
{
  const unsigned long long deadline = global_ns() + budget_ns;
  unsigned target                   = 0;
  for (int i = 0; i < L; ++i) {
    pe.it_off = i;
    for (int vb = blockIdx.x; vb < grid_p; vb += gridDim.x)
      sell_map_block<TX, TX, PE, true>(AT, y, pe, nullptr, vb);
    target += gridDim.x;
    if (!persist_barrier(ctl, target, deadline)) return;
    de.it_off = i;
    for (int vb = blockIdx.x; vb < grid_d; vb += gridDim.x)
      sell_map_block<TX, TX, DE, true>(A, xbar, de, nullptr, vb);
    target += gridDim.x;
    if (!persist_barrier(ctl, target, deadline)) return;
  }
  if (blockIdx.x == 0) adv(L);
}

// The barrier alone, for measuring its cost and for checking that a wait which cannot complete
// (`unreachable` > 0 asks for more arrivals than the grid has blocks) ends with a status instead
// of hanging: `rounds` barriers, then block 0 records the elapsed nanoseconds.
static __global__ void persist_barrier_probe_kernel(persist_ctl* ctl, int rounds, unsigned unreachable,
                                                    unsigned long long budget_ns,
                                                    unsigned long long* elapsed)
{
  const unsigned long long t0 = global_ns(), deadline = t0 + budget_ns;
  unsigned target = 0;
  for (int r = 0; r < rounds; ++r) {
    target += gridDim.x;
    if (!persist_barrier(ctl, target + unreachable, deadline)) break;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *elapsed = global_ns() - t0;
}

// ---------------------------------------------------------------------------------------------
// PDHG epilogues (reflected variant, reference pdhg.cu:431-530 and pdlp.cu:2506-2563).

// The primal update of one variable j (shared by the single-LP and batch epilogues); `p` holds
// x_j, c_j, l_j, u_j and the anchor x_a,j, `st` the step scalars of j's LP.
// Receives the value a row step stores into the vector the next sweep gathers (x_bar for the
// primal step, y for the fused-Halpern dual step); the cluster-resident form copies it into the
// cluster's shared-memory copies.
struct no_sink {
  __device__ __forceinline__ void operator()(int, double) const {}
};

// w: the Halpern weight of the step (used with HALPERN).
template <typename TX, bool MAJOR, bool HALPERN, bool SAVE_ATY, class P, class Sink = no_sink>
__device__ __forceinline__ void primal_row_step(int j, double acc, const P& p, double tau, double w,
                                                TX* xbar, TX* xout, TX* xhat, TX* slack, TX* aty,
                                                const Sink& sink = Sink{})
{
  const double xj   = (double)p.x;
  const double next = xj - tau * ((double)p.c - acc);
  const double cl   = fmax(fmin(next, (double)p.up), (double)p.lo);
  if constexpr (MAJOR) {
    xhat[j]  = (TX)cl;
    slack[j] = (TX)((cl - next) / tau);
  }
  const double xb = 2.0 * cl - xj;
  if constexpr (SAVE_ATY) aty[j] = (TX)acc;
  if constexpr (HALPERN) {
    xbar[j] = (TX)xb;
    xout[j] = (TX)halpern_mix(w, xb, (double)p.xa);
  } else {
    xbar[j] = (TX)xb;
  }
  sink(j, (double)(TX)xb);
}

// The dual update of one constraint i (ratio: y_i / sigma); returns (y_bar_i - y_i)^2 for the
// fixed-point error.
template <typename TX, bool MAJOR, bool HALPERN, class P, class Sink = no_sink>
__device__ __forceinline__ double dual_row_step(int i, double acc, const P& p, double sigma,
                                                double ratio, double w, TX* ybar, TX* yout,
                                                TX* yhat, const Sink& sink = Sink{})
{
  const double yi    = (double)p.y;
  const double t     = ratio - acc;
  const double tp    = fmax(-(double)p.up, fmin(t, -(double)p.lo));
  const double ny    = (t - tp) * sigma;
  if constexpr (MAJOR) yhat[i] = (TX)ny;
  const double yb = 2.0 * ny - yi;
  if constexpr (HALPERN) {
    const TX y_next = (TX)halpern_mix_y(w, yb, (double)p.ya);
    yout[i]         = y_next;
    sink(i, (double)y_next);
  } else {
    ybar[i] = (TX)yb;
  }
  const double d = yb - yi;
  return d * d;
}

// The same with the step's scalars read from `st`.
template <typename TX, bool MAJOR, bool HALPERN, bool SAVE_ATY, class P, class Sink = no_sink>
__device__ __forceinline__ void primal_row_step(int j, double acc, const P& p,
                                                const pdlp_scalars* st, int it_off, TX* xbar,
                                                TX* xout, TX* xhat, TX* slack, TX* aty,
                                                const Sink& sink = Sink{})
{
  primal_row_step<TX, MAJOR, HALPERN, SAVE_ATY>(j, acc, p, st->tau,
                                                HALPERN ? halpern_weight(st, it_off) : 0.0, xbar,
                                                xout, xhat, slack, aty, sink);
}
template <typename TX, bool MAJOR, bool HALPERN, class P, class Sink = no_sink>
__device__ __forceinline__ double dual_row_step(int i, double acc, const P& p,
                                                const pdlp_scalars* st, int it_off, TX* ybar,
                                                TX* yout, TX* yhat, const Sink& sink = Sink{})
{
  const double sigma = st->sigma;
  return dual_row_step<TX, MAJOR, HALPERN>(i, acc, p, sigma, (double)p.y / sigma,
                                           HALPERN ? halpern_weight(st, it_off) : 0.0, ybar, yout,
                                           yhat, sink);
}

// Row j of A^T:  x_next = x - tau (c - A^T y);  x_hat = clamp(x_next, l, u);
//                slack = (x_hat - x_next) / tau;  x_bar = 2 x_hat - x;
//                (fused Halpern)  x <- w x_bar + (1 - w) x_anchor.
template <typename TX, bool MAJOR, bool HALPERN, bool SAVE_ATY>
struct primal_epi {
  static constexpr int kRed = 0;
  const TX* x;
  const TX* c;
  const TX* lo;
  const TX* up;
  const TX* xa;
  TX* xbar;
  TX* xout;
  TX* xhat;
  TX* slack;
  TX* aty;
  const pdlp_scalars* st;
  int it_off;
  struct pre_t {
    TX x, c, lo, up, xa;
  };
  __device__ __forceinline__ pre_t load(int j) const
  {
    return pre_t{x[j], c[j], lo[j], up[j], HALPERN ? xa[j] : TX(0)};
  }
  __device__ __forceinline__ void operator()(int j, double acc, const pre_t& p, red_t<0>&) const
  {
    primal_row_step<TX, MAJOR, HALPERN, SAVE_ATY>(j, acc, p, st, it_off, xbar, xout, xhat, slack,
                                                  aty);
  }
};

// Row i of A:  t = y / sigma - A x_bar;  y_hat = (t - clamp(t, -u, -l)) sigma;  y_bar = 2 y_hat - y;
//              (fused Halpern) y <- w y_bar + (1 - w) y_anchor;  (FPE) red += (y_bar - y)^2.
template <typename TX, bool MAJOR, bool HALPERN, bool FPE>
struct dual_epi {
  static constexpr int kRed = FPE ? 1 : 0;
  const TX* y;
  const TX* lo;
  const TX* up;
  const TX* ya;
  TX* ybar;
  TX* yout;
  TX* yhat;
  const pdlp_scalars* st;
  int it_off;
  struct pre_t {
    TX y, lo, up, ya;
  };
  __device__ __forceinline__ pre_t load(int i) const
  {
    return pre_t{y[i], lo[i], up[i], HALPERN ? ya[i] : TX(0)};
  }
  __device__ __forceinline__ void operator()(int i, double acc, const pre_t& p,
                                             red_t<kRed>& r) const
  {
    const double d2 = dual_row_step<TX, MAJOR, HALPERN>(i, acc, p, st, it_off, ybar, yout, yhat);
    if constexpr (FPE) r.v[0] += d2;
  }
};

// ---------------------------------------------------------------------------------------------
// Cluster-resident plain iterations for small LPs: one thread-block cluster of C blocks runs L plain
// iterations, the last of which may be one that keeps x_hat, y_hat and the slack for a termination
// check.  Every block holds a full copy of both gathered vectors (y for the primal sweep, x_bar for
// the dual sweep) in its shared memory and sends each new entry to every block's copy through
// distributed shared memory (mapa + st.shared::cluster: posted, only the barrier waits for them).  A
// cluster barrier (arrive.release / wait.acquire: hardware, no spin loop) follows every sweep.
// Every row is computed by one warp exactly as in sell_map_kernel: same products, same order.
//
// With CACHED, each block also keeps its share of A and A^T and its rows' operands and iterates in
// shared memory (16-bit column indices), so an iteration touches no global memory: what bounds it
// is the shared-memory requests of the products, the broadcasts and two cluster barriers.  Without
// (the shares do not fit), the matrices and operands are read from L2 every iteration, as the
// only form of this kernel once did: its iteration is bound by the latency of those dependent reads
// (2000 x 5000 LP, FP64: 8.95 us an iteration).
constexpr int kResidentThreads = 512;
constexpr int kResidentWarps   = kResidentThreads / kWarp;

__device__ __forceinline__ unsigned cluster_rank()
{
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size()
{
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier()
{
  __syncwarp();
  asm volatile(
    "barrier.cluster.arrive.release.aligned;\n"
    "barrier.cluster.wait.acquire.aligned;\n" ::
      : "memory");
}
// Stores v at shared-memory address saddr (a byte offset in this block's window) of block `rank`
// of the cluster.
__device__ __forceinline__ void dsmem_store(unsigned saddr, unsigned rank, double v)
{
  unsigned remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(saddr), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote), "d"(v) : "memory");
}
__device__ __forceinline__ void dsmem_store(unsigned saddr, unsigned rank, float v)
{
  unsigned remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(saddr), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}

// Copies a row's new value into every block's shared-memory copy of its vector (at: the
// shared-memory address of the entry in this block's copy).
template <typename TX>
struct dsmem_sink {
  unsigned at;
  unsigned blocks;
  __device__ __forceinline__ void operator()(int, double v) const
  {
    for (unsigned c = 0; c < blocks; ++c) dsmem_store(at, c, (TX)v);
  }
};

// Shares of a matrix: units are its long rows, then its slices; unit u belongs to block u % C as
// its unit u / C.  Capacities of a block's share: units, and elements (each unit's start is padded
// to 4, so that chunk loads are aligned).
struct resident_dims {
  int blocks = 0;       // C
  int units[2] = {0, 0};     // A^T, A
  int elems[2] = {0, 0};
  B200_HD static size_t pad(size_t b) { return (b + 15) & ~(size_t)15; }
  // The image of a block's constant data (device memory, copied to shared memory by each launch):
  // {start, length} of the units of A^T and A, the operands c, l, u and l_c, u_c per unit lane,
  // values and indices of A^T and A, the blocks that need the entry of each unit lane of A^T and A
  // (resident_needs_kernel), and the numbers of x_bar and y entries that this block needs.
  template <typename TX>
  B200_HD size_t image_at(int part) const
  {
    const size_t bytes[11] = {(size_t)units[0] * 8,
                             (size_t)units[1] * 8,
                             (size_t)units[0] * 3 * kWarp * sizeof(TX),
                             (size_t)units[1] * 2 * kWarp * sizeof(TX),
                             (size_t)elems[0] * sizeof(TX),
                             (size_t)elems[1] * sizeof(TX),
                             (size_t)elems[0] * 2,
                             (size_t)elems[1] * 2,
                             (size_t)units[0] * kWarp * 2,
                             (size_t)units[1] * kWarp * 2,
                             8};
    size_t at = 0;
    for (int q = 0; q < part; ++q) at += pad(bytes[q]);
    return at;
  }
  template <typename TX>
  B200_HD size_t image_bytes() const
  {
    return image_at<TX>(11);
  }
  // Shared memory of a launch: y, x_bar, then (CACHED) the iterates x, x_anchor, y, y_anchor per
  // unit lane and the image.
  template <typename TX>
  B200_HD static size_t vector_bytes(int m, int n)
  {
    return pad((size_t)m * sizeof(TX)) + pad((size_t)n * sizeof(TX));
  }
  template <typename TX>
  B200_HD size_t state_bytes() const
  {
    return (size_t)(units[0] + units[1]) * 2 * kWarp * sizeof(TX);
  }
};

template <typename TX>
__device__ __forceinline__ void unit_range(const dev_sell<TX>& M, int u, int64_t& lo, int64_t& hi)
{
  if (u < M.n_long) {
    lo = M.long_off[u];
    hi = M.long_off[u + 1];
  } else {
    lo = M.slice_off[u - M.n_long];
    hi = M.slice_off[u - M.n_long + 1];
  }
}

// Which blocks need an entry of x_bar or y: bit r of needs[j] for column j of block r's share of A,
// of needs[n + i] for column i (row of A) of its share of A^T; and the first entry of every unit goes
// to every block that has units of the other sweep, so that a block which has all the entries that it
// needs also knows that every unit of the sweep before has read its own (see resident_unit_kernel).
// needs must be zeroed first.  One block per block of the cluster.
template <typename TX>
__global__ void __launch_bounds__(kResidentThreads)
  resident_needs_kernel(const dev_sell<TX> AT, const dev_sell<TX> A, resident_dims D, int n,
                        unsigned* needs)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int w = 0; w < 2; ++w) {
    const dev_sell<TX>&M = w == 0 ? AT : A, &O = w == 0 ? A : AT;
    const int total = M.n_long + M.n_slices, other = O.n_long + O.n_slices;
    unsigned* read  = needs + (w == 0 ? n : 0);  // the vector that M's rows gather
    unsigned* own   = needs + (w == 0 ? 0 : n);  // the vector of M's rows
    const unsigned all = other >= 32 ? ~0u : (1u << min(other, D.blocks)) - 1u;
    for (int u = (int)blockIdx.x + D.blocks * warp; u < total; u += D.blocks * kResidentWarps) {
      int64_t b, e;
      unit_range(M, u, b, e);
      for (int64_t k = b + lane; k < e; k += kWarp) atomicOr(read + M.idx[k], 1u << blockIdx.x);
      if (lane == 0)
        atomicOr(own + (u < M.n_long ? u : M.n_long + (u - M.n_long) * kWarp),
                 all & ((1u << D.blocks) - 1u));
    }
  }
}

// Builds the image of block blockIdx.x (once per solve).
template <typename TX>
__global__ void __launch_bounds__(kResidentThreads)
  resident_image_kernel(const dev_sell<TX> AT, const dev_sell<TX> A, const TX* c, const TX* lo,
                        const TX* up, const TX* lc, const TX* uc, resident_dims D, int m, int n,
                        const unsigned* needs, unsigned char* images)
{
  unsigned char* img = images + blockIdx.x * D.image_bytes<TX>();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ int count[2];
  if (threadIdx.x < 2) count[threadIdx.x] = 0;
  for (int w = 0; w < 2; ++w) {
    const dev_sell<TX>& M = w == 0 ? AT : A;
    const int total       = M.n_long + M.n_slices;
    int2* table           = reinterpret_cast<int2*>(img + D.image_at<TX>(w));
    for (int i = threadIdx.x; i < D.units[w]; i += kResidentThreads) {
      const int u = (int)blockIdx.x + D.blocks * i;
      int64_t b = 0, e = 0;
      if (u < total) unit_range(M, u, b, e);
      table[i] = make_int2(0, (int)(e - b));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int at = 0;
      for (int i = 0; i < D.units[w]; ++i) {
        const int len = table[i].y;
        table[i].x    = at;
        at += (len + 3) & ~3;
      }
    }
    __syncthreads();
    TX* ops              = reinterpret_cast<TX*>(img + D.image_at<TX>(2 + w));
    TX* val              = reinterpret_cast<TX*>(img + D.image_at<TX>(4 + w));
    unsigned short* x    = reinterpret_cast<unsigned short*>(img + D.image_at<TX>(6 + w));
    unsigned short* mask = reinterpret_cast<unsigned short*>(img + D.image_at<TX>(8 + w));
    const unsigned* need = needs + (w == 0 ? 0 : n);
    const int slots      = D.units[w] * kWarp;
    for (int i = warp; i < D.units[w]; i += kResidentWarps) {
      const int u  = (int)blockIdx.x + D.blocks * i;
      const int2 t = table[i];
      int row      = -1;
      if (u < M.n_long) {
        if (lane == 0) row = u;
      } else if (u < total) {
        row = M.n_long + (u - M.n_long) * kWarp + lane;
        if (row >= M.rows) row = -1;
      }
      const int s = i * kWarp + lane;
      if (w == 0) {
        ops[s]             = row >= 0 ? c[row] : TX(0);
        ops[slots + s]     = row >= 0 ? lo[row] : TX(0);
        ops[2 * slots + s] = row >= 0 ? up[row] : TX(0);
      } else {
        ops[s]         = row >= 0 ? lc[row] : TX(0);
        ops[slots + s] = row >= 0 ? uc[row] : TX(0);
      }
      mask[s] = row >= 0 ? (unsigned short)need[row] : (unsigned short)0;
      int64_t b = 0, e = 0;
      if (u < total) unit_range(M, u, b, e);
      for (int k = lane; k < t.y; k += kWarp) {
        val[t.x + k] = M.val[b + k];
        x[t.x + k]   = (unsigned short)M.idx[b + k];
      }
    }
    // Entries of this sweep's vector that this block needs.
    int mine = 0;
    for (int j = threadIdx.x; j < (w == 0 ? n : m); j += kResidentThreads)
      mine += (need[j] >> blockIdx.x) & 1u;
    atomicAdd(count + w, mine);
    __syncthreads();
  }
  if (threadIdx.x < 2) reinterpret_cast<int*>(img + D.image_at<TX>(10))[threadIdx.x] = count[threadIdx.x];
}

__device__ __forceinline__ void shared_chunk(const float* p, double (&v)[4])
{
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0]           = t.x;
  v[1]           = t.y;
  v[2]           = t.z;
  v[3]           = t.w;
}
__device__ __forceinline__ void shared_chunk(const double* p, double (&v)[4])
{
  const double2 a = reinterpret_cast<const double2*>(p)[0];
  const double2 b = reinterpret_cast<const double2*>(p)[1];
  v[0]            = a.x;
  v[1]            = a.y;
  v[2]            = b.x;
  v[3]            = b.y;
}

// The product of a slice's row (this lane's) from shared memory, in sell_map_block's order.
template <typename TX, typename TG>
__device__ __forceinline__ double resident_slice(const TX* v, const unsigned short* x, int nchunk,
                                                 const TG* g)
{
  double acc = 0.0;
#pragma unroll 2
  for (int q = 0; q < nchunk; ++q) {
    const ushort4 i = *reinterpret_cast<const ushort4*>(x);
    double w[4];
    shared_chunk(v, w);
    const TG g0 = g[i.x], g1 = g[i.y], g2 = g[i.z], g3 = g[i.w];
    acc += w[0] * (double)g0;
    acc += w[1] * (double)g1;
    acc += w[2] * (double)g2;
    acc += w[3] * (double)g3;
    v += kWarp * kChunk;
    x += kWarp * kChunk;
  }
  return acc;
}
template <typename TX, typename TG>
__device__ __forceinline__ double resident_long(const TX* v, const unsigned short* x, int len,
                                                const TG* g, bool wide)
{
  if (wide)
    return wide_row_by_warp(
      len, [&](int k, double& a) { a += (double)v[k] * (double)g[x[k]]; });
  double acc = 0.0;
  for (int k = threadIdx.x & 31; k < len; k += kWarp) acc += (double)v[k] * (double)g[x[k]];
  return warp_sum(acc);
}

// The plain epilogues with the new x_bar_j, or y_i, also sent to the cluster's copies.
template <typename TX, bool MAJOR>
struct cluster_primal_epi {
  static constexpr int kRed = 0;
  using base_t              = primal_epi<TX, false, true, false>;
  using pre_t               = typename base_t::pre_t;
  base_t base;
  unsigned copy, blocks;
  __device__ __forceinline__ pre_t load(int j) const { return base.load(j); }
  __device__ __forceinline__ void operator()(int j, double acc, const pre_t& p, red_t<0>&) const
  {
    const dsmem_sink<TX> sink{copy + (unsigned)j * (unsigned)sizeof(TX), blocks};
    primal_row_step<TX, MAJOR, true, false>(j, acc, p, base.st, base.it_off, base.xbar, base.xout,
                                            base.xhat, base.slack, base.aty, sink);
  }
};
template <typename TX, bool MAJOR>
struct cluster_dual_epi {
  static constexpr int kRed = 0;
  using base_t              = dual_epi<TX, false, true, false>;
  using pre_t               = typename base_t::pre_t;
  base_t base;
  unsigned copy, blocks;
  __device__ __forceinline__ pre_t load(int i) const { return base.load(i); }
  __device__ __forceinline__ void operator()(int i, double acc, const pre_t& p, red_t<0>&) const
  {
    const dsmem_sink<TX> sink{copy + (unsigned)i * (unsigned)sizeof(TX), blocks};
    dual_row_step<TX, MAJOR, true>(i, acc, p, base.st, base.it_off, base.ybar, base.yout,
                                   base.yhat, sink);
  }
};

// L plain iterations, the last one a keeping one when `keep`.  pe / de: the plain primal / dual
// epilogues (it_off set per iteration), whose gathered vectors are y (de.y = de.yout) and x_bar
// (pe.xbar).  Without CACHED a block runs kResidentWarps / kWarpsPerBlock groups of kWarpsPerBlock
// warps, which take the sweep's 8-warp virtual blocks in turn.
template <typename TX, bool CACHED>
__global__ void __launch_bounds__(kResidentThreads)
  resident_plain_kernel(const dev_sell<TX> AT, const dev_sell<TX> A,
                        primal_epi<TX, false, true, false> pe, dual_epi<TX, false, true, false> de,
                        int L, int keep, int m, int n, resident_dims D,
                        const unsigned char* images, pdlp_scalars* st, int*)
{
  extern __shared__ __align__(16) unsigned char cl_smem[];
  TX* ys  = reinterpret_cast<TX*>(cl_smem);
  TX* xbs = reinterpret_cast<TX*>(cl_smem + resident_dims::pad((size_t)m * sizeof(TX)));
  const unsigned rank = cluster_rank(), blocks = cluster_size();
  const unsigned y_copy  = (unsigned)__cvta_generic_to_shared(ys);
  const unsigned xb_copy = (unsigned)__cvta_generic_to_shared(xbs);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < m; i += kResidentThreads) ys[i] = de.y[i];

  if constexpr (CACHED) {
    const int ut = AT.n_long + AT.n_slices, ua = A.n_long + A.n_slices;
    const int sp = D.units[0] * kWarp, sd = D.units[1] * kWarp;
    TX* xs             = reinterpret_cast<TX*>(cl_smem + resident_dims::vector_bytes<TX>(m, n));
    TX *xas = xs + sp, *yis = xas + sp, *yas = yis + sd;
    unsigned char* img = reinterpret_cast<unsigned char*>(yas + sd);
    {
      const size_t bytes       = D.image_bytes<TX>();
      const unsigned char* src = images + rank * bytes;
      for (size_t b = (size_t)threadIdx.x * 16; b < bytes; b += kResidentThreads * 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                       (unsigned)__cvta_generic_to_shared(img + b)),
                     "l"(src + b)
                     : "memory");
    }
    // The row of this lane in the block's unit i of the sweep (-1: none).
    auto row_of = [&](const dev_sell<TX>& M, int total, int i) {
      const int u = (int)rank + D.blocks * i;
      if (u < M.n_long) return lane == 0 ? u : -1;
      if (u >= total) return -1;
      const int r = M.n_long + (u - M.n_long) * kWarp + lane;
      return r < M.rows ? r : -1;
    };
    for (int i = warp; i < D.units[0]; i += kResidentWarps) {
      const int j = row_of(AT, ut, i);
      if (j >= 0) {
        xs[i * kWarp + lane]  = pe.x[j];
        xas[i * kWarp + lane] = pe.xa[j];
      }
    }
    for (int i = warp; i < D.units[1]; i += kResidentWarps) {
      const int r = row_of(A, ua, i);
      if (r >= 0) {
        yis[i * kWarp + lane] = de.y[r];
        yas[i * kWarp + lane] = de.ya[r];
      }
    }
    const pdlp_scalars sc = *st;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int2* tab_p           = reinterpret_cast<const int2*>(img + D.image_at<TX>(0));
    const int2* tab_d           = reinterpret_cast<const int2*>(img + D.image_at<TX>(1));
    const TX* op_p              = reinterpret_cast<const TX*>(img + D.image_at<TX>(2));
    const TX* op_d              = reinterpret_cast<const TX*>(img + D.image_at<TX>(3));
    const TX* val_p             = reinterpret_cast<const TX*>(img + D.image_at<TX>(4));
    const TX* val_d             = reinterpret_cast<const TX*>(img + D.image_at<TX>(5));
    const unsigned short* idx_p = reinterpret_cast<const unsigned short*>(img + D.image_at<TX>(6));
    const unsigned short* idx_d = reinterpret_cast<const unsigned short*>(img + D.image_at<TX>(7));
    // Every block of the cluster is running (and has its copy of y) before any block stores into
    // another's shared memory.
    cluster_barrier();
    for (int it = 0; it < L; ++it) {
      const bool last = it == L - 1;
      for (int i = warp; i < D.units[0]; i += kResidentWarps) {
        const int u = (int)rank + D.blocks * i;
        if (u >= ut) break;
        const int2 t     = tab_p[i];
        const int s      = i * kWarp + lane;
        const int j      = row_of(AT, ut, i);
        const double acc = u < AT.n_long
                             ? resident_long(val_p + t.x, idx_p + t.x, t.y, ys, u < AT.n_wide)
                             : resident_slice(val_p + t.x + lane * kChunk,
                                              idx_p + t.x + lane * kChunk, t.y >> 7, ys);
        if (j >= 0) {
          const typename primal_epi<TX, false, true, false>::pre_t p{
            xs[s], op_p[s], op_p[sp + s], op_p[2 * sp + s], xas[s]};
          const dsmem_sink<TX> sink{xb_copy + (unsigned)j * (unsigned)sizeof(TX), blocks};
          TX xb;
          if (last && keep)
            primal_row_step<TX, true, true, false>(0, acc, p, &sc, it, &xb, xs + s, pe.xhat + j,
                                                   pe.slack + j, (TX*)nullptr, sink);
          else
            primal_row_step<TX, false, true, false>(0, acc, p, &sc, it, &xb, xs + s, (TX*)nullptr,
                                                    (TX*)nullptr, (TX*)nullptr, sink);
          if (last) {
            pe.xout[j] = xs[s];
            pe.xbar[j] = xb;
          }
        }
      }
      cluster_barrier();
      for (int i = warp; i < D.units[1]; i += kResidentWarps) {
        const int u = (int)rank + D.blocks * i;
        if (u >= ua) break;
        const int2 t     = tab_d[i];
        const int s      = i * kWarp + lane;
        const int r      = row_of(A, ua, i);
        const double acc = u < A.n_long
                             ? resident_long(val_d + t.x, idx_d + t.x, t.y, xbs, u < A.n_wide)
                             : resident_slice(val_d + t.x + lane * kChunk,
                                              idx_d + t.x + lane * kChunk, t.y >> 7, xbs);
        if (r >= 0) {
          const typename dual_epi<TX, false, true, false>::pre_t p{yis[s], op_d[s], op_d[sd + s],
                                                                   yas[s]};
          const dsmem_sink<TX> sink{y_copy + (unsigned)r * (unsigned)sizeof(TX), blocks};
          if (last && keep)
            dual_row_step<TX, true, true>(0, acc, p, &sc, it, (TX*)nullptr, yis + s, de.yhat + r,
                                          sink);
          else
            dual_row_step<TX, false, true>(0, acc, p, &sc, it, (TX*)nullptr, yis + s,
                                           (TX*)nullptr, sink);
          if (last) de.yout[r] = yis[s];
        }
      }
      cluster_barrier();
    }
  } else {
    cluster_barrier();
    const int gp = sweep_grid(AT), gd = sweep_grid(A);
    const int group  = warp / kWarpsPerBlock;
    const int first  = (int)rank + (int)blocks * group;
    const int stride = (int)blocks * (kResidentWarps / kWarpsPerBlock);
    for (int it = 0; it < L; ++it) {
      pe.it_off = de.it_off = it;
      const bool kept       = keep && it == L - 1;
      for (int vb = first; vb < gp; vb += stride)
        if (kept)
          sell_map_block<TX, TX>(AT, ys, cluster_primal_epi<TX, true>{pe, xb_copy, blocks}, nullptr, vb);
        else
          sell_map_block<TX, TX>(AT, ys, cluster_primal_epi<TX, false>{pe, xb_copy, blocks}, nullptr, vb);
      cluster_barrier();
      for (int vb = first; vb < gd; vb += stride)
        if (kept)
          sell_map_block<TX, TX>(A, xbs, cluster_dual_epi<TX, true>{de, y_copy, blocks}, nullptr, vb);
        else
          sell_map_block<TX, TX>(A, xbs, cluster_dual_epi<TX, false>{de, y_copy, blocks}, nullptr, vb);
      cluster_barrier();
    }
  }
  if (rank == 0 && threadIdx.x == 0) st->t0 += L;
}

// The CACHED form where no warp takes more than one slice of either sweep and no row is long (up to
// 16 x 10 slices, that is 5 120 rows of each matrix, with clusters of 16).  What bounds an iteration
// here is the exchange of x_bar and y (a block sends some 16 bytes a cycle), the chain of a row's
// products, and the latency of each.  A cluster barrier behind posted stores waits for every store
// to be acknowledged: 2 300 (2048 entries, 16 blocks) and 4 300 cycles (5120) of a phase.  So:
//   * an entry goes, only to the blocks that gather it, with st.async, whose bytes count towards the
//     receiving block's mbarrier: no barrier at all (1 480 and 2 960 cycles for all entries);
//   * the first entry of every slice goes to every block of the other sweep.  A warp sends after the
//     gathers of all its lanes (a warp barrier stands between: lanes leave the wait and the gathers one
//     by one), so a block that has its bytes of one sweep knows that every warp of that sweep is done
//     reading the vector that the block is about to write next;
//   * the cluster is the smallest of 4, 8 and 16 blocks whose warps suffice: every further block is
//     one more store for every entry;
//   * a row's gathers run two chunks ahead of its sum (1 870 cycles for 9 chunks without);
//   * a row's operands and the remote addresses stay in registers, and the Halpern weight and
//     y / sigma (two FP64 divisions) are formed between sending and waiting.
// Waits are bounded: one that runs out sets the launch's status, and every block leaves through the
// closing cluster barrier.
// At most kUnitWarps slices a block: with 10, an iteration of a 2000 x 5000 LP takes 5.20 us (FP64; 5.46
// in the form of several slices a warp) and of 2400 x 6000, 12 slices a block, 6.22 in that form;
// compiled for 12 it takes 5.94 here, but smaller LPs up to 0.07 us more, and 8000 columns with 16
// lose (7.46, 7.26 there).
constexpr int kClusterBlocks = 16;
constexpr int kUnitWarps     = 10;

// Stores v at offset `off` from the mapped base addresses in the blocks of `mask`, counted by the
// barrier at offset `bar` there.  Predicated, not branched over: with sixteen branches a warp's step
// and sends took 1 200 to 2 300 cycles.
template <int C>
__device__ __forceinline__ void exchange_send(const unsigned (&base)[C], unsigned mask, unsigned off,
                                              unsigned bar, double v)
{
#pragma unroll
  for (int c = 0; c < C; ++c)
    asm volatile(
      "{\n .reg .pred p;\n"
      " setp.ne.u32 p, %3, 0;\n"
      " @p st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];\n}" ::"r"(
        base[c] + off),
      "d"(v), "r"(base[c] + bar), "r"(mask & (1u << c))
      : "memory");
}
template <int C>
__device__ __forceinline__ void exchange_send(const unsigned (&base)[C], unsigned mask, unsigned off,
                                              unsigned bar, float v)
{
#pragma unroll
  for (int c = 0; c < C; ++c)
    asm volatile(
      "{\n .reg .pred p;\n"
      " setp.ne.u32 p, %3, 0;\n"
      " @p st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];\n}" ::"r"(
        base[c] + off),
      "f"(v), "r"(base[c] + bar), "r"(mask & (1u << c))
      : "memory");
}

// This lane's row (-1: none) of a warp's slice, and its elements (first chunk in registers).
template <typename TX>
struct held_unit {
  int row    = -1;
  int chunks = -1;  // -1: the warp has no slice
  TX v0[4];
  ushort4 x0, x1;
  const TX* val;
  const unsigned short* idx;
  __device__ __forceinline__ void load(const dev_sell<TX>& M, int s, const int2& t, const TX* vals,
                                       const unsigned short* idxs)
  {
    const int lane = threadIdx.x & 31;
    x0 = x1 = make_ushort4(0, 0, 0, 0);
#pragma unroll
    for (int e = 0; e < 4; ++e) v0[e] = TX(0);
    val = vals + t.x + lane * kChunk;
    idx = idxs + t.x + lane * kChunk;
    if (s >= M.n_slices) return;
    row = s * kWarp + lane;
    if (row >= M.rows) row = -1;
    chunks = t.y >> 7;
    if (chunks > 0) {
#pragma unroll
      for (int e = 0; e < 4; ++e) v0[e] = val[e];
      x0 = *reinterpret_cast<const ushort4*>(idx);
    }
    if (chunks > 1) x1 = *reinterpret_cast<const ushort4*>(idx + kWarp * kChunk);
  }
  // The row's product, in sell_map_block's order: while chunk q is added, the entries of chunk q + 1
  // and the indices of chunk q + 2 are on their way.
  __device__ __forceinline__ double product(const TX* g) const
  {
    double acc = 0.0;
    if (chunks <= 0) return acc;
    TX gq[4] = {g[x0.x], g[x0.y], g[x0.z], g[x0.w]};
    double vq[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) vq[e] = (double)v0[e];
    ushort4 x = x1;
    for (int q = 0; q < chunks; ++q) {
      TX gn[4]     = {TX(0), TX(0), TX(0), TX(0)};
      double vn[4] = {0.0, 0.0, 0.0, 0.0};
      if (q + 1 < chunks) {
        gn[0] = g[x.x];
        gn[1] = g[x.y];
        gn[2] = g[x.z];
        gn[3] = g[x.w];
        shared_chunk(val + (q + 1) * kWarp * kChunk, vn);
        if (q + 2 < chunks) x = *reinterpret_cast<const ushort4*>(idx + (q + 2) * kWarp * kChunk);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) acc += vq[e] * (double)gq[e];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        gq[e] = gn[e];
        vq[e] = vn[e];
      }
    }
    return acc;
  }
};

// Shared memory: the barriers of x_bar and y, y, x_bar, the image.
constexpr unsigned kUnitBars = 16;
template <typename TX, int C>
__global__ void __launch_bounds__(kUnitWarps * kWarp, 1)
  resident_unit_kernel(const dev_sell<TX> AT, const dev_sell<TX> A,
                       primal_epi<TX, false, true, false> pe, dual_epi<TX, false, true, false> de,
                       int L, int keep, int m, int n, resident_dims D, const unsigned char* images,
                       pdlp_scalars* st, int* status)
{
  extern __shared__ __align__(16) unsigned char cl_smem[];
  const unsigned xb_0 = kUnitBars + (unsigned)resident_dims::pad((size_t)m * sizeof(TX));
  TX* ys              = reinterpret_cast<TX*>(cl_smem + kUnitBars);
  TX* xbs             = reinterpret_cast<TX*>(cl_smem + xb_0);
  unsigned char* img  = cl_smem + kUnitBars + resident_dims::vector_bytes<TX>(m, n);
  const unsigned rank = cluster_rank();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned bar_x = (unsigned)__cvta_generic_to_shared(cl_smem), bar_y = bar_x + 8;
  if (threadIdx.x == 0) {
    phase_init(bar_x);
    phase_init(bar_y);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  {
    const size_t bytes       = D.image_bytes<TX>();
    const unsigned char* src = images + rank * bytes;
    for (size_t b = (size_t)threadIdx.x * 16; b < bytes; b += (size_t)blockDim.x * 16)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(img + b)),
                   "l"(src + b)
                   : "memory");
  }
  for (int i = threadIdx.x; i < m; i += blockDim.x) ys[i] = de.y[i];
  const pdlp_scalars sc = *st;
  unsigned base[C];
#pragma unroll
  for (int c = 0; c < C; ++c)
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(base[c]) : "r"(bar_x), "r"(c));
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int slice = (int)rank + D.blocks * warp;
  held_unit<TX> P, Q;
  typename primal_epi<TX, false, true, false>::pre_t px{};
  typename dual_epi<TX, false, true, false>::pre_t dy{};
  unsigned to_p = 0, to_d = 0;  // blocks that need this lane's x_bar, y
  if (warp < D.units[0]) {
    P.load(AT, slice, reinterpret_cast<const int2*>(img + D.image_at<TX>(0))[warp],
           reinterpret_cast<const TX*>(img + D.image_at<TX>(4)),
           reinterpret_cast<const unsigned short*>(img + D.image_at<TX>(6)));
    const TX* op = reinterpret_cast<const TX*>(img + D.image_at<TX>(2)) + warp * kWarp + lane;
    to_p = reinterpret_cast<const unsigned short*>(img + D.image_at<TX>(8))[warp * kWarp + lane];
    if (P.row >= 0)
      px = {pe.x[P.row], op[0], op[D.units[0] * kWarp], op[2 * D.units[0] * kWarp], pe.xa[P.row]};
  }
  if (warp < D.units[1]) {
    Q.load(A, slice, reinterpret_cast<const int2*>(img + D.image_at<TX>(1))[warp],
           reinterpret_cast<const TX*>(img + D.image_at<TX>(5)),
           reinterpret_cast<const unsigned short*>(img + D.image_at<TX>(7)));
    const TX* op = reinterpret_cast<const TX*>(img + D.image_at<TX>(3)) + warp * kWarp + lane;
    to_d = reinterpret_cast<const unsigned short*>(img + D.image_at<TX>(9))[warp * kWarp + lane];
    if (Q.row >= 0) dy = {de.y[Q.row], op[0], op[D.units[1] * kWarp], de.ya[Q.row]};
  }
  const int2 need = *reinterpret_cast<const int2*>(img + D.image_at<TX>(10));
  const unsigned bytes_x = need.x * (unsigned)sizeof(TX), bytes_y = need.y * (unsigned)sizeof(TX);
  if (threadIdx.x == 0) {
    phase_expect(bar_x, bytes_x);
    phase_expect(bar_y, bytes_y);
  }
  double w = halpern_weight(&sc, 0), ratio = (double)dy.y / sc.sigma;
  // Every block of the cluster is running, with its copy of y and its barriers, before any block
  // stores into another's shared memory.
  cluster_barrier();
  unsigned phase_x = 0, phase_y = 0;
  bool ok = true;
  for (int it = 0; it < L; ++it) {
    const bool last = it == L - 1;
    if (P.chunks >= 0) {
      if (it > 0) {
        if (!(ok = phase_wait(bar_y, phase_y))) break;
        phase_y ^= 1;
        if (threadIdx.x == 0) phase_expect(bar_y, bytes_y);
      }
      const double acc = P.product(ys);
      __syncwarp();  // lane 0's entry tells the receivers that all lanes have gathered
      if (P.row >= 0) {
        const auto send = [&](int, double v) {
          exchange_send(base, to_p, xb_0 + (unsigned)P.row * (unsigned)sizeof(TX), 0, (TX)v);
        };
        TX xb, xn;
        if (last && keep)
          primal_row_step<TX, true, true, false>(0, acc, px, sc.tau, w, &xb, &xn,
                                                 pe.xhat + P.row, pe.slack + P.row, (TX*)nullptr,
                                                 send);
        else
          primal_row_step<TX, false, true, false>(0, acc, px, sc.tau, w, &xb, &xn, (TX*)nullptr,
                                                  (TX*)nullptr, (TX*)nullptr, send);
        px.x = xn;
        if (last) {
          pe.xout[P.row] = xn;
          pe.xbar[P.row] = xb;
        }
      }
    }
    if (Q.chunks >= 0) {
      if (!(ok = phase_wait(bar_x, phase_x))) break;
      phase_x ^= 1;
      if (threadIdx.x == 0) phase_expect(bar_x, bytes_x);
      const double acc = Q.product(xbs);
      __syncwarp();
      if (Q.row >= 0) {
        const auto send = [&](int, double v) {
          exchange_send(base, to_d, kUnitBars + (unsigned)Q.row * (unsigned)sizeof(TX), 8, (TX)v);
        };
        TX yn;
        if (last && keep)
          dual_row_step<TX, true, true>(0, acc, dy, sc.sigma, ratio, w, (TX*)nullptr, &yn,
                                        de.yhat + Q.row, send);
        else
          dual_row_step<TX, false, true>(0, acc, dy, sc.sigma, ratio, w, (TX*)nullptr, &yn,
                                         (TX*)nullptr, send);
        dy.y = yn;
        if (last) de.yout[Q.row] = yn;
      }
    }
    w     = halpern_weight(&sc, it + 1);
    ratio = (double)dy.y / sc.sigma;
  }
  // No block leaves while entries of the last sweep are on their way to it.
  if (ok && P.chunks >= 0) ok = phase_wait(bar_y, phase_y);
  if (!ok) atomicCAS(status, 0, kBarrierPollLimit);
  __syncthreads();
  cluster_barrier();
  if (rank == 0 && threadIdx.x == 0) st->t0 += L;
}

// Row j of A^T applied to y_bar: interaction (A^T y_bar - A^T y) . (x_bar - x) and |x_bar - x|^2
// (reference adaptive_step_size_strategy.cu:352-518).
template <typename TX>
struct fpe_epi {
  static constexpr int kRed = 2;
  const TX* aty;
  const TX* xbar;
  const TX* x;
  struct pre_t {
    TX aty, xbar, x;
  };
  __device__ __forceinline__ pre_t load(int j) const { return pre_t{aty[j], xbar[j], x[j]}; }
  __device__ __forceinline__ void operator()(int j, double acc, const pre_t& p, red_t<2>& r) const
  {
    const double d  = acc - (double)p.aty;
    const double dx = (double)p.xbar - (double)p.x;
    r.v[0] += d * dx;
    r.v[1] += dx * dx;
  }
};

// Halpern update for iterations whose step kept x / y (fixed-point-error iterations).
template <typename TX>
__global__ void halpern_kernel(TX* x, const TX* xbar, const TX* xa, int n, TX* y, const TX* ybar,
                               const TX* ya, int m, const pdlp_scalars* st)
{
  const double w = halpern_weight(st, 0);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += gridDim.x * blockDim.x) {
    if (i < n)
      x[i] = (TX)halpern_mix(w, (double)xbar[i], (double)xa[i]);
    else {
      const int r = i - n;
      y[r]        = (TX)halpern_mix(w, (double)ybar[r], (double)ya[r]);
    }
  }
}

static __global__ void advance_kernel(pdlp_scalars* st, int steps) { st->t0 += steps; }
static __global__ void set_scalars_kernel(pdlp_scalars* st, double tau, double sigma, double eta,
                                   double omega, long long t0)
{
  st->tau   = tau;
  st->sigma = sigma;
  st->eta   = eta;
  st->omega = omega;
  st->t0    = t0;
}

// ---------------------------------------------------------------------------------------------
// Termination (reference convergence_information.cu:492-811) on the unscaled FP64 problem.

// x_u = (x_hat dc) / beta ; y_u = (y_hat dr) / gamma ; s_u = (slack / dc) / gamma
// (unscale_solutions, initial_scaling.cu:684-790).
template <typename TX>
__global__ void unscale_kernel(const TX* xhat, const TX* yhat, const TX* slack, const double* dc,
                               const double* dr, double inv_beta, double inv_gamma, int n, int m,
                               double* xu, double* yu, double* su)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += gridDim.x * blockDim.x) {
    if (i < n) {
      const double d = dc[i];
      xu[i]          = ((double)xhat[i] * d) * inv_beta;
      const double s = (double)slack[i];
      su[i]          = (d != 0.0 ? s / d : s) * inv_gamma;
    } else {
      const int r = i - n;
      yu[r]       = ((double)yhat[r] * dr[r]) * inv_gamma;
    }
  }
}

__device__ __forceinline__ double finite_or_zero(double v) { return isfinite(v) ? v : 0.0; }

// Row i of A (unscaled): r_p = Ax - clamp(Ax, lc, uc); primal slack for the dual objective.
struct term_primal_epi {
  static constexpr int kRed = 2;
  const double* lc;
  const double* uc;
  const double* y;
  struct pre_t {
    double l, u, y;
  };
  __device__ __forceinline__ pre_t load(int i) const { return pre_t{lc[i], uc[i], y[i]}; }
  __device__ __forceinline__ void operator()(int i, double ax, const pre_t& p, red_t<2>& r) const
  {
    const double l = p.l, u = p.u;
    const double cl = fmax(l, fmin(ax, u));
    const double rp = ax - cl;
    const double yi = p.y;
    r.v[0] += rp * rp;
    r.v[1] += fmax(yi, 0.0) * finite_or_zero(l) + fmin(yi, 0.0) * finite_or_zero(u);
  }
};

// Row j of A^T (unscaled): r_d = (c - A^T y) - slack; c.x; slack.x.
struct term_dual_epi {
  static constexpr int kRed = 3;
  const double* c;
  const double* x;
  const double* s;
  struct pre_t {
    double c, x, s;
  };
  __device__ __forceinline__ pre_t load(int j) const { return pre_t{c[j], x[j], s[j]}; }
  __device__ __forceinline__ void operator()(int j, double aty, const pre_t& p, red_t<3>& r) const
  {
    const double cj = p.c, xj = p.x, sj = p.s;
    const double rd = (cj - aty) - sj;
    r.v[0] += rd * rd;
    r.v[1] += cj * xj;
    r.v[2] += sj * xj;
  }
};

// Both termination sweeps in one launch (blocks [0, gp) the rows of A, the others the rows of A^T),
// and their sums by the block that finishes last, in finalize_sum_kernel's order, written to the pinned
// host buffer that the host reads once the launch's event has completed (with the two error flags
// behind them, see enqueue_conv).  As two sweeps, two one-block sums and a copy this took five stream
// operations per check; on a 2000 x 5000 LP they were the longer part of it.  arrived must be 0
// before the launch and is 0 after it.
// At 5 resident blocks: 1M x 2M 192 us at 3, 178 at 4, 173 at 5, 187 at 6 (spills); the sums are 28 of them.
constexpr int kCheckBlocks = 5;
static __global__ void __launch_bounds__(kBlock, kCheckBlocks)
  term_kernel(const dev_sell<double> A, const dev_sell<double> AT, const double* __restrict__ xu,
              const double* __restrict__ yu, term_primal_epi ep, term_dual_epi ed, int gp, int gd,
              double* partials, unsigned* arrived, double* host, const int* flag_a, const int* flag_b)
{
  double* part_d = partials + 2 * (size_t)gp;
  if ((int)blockIdx.x < gp)
    sell_map_block(A, xu, ep, partials, (int)blockIdx.x);
  else
    sell_map_block(AT, yu, ed, part_d, (int)blockIdx.x - gp);
  __shared__ int last;
  __syncthreads();  // threads 0 .. 2 wrote the block's partials
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(arrived, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  __shared__ double sums[5];
  ordered_block_sum<2, true>(partials, gp, sums);
  ordered_block_sum<3, true>(part_d, gd, sums + 2);
  if (threadIdx.x < 5) host[threadIdx.x] = sums[threadIdx.x];
  if (threadIdx.x == 0) {
    int* flags = reinterpret_cast<int*>(host + 8);
    flags[0]   = *flag_a;
    flags[1]   = flag_b ? *flag_b : 0;
    *arrived   = 0;
  }
}

// Per-constraint forms of the residuals (per_constraint_residual; reference
// convergence_information.cu:390-420, 453-470 with relative_residual_t, utils.cuh:578-590):
// max(0, max_i r_p,i - rel * max(|l_i|, |u_i|) over the finite bounds (combine_finite_abs_bounds,
// utils.cuh:180-188)) over the rows of A, and max(0, max_j r_d,j - rel * c_j) over the rows of A^T.
struct term_linf_primal_epi {
  static constexpr int kRed     = 1;
  static constexpr bool kMaxRed = true;
  const double* lc;
  const double* uc;
  double rel;
  struct pre_t {
    double l, u;
  };
  __device__ __forceinline__ pre_t load(int i) const { return pre_t{lc[i], uc[i]}; }
  __device__ __forceinline__ void operator()(int, double ax, const pre_t& p, red_t<1>& r) const
  {
    const double rp = ax - fmax(p.l, fmin(ax, p.u));
    double cb       = 0.0;
    if (isfinite(p.u)) cb = fmax(cb, fabs(p.u));
    if (isfinite(p.l)) cb = fmax(cb, fabs(p.l));
    r.v[0] = fmax(r.v[0], rp - rel * cb);
  }
};
struct term_linf_dual_epi {
  static constexpr int kRed     = 1;
  static constexpr bool kMaxRed = true;
  const double* c;
  const double* s;
  double rel;
  struct pre_t {
    double c, s;
  };
  __device__ __forceinline__ pre_t load(int j) const { return pre_t{c[j], s[j]}; }
  __device__ __forceinline__ void operator()(int, double aty, const pre_t& p, red_t<1>& r) const
  {
    const double rd = (p.c - aty) - p.s;
    r.v[0]          = fmax(r.v[0], rd - rel * p.c);
  }
};

// ---------------------------------------------------------------------------------------------
// Reductions over plain vectors (block partials; finalize with finalize_sum_kernel).

// mode 0: sum x^2 ; mode 1: sum (a-b)^2 ; mode 2: bound norm terms of (lo, up)
template <int MODE, typename TA>
__global__ void __launch_bounds__(kBlock) vec_reduce_kernel(const TA* a, const TA* b, int n,
                                                            double* partials)
{
  red_t<1> r;
  r.v[0] = 0.0;
  for (int i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock) {
    if constexpr (MODE == 0) {
      const double v = (double)a[i];
      r.v[0] += v * v;
    } else if constexpr (MODE == 1) {
      const double d = (double)a[i] - (double)b[i];
      r.v[0] += d * d;
    } else {
      const double l = (double)a[i], u = (double)b[i];
      double s       = 0.0;
      if (isfinite(l) && l != u) s += l * l;
      if (isfinite(u)) s += u * u;
      r.v[0] += s;
    }
  }
  block_reduce_store<1>(r, partials);
}

// ---------------------------------------------------------------------------------------------
// Golub-Kahan-Lanczos bidiagonalisation of the scaled A (the step size).  The vectors are stored
// unnormalised; gk_state holds their norms: u has norm beta (beta_k), v has norm alpha
// (alpha_{k-1}, or 0 before the first step), the steps done, and the blocks of the running sweep
// that have finished.
struct gk_state {
  double beta;
  double alpha;
  int step;
  unsigned arrived;
};

// p_j = (A^T u)_j / beta - beta v_j / alpha (no second term before the first step), and
// q_i = (A v)_i / alpha - alpha u_i / beta, rounded the same way in every kernel.
__device__ __forceinline__ double gk_next_v(double acc, double v, double beta, double alpha)
{
  return alpha > 0.0 ? __dsub_rn(acc / beta, __dmul_rn(beta, v / alpha)) : acc / beta;
}
__device__ __forceinline__ double gk_next_u(double acc, double u, double alpha, double beta)
{
  return fma(-alpha, u / beta, acc / alpha);
}

// Row j of A^T applied to u:  p_j = (A^T u)_j / beta - beta v_j / alpha  (written over v_j).
struct gk_primal_epi {
  static constexpr int kRed = 1;
  double* v;
  double beta = 0.0, alpha = 0.0;  // set by the kernel
  struct pre_t {
    double v;
  };
  __device__ __forceinline__ pre_t load(int j) const { return pre_t{v[j]}; }
  __device__ __forceinline__ void operator()(int j, double acc, const pre_t& p, red_t<1>& r) const
  {
    const double pj = gk_next_v(acc, p.v, beta, alpha);
    v[j]            = pj;
    r.v[0] += pj * pj;
  }
};

// Row i of A applied to v:  q_i = (A v)_i / alpha - alpha u_i / beta  (written over u_i).
struct gk_dual_epi {
  static constexpr int kRed = 1;
  double* u;
  double beta = 0.0, alpha = 0.0;
  struct pre_t {
    double u;
  };
  __device__ __forceinline__ pre_t load(int i) const { return pre_t{u[i]}; }
  __device__ __forceinline__ void operator()(int i, double acc, const pre_t& p, red_t<1>& r) const
  {
    const double qi = gk_next_u(acc, p.u, alpha, beta);
    u[i]            = qi;
    r.v[0] += qi * qi;
  }
};

// The norm |z0| that the recurrence starts from: beta and the first entry of its history.
static __global__ void gk_start_kernel(gk_state* st, const double* sumsq, double* betas)
{
  st->beta = betas[0] = sqrt(*sumsq);
}

// One half step: the sweep with its fused recurrence, and the norm of the new vector, which the
// block that finishes last sums from the block partials (in the order of finalize_sum_kernel).
// FIELD 0 (rows of A^T) records alpha of the step, FIELD 1 (rows of A) beta, and moves the step on.
// A step is two launches; with the sum and its recording as kernels of their own it was six, and
// on a 12k x 30k LP those four one-block kernels were the larger part of it.
template <int FIELD, typename TM, class Epi>
__global__ void __launch_bounds__(kBlock, kSweepBlocks<TM, Epi>)
  gk_sweep_kernel(const dev_sell<TM> A, const double* __restrict__ g, Epi epi, double* partials,
                  gk_state* st, double* hist)
{
  epi.beta  = st->beta;
  epi.alpha = st->alpha;
  sell_map_block(A, g, epi, partials, (int)blockIdx.x);
  __shared__ int last;
  if (threadIdx.x == 0) {  // the thread that wrote this block's partial
    __threadfence();
    last = atomicAdd(&st->arrived, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  __shared__ double total;
  ordered_block_sum<1, true>(partials, (int)gridDim.x, &total);
  if (threadIdx.x == 0) {
    const double v = sqrt(total);
    const int k    = st->step;
    if (FIELD == 0) {
      st->alpha = v;
      hist[k]   = v;
    } else {
      st->beta    = v;
      hist[k + 1] = v;
      st->step    = k + 1;
    }
    st->arrived = 0;
  }
}

// sqrt of the sum of at most kBlock block partials, in ordered_block_sum's tree, by every warp.
__device__ __forceinline__ double gk_tree(double (&e)[kBlock / kWarp])
{
#pragma unroll
  for (int h = kBlock / kWarp / 2; h > 0; h >>= 1)
#pragma unroll
    for (int j = 0; j < h; ++j) e[j] += e[j + h];
#pragma unroll
  for (int h = kWarp / 2; h > 0; h >>= 1) e[0] += __shfl_down_sync(0xffffffffu, e[0], h);
  return sqrt(__shfl_sync(0xffffffffu, e[0], 0));
}
__device__ __forceinline__ double gk_partials_norm(const double* partials, int blocks)
{
  double e[kBlock / kWarp];
#pragma unroll
  for (int j = 0; j < kBlock / kWarp; ++j) {
    const int b = (threadIdx.x & 31) + j * kWarp;
    e[j]        = b < blocks ? partials[b] : 0.0;
  }
  return gk_tree(e);
}

// The half step of an LP whose sweeps have at most kBlock blocks: the norm of the vector gathered
// is formed at the start of the sweep, by every warp from the `nin` block partials of the sweep
// before (nin 0: it is in st), instead of at the end of that sweep.  There, the fence, the count of
// blocks and the sums of the last one follow one another: a half step on a 12 007 x 30 011 LP took
// 7.7 us and takes 6.6 us.  With more partials every block would read more than one a thread.
template <int FIELD, typename TM, class Epi>
__global__ void __launch_bounds__(kBlock, kSweepBlocks<TM, Epi>)
  gk_chain_kernel(const dev_sell<TM> A, const double* __restrict__ g, Epi epi, const double* pin,
                  int nin, double* pout, gk_state* st, double* hist, int k)
{
  double& own = FIELD == 0 ? st->beta : st->alpha;  // written by block 0, read by later kernels
  const double norm = nin > 0 ? gk_partials_norm(pin, nin) : own;
  epi.beta          = FIELD == 0 ? norm : st->beta;
  epi.alpha         = FIELD == 0 ? st->alpha : norm;
  if (nin > 0 && blockIdx.x == 0 && threadIdx.x == 0) own = hist[k] = norm;
  sell_map_block(A, g, epi, pout, (int)blockIdx.x);
}
// beta after the last step of a chain.
static __global__ void gk_chain_end_kernel(const double* partials, int blocks, gk_state* st,
                                           double* betas, int k)
{
  const double norm = gk_partials_norm(partials, blocks);
  if (threadIdx.x == 0) {
    st->beta = betas[k] = norm;
    st->step = k;
  }
}

// `steps` steps of the recurrence for a small LP in one launch: a cluster of C blocks whose blocks
// keep copies of u and v and their shares of the matrices (the images of the resident form) in
// shared memory.  A half step is this block's products, its new entries sent to every copy, one
// cluster barrier and the norm, formed as gk_sweep_kernel forms it: the sum of every warp goes to
// its place in ws (8 per block of the sweep's grid, in every copy), each block's 8 are added in order,
// and the blocks' in ordered_block_sum's tree (at most kBlock blocks: one partial a thread), so both
// forms give the same coefficients bit for bit.  Two launches a step took 22 us on a 2000 x 5000 LP.
constexpr int kClusterGkSums = kBlock * kWarpsPerBlock;  // most entries of ws per sweep
template <typename TX>
B200_HD inline size_t cluster_gk_smem(int m, int n, int gt, int ga, const resident_dims& D)
{
  return resident_dims::vector_bytes<double>(m, n) +
         (size_t)(gt + ga) * kWarpsPerBlock * sizeof(double) + D.image_bytes<TX>();
}
// The place in ws of the sum of the warp that takes unit u of M.
template <typename TX>
__device__ __forceinline__ int unit_sum(const dev_sell<TX>& M, int u)
{
  if (u < M.n_wide) return u * kWarpsPerBlock;
  const int q = u < M.n_long ? u - M.n_wide : u - M.n_long;
  return (u < M.n_long ? M.n_wide : row_blocks(M)) * kWarpsPerBlock + q;
}
__device__ __forceinline__ double cluster_gk_norm(const double* ws, int blocks)
{
  const int lane = threadIdx.x & 31;
  double e[kBlock / kWarp];
#pragma unroll
  for (int j = 0; j < kBlock / kWarp; ++j) {
    const int b = lane + j * kWarp;
    double t    = 0.0;
    if (b < blocks)
      for (int w = 0; w < kWarpsPerBlock; ++w) t += ws[b * kWarpsPerBlock + w];
    e[j] = t;
  }
  return gk_tree(e);
}

template <typename TX>
__global__ void __launch_bounds__(kResidentThreads, 1)
  cluster_gk_kernel(const dev_sell<TX> AT, const dev_sell<TX> A, double* u_out, double* v_out,
                    gk_state* st, double* alphas, double* betas, int steps, int m, int n,
                    resident_dims D, const unsigned char* images)
{
  extern __shared__ __align__(16) unsigned char gk_smem[];
  const unsigned rank = cluster_rank(), blocks = cluster_size();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int grid[2] = {sweep_grid(AT), sweep_grid(A)};
  double* u  = reinterpret_cast<double*>(gk_smem);
  double* v  = reinterpret_cast<double*>(gk_smem + resident_dims::pad((size_t)m * 8));
  double* ws = reinterpret_cast<double*>(gk_smem + resident_dims::vector_bytes<double>(m, n));
  unsigned char* img = reinterpret_cast<unsigned char*>(ws + (grid[0] + grid[1]) * kWarpsPerBlock);
  {
    const size_t bytes       = D.image_bytes<TX>();
    const unsigned char* src = images + rank * bytes;
    for (size_t b = (size_t)threadIdx.x * 16; b < bytes; b += kResidentThreads * 16)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(img + b)),
                   "l"(src + b)
                   : "memory");
  }
  for (int i = threadIdx.x; i < m; i += kResidentThreads) u[i] = u_out[i];
  for (int i = threadIdx.x; i < n; i += kResidentThreads) v[i] = v_out[i];
  for (int i = threadIdx.x; i < (grid[0] + grid[1]) * kWarpsPerBlock; i += kResidentThreads)
    ws[i] = 0.0;
  double beta = st->beta, alpha = st->alpha;
  const int k0 = st->step;
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  // Every block is running, with its copies, before any stores into another's shared memory (and
  // has read the state before block 0 writes it).
  cluster_barrier();
  // The half step of matrix M (w = 0: rows of A^T from u to v, w = 1: rows of A from v to u).
  auto half = [&](const dev_sell<TX>& M, int w, const double* g, double* own, double nrm,
                  double other) {
    const int total             = M.n_long + M.n_slices;
    const int2* tab             = reinterpret_cast<const int2*>(img + D.image_at<TX>(w));
    const TX* val               = reinterpret_cast<const TX*>(img + D.image_at<TX>(4 + w));
    const unsigned short* idx   = reinterpret_cast<const unsigned short*>(img + D.image_at<TX>(6 + w));
    double* sums                = ws + (w == 0 ? 0 : grid[0] * kWarpsPerBlock);
    for (int i = warp; i < D.units[w]; i += kResidentWarps) {
      const int q = (int)rank + D.blocks * i;
      if (q >= total) break;
      const int2 t = tab[i];
      int row      = -1;
      double acc;
      if (q < M.n_long) {
        if (lane == 0) row = q;
        acc = resident_long(val + t.x, idx + t.x, t.y, g, q < M.n_wide);
      } else {
        row = M.n_long + (q - M.n_long) * kWarp + lane;
        if (row >= M.rows) row = -1;
        acc = resident_slice(val + t.x + lane * kChunk, idx + t.x + lane * kChunk, t.y >> 7, g);
      }
      double sq = 0.0;
      if (row >= 0) {
        const double e = w == 0 ? gk_next_v(acc, own[row], nrm, other)
                                : gk_next_u(acc, own[row], nrm, other);
        const unsigned at = (unsigned)__cvta_generic_to_shared(own + row);
        for (unsigned c = 0; c < blocks; ++c) dsmem_store(at, c, e);
        sq = e * e;
      }
      sq = warp_sum(sq);
      if (lane < (int)blocks)
        dsmem_store((unsigned)__cvta_generic_to_shared(sums + unit_sum(M, q)), lane, sq);
    }
    cluster_barrier();
    return cluster_gk_norm(sums, grid[w]);
  };
  for (int k = 0; k < steps; ++k) {
    alpha = half(AT, 0, u, v, beta, alpha);
    beta  = half(A, 1, v, u, alpha, beta);
    if (rank == 0 && threadIdx.x == 0) {
      alphas[k0 + k]    = alpha;
      betas[k0 + k + 1] = beta;
    }
  }
  if (rank == 0) {
    for (int i = threadIdx.x; i < m; i += kResidentThreads) u_out[i] = u[i];
    for (int i = threadIdx.x; i < n; i += kResidentThreads) v_out[i] = v[i];
    if (threadIdx.x == 0) {
      st->beta  = beta;
      st->alpha = alpha;
      st->step  = k0 + steps;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Scaling (reference initial_scaling.cu:152-569).

// One pass of the scaling: for every row of A, drn_i = dr_i / sqrt(v_i) with v_i = max_k |a_ik dr_i
// dc_k| (MODE 0) or sum_k |a_ik dr_i dc_k|^alpha_r (MODE 1), and for every row of A^T the same with
// dc (a_divides_sqrt_b_bounded, utils.cuh:156-163: unchanged where v is 0).  Both sides read the old
// factors, so they run in one launch (blocks [0, ga) the rows of A) that writes the new ones beside
// them; as two sweeps and two vector steps a pass was four launches, and the 11 passes the longer
// part of a small LP's scaling.
template <int MODE, bool TRANSPOSED>
__device__ __forceinline__ void scale_pass_block(const dev_sell<double>& A, const double* dr,
                                                 const double* dc, double alpha, double* out, int vb)
{
  const double* own = TRANSPOSED ? dc : dr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lb   = long_blocks(A.n_long);
  auto term      = [&](double v, int row, int col) {
    const double p = TRANSPOSED ? (v * dr[col]) * dc[row] : (v * dr[row]) * dc[col];
    const double a = fabs(p);
    return MODE == 0 ? a : pow(a, alpha);
  };
  auto store = [&](int row, double v) {
    const double d = own[row];
    out[row]       = v > 0.0 ? d / sqrt(v) : d;
  };
  if (vb < lb) {
    const int row = vb * kWarpsPerBlock + warp;
    if (row < A.n_long) {
      double acc = 0.0;
      for (int64_t k = A.long_off[row] + lane; k < A.long_off[row + 1]; k += kWarp) {
        const double t = term(A.val[k], row, A.idx[k]);
        acc            = MODE == 0 ? fmax(acc, t) : acc + t;
      }
      acc = MODE == 0 ? warp_max(acc) : warp_sum(acc);
      if (lane == 0) store(row, acc);
    }
  } else {
    const int s = (vb - lb) * kWarpsPerBlock + warp;
    if (s < A.n_slices) {
      const int64_t base = A.slice_off[s];
      const int len      = (int)((A.slice_off[s + 1] - base) >> 5);
      const int row      = A.n_long + s * kWarp + lane;
      if (row < A.rows) {
        double acc = 0.0;
        for (int k = 0; k < len; ++k) {
          const int64_t p = sell_pos(base, k, lane);
          const double v  = A.val[p];
          if (v == 0.0) continue;  // padding (and explicit zeros, which contribute nothing)
          const double t = term(v, row, A.idx[p]);
          acc            = MODE == 0 ? fmax(acc, t) : acc + t;
        }
        store(row, acc);
      }
    }
  }
}
template <int MODE>
__global__ void __launch_bounds__(kBlock)
  scale_pass_kernel(const dev_sell<double> A, const dev_sell<double> AT, const double* dr,
                    const double* dc, double alpha_r, double alpha_c, double* drn, double* dcn,
                    int ga)
{
  if ((int)blockIdx.x < ga)
    scale_pass_block<MODE, false>(A, dr, dc, alpha_r, drn, (int)blockIdx.x);
  else
    scale_pass_block<MODE, true>(AT, dr, dc, alpha_c, dcn, (int)blockIdx.x - ga);
}

// Ruiz (`ruiz` passes) then Pock-Chambolle (reference initial_scaling.cu:152-365) on factors that
// start at 1 in dr / dc; rt / ct: buffers of the same lengths.  Returns the launches.
inline int scale_passes(const dev_sell<double>& A, const dev_sell<double>& AT, int ruiz, double alpha,
                        dbuf<double>& dr, dbuf<double>& dc, dbuf<double>& rt, dbuf<double>& ct,
                        cudaStream_t s)
{
  const int ga = sell_grid(A), g = ga + sell_grid(AT);
  for (int it = 0; it <= ruiz; ++it) {
    if (it < ruiz)
      scale_pass_kernel<0><<<g, kBlock, 0, s>>>(A, AT, dr.data(), dc.data(), 0.0, 0.0, rt.data(),
                                               ct.data(), ga);
    else
      scale_pass_kernel<1><<<g, kBlock, 0, s>>>(A, AT, dr.data(), dc.data(), alpha, 2.0 - alpha,
                                               rt.data(), ct.data(), ga);
    std::swap(dr, rt);
    std::swap(dc, ct);
  }
  B200_LAUNCH_CHECK();
  return ruiz + 1;
}

// Scaled copy of the matrix values: A_s = (a dr_i) dc_j, A^T_s = (a dc_j) dr_i.
template <typename TM, bool TRANSPOSED>
__global__ void __launch_bounds__(kBlock) scale_values_kernel(const dev_sell<double> A,
                                                              const double* dr, const double* dc,
                                                              TM* out)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lb   = long_blocks(A.n_long);
  auto scaled    = [&](double v, int row, int col) {
    return TRANSPOSED ? (v * dc[row]) * dr[col] : (v * dr[row]) * dc[col];
  };
  if ((int)blockIdx.x < lb) {
    const int row = blockIdx.x * kWarpsPerBlock + warp;
    if (row < A.n_long)
      for (int64_t k = A.long_off[row] + lane; k < A.long_off[row + 1]; k += kWarp)
        out[k] = (TM)scaled(A.val[k], row, A.idx[k]);
  } else {
    const int s = (blockIdx.x - lb) * kWarpsPerBlock + warp;
    if (s < A.n_slices) {
      const int64_t base = A.slice_off[s];
      const int len      = (int)((A.slice_off[s + 1] - base) >> 5);
      const int row      = A.n_long + s * kWarp + lane;
      for (int k = 0; k < len; ++k) {
        const int64_t p = sell_pos(base, k, lane);
        out[p]          = row < A.rows ? (TM)scaled(A.val[p], row, A.idx[p]) : (TM)0;
      }
    }
  }
}

// First pass of the vector scaling: c*dc, bounds/dc (divide_check_zero), constraint bounds*dr.
static __global__ void scale_vectors_kernel(const double* c, const double* l, const double* u,
                                     const double* lc, const double* uc, const double* dc,
                                     const double* dr, int n, int m, double* cs, double* ls,
                                     double* us, double* lcs, double* ucs)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += gridDim.x * blockDim.x) {
    if (i < n) {
      const double d = dc[i];
      cs[i]          = c[i] * d;
      if (d == 0.0) {
        ls[i] = 0.0;
        us[i] = 0.0;
      } else {
        ls[i] = l[i] / d;
        us[i] = u[i] / d;
      }
    } else {
      const int r = i - n;
      lcs[r]      = lc[r] * dr[r];
      ucs[r]      = uc[r] * dr[r];
    }
  }
}

// Second pass: bound rescaling beta and objective rescaling gamma; converts to the iterate type.
template <typename TX>
__global__ void rescale_vectors_kernel(const double* cs, const double* ls, const double* us,
                                       const double* lcs, const double* ucs, double beta,
                                       double gamma, int n, int m, TX* c_out, TX* l_out, TX* u_out,
                                       TX* lc_out, TX* uc_out)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += gridDim.x * blockDim.x) {
    if (i < n) {
      c_out[i] = (TX)(cs[i] * gamma);
      l_out[i] = (TX)(ls[i] * beta);
      u_out[i] = (TX)(us[i] * beta);
    } else {
      const int r = i - n;
      lc_out[r]   = (TX)(lcs[r] * beta);
      uc_out[r]   = (TX)(ucs[r] * beta);
    }
  }
}

// Initial iterate in scaled space: v / d (d != 0) times factor, written to three buffers
// (scale_solutions, initial_scaling.cu:571-640).
template <typename TX>
__global__ void scale_initial_kernel(const double* v, const double* d, double factor, int n, TX* a,
                                     TX* b, TX* c)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double s = d[i] != 0.0 ? v[i] / d[i] : v[i];
    const TX w     = (TX)(s * factor);
    a[i]           = w;
    b[i]           = w;
    c[i]           = w;
  }
}

// ---------------------------------------------------------------------------------------------
// Infeasibility detection (reference infeasibility_information.cu:230-490, the cuPDLPx branch).
// The rays are the step's deltas x_bar - x and y_bar - y in the scaled space, clamped to the
// recession cones of the bounds.

// d_j = clamp(x_bar_j - x_j) (>= 0 on a finite lower bound, <= 0 on a finite upper bound) and
// cd_j = c_j d_j;  e_i = clamp(y_bar_i - y_i) (<= 0 without a finite lower bound, >= 0 without a
// finite upper bound) and pe_i = max(e_i, 0) fin(lc_i) + min(e_i, 0) fin(uc_i).
template <typename TX>
__global__ void ray_vectors_kernel(const TX* x, const TX* xbar, const TX* l, const TX* u,
                                   const TX* c, int n, const TX* y, const TX* ybar, const TX* lc,
                                   const TX* uc, int m, double* d, double* cd, double* e,
                                   double* pe)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += gridDim.x * blockDim.x) {
    if (i < n) {
      double v = (double)xbar[i] - (double)x[i];
      if (isfinite((double)l[i])) v = fmax(v, 0.0);
      if (isfinite((double)u[i])) v = fmin(v, 0.0);
      d[i]  = v;
      cd[i] = (double)c[i] * v;
    } else {
      const int r = i - n;
      double v    = (double)ybar[r] - (double)y[r];
      if (!isfinite((double)lc[r])) v = fmin(v, 0.0);
      if (!isfinite((double)uc[r])) v = fmax(v, 0.0);
      e[r]  = v;
      pe[r] = fmax(v, 0.0) * finite_or_zero((double)lc[r]) + fmin(v, 0.0) * finite_or_zero((double)uc[r]);
    }
  }
}

// Row i of A applied to d: violation of the primal ray, (max(-Ad, 0) [lc finite] +
// max(Ad, 0) [uc finite]) dr_i with Ad scaled by 1 / |d|_inf.
template <typename TX>
struct ray_primal_epi {
  static constexpr int kRed = 0;
  const TX* lc;
  const TX* uc;
  const double* dr;
  double inv_norm;
  double* out;
  struct pre_t {};
  __device__ __forceinline__ pre_t load(int) const { return pre_t{}; }
  __device__ __forceinline__ void operator()(int i, double acc, const pre_t&, red_t<0>&) const
  {
    const double ad = acc * inv_norm;
    out[i]          = (fmax(-ad, 0.0) * (isfinite((double)lc[i]) ? 1.0 : 0.0) +
              fmax(ad, 0.0) * (isfinite((double)uc[i]) ? 1.0 : 0.0)) *
             dr[i];
  }
};

// Row j of A^T applied to e (g = (A^T e)_j): dual-slack objective term and dual-ray violation.
template <typename TX>
struct ray_dual_epi {
  static constexpr int kRed = 0;
  const TX* l;
  const TX* u;
  const double* dc;
  double* slack_term;
  double* violation;
  struct pre_t {};
  __device__ __forceinline__ pre_t load(int) const { return pre_t{}; }
  __device__ __forceinline__ void operator()(int j, double g, const pre_t&, red_t<0>&) const
  {
    const double lj = (double)l[j], uj = (double)u[j];
    slack_term[j] = fmax(-g, 0.0) * finite_or_zero(lj) + fmin(-g, 0.0) * finite_or_zero(uj);
    violation[j]  = (fmax(-g, 0.0) * (isfinite(lj) ? 0.0 : 1.0) -
                    fmin(-g, 0.0) * (isfinite(uj) ? 0.0 : 1.0)) *
                   dc[j];
  }
};

// Per-block sum (MAX = false) or maximum of |a| (MAX = true) into partials[blockIdx.x].
template <bool MAX>
__global__ void __launch_bounds__(kBlock) block_stat_kernel(const double* a, int n, double* partials)
{
  __shared__ double sm[kBlock];
  double v = 0.0;
  for (int i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock)
    v = MAX ? fmax(v, fabs(a[i])) : v + a[i];
  sm[threadIdx.x] = v;
  __syncthreads();
  for (int h = kBlock / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h)
      sm[threadIdx.x] = MAX ? fmax(sm[threadIdx.x], sm[threadIdx.x + h])
                            : sm[threadIdx.x] + sm[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) partials[blockIdx.x] = sm[0];
}

// Elementwise helpers
template <typename TX>
__global__ void clamp_kernel(TX* x, const TX* l, const TX* u, int n)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    x[i] = (TX)fmin(fmax((double)x[i], (double)l[i]), (double)u[i]);
}

template <typename TA, typename TB>
__global__ void copy_convert_kernel(TB* dst, const TA* src, int n)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    dst[i] = (TB)src[i];
}

}  // namespace cuopt_b200
