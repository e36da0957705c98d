// Batched PDLP: many independent LPs solved together as one block-diagonal LP.
//
// Counterpart of the reference's batch solve (the Python BatchSolve through
// cuopt::cython::call_batch_solve, cpp/src/pdlp/utilities/cython_solve.cu:317-352, which runs one
// PDLP per problem on host threads) and of its batch climbers (cpp/src/pdlp/pdlp.cu:1447-1746).
// Here the instances are concatenated into one block-diagonal matrix and every PDHG sweep is one
// launch over all of them; each row reads the step sizes of its own instance.  Every instance
// keeps its own Stable3 state — scaling factors, step size (its own power iteration), primal
// weight, restart / PID state and termination — and follows the schedule of a single solve: that
// schedule depends only on the iteration count, which all instances share.  An instance that
// terminates is frozen: the sweeps skip its rows and no kernel writes its vectors again.
//
// Per-instance sums (norms, residuals, fixed-point errors) are formed deterministically: the
// epilogues write one value per row into a row buffer, and one block per instance adds its rows in
// a fixed order (the layout keeps every instance's rows contiguous inside the long-row and the
// sliced parts, see make_keys_kernel).
#include "device_layout.cuh"
#include "host_io.hpp"
#include "kernels.cuh"
#include "pdlp_engine.hpp"
#include "pdlp_schedule.hpp"
#include "plain_form.hpp"

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <map>
#include <tuple>
#include <random>
#include <stdexcept>

namespace cuopt_b200 {

namespace {

double now_s()
{
  return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

template <typename T>
dev_sell<T> bview(const dev_matrix& M, const T* v)
{
  return dev_sell<T>{M.rows, M.n_long, M.n_slices, M.long_off.data(), M.slice_off.data(),
                     M.idx.data(), v};
}

// ------------------------------------------------------------------------------------------------
// Device side

// Instance lookup shared by the batch epilogues.
struct inst_ctx {
  const int* inst;         // instance of every internal row of the swept matrix
  const int* active;       // per instance: still iterating
  const pdlp_scalars* sc;  // per instance step scalars
  // Rows r0..r1 lie in one class (long or sliced), where instances are sorted, so the instances
  // present are inst[r0]..inst[r1].
  __device__ __forceinline__ bool all_frozen(int r0, int r1) const
  {
    for (int b = inst[r0]; b <= inst[r1]; ++b)
      if (active[b]) return false;
    return true;
  }
};

template <typename TX, bool MAJOR, bool HALPERN, bool SAVE_ATY>
struct b_primal_epi {
  static constexpr int kRed = 0;
  const TX *x, *c, *lo, *up, *xa;
  TX *xbar, *xout, *xhat, *slack, *aty;
  inst_ctx ctx;
  int it_off;
  struct pre_t {
    TX x, c, lo, up, xa;
    int b;
  };
  __device__ bool skip_range(int r0, int r1) const { return ctx.all_frozen(r0, r1); }
  __device__ __forceinline__ pre_t load(int j) const
  {
    return pre_t{x[j], c[j], lo[j], up[j], HALPERN ? xa[j] : TX(0), ctx.inst[j]};
  }
  __device__ __forceinline__ void operator()(int j, double acc, const pre_t& p, red_t<0>&) const
  {
    if (!ctx.active[p.b]) return;
    primal_row_step<TX, MAJOR, HALPERN, SAVE_ATY>(j, acc, p, ctx.sc + p.b, it_off, xbar, xout,
                                                  xhat, slack, aty);
  }
};

// FPE: rowbuf[i] = (y_bar_i - y_i)^2.
template <typename TX, bool MAJOR, bool HALPERN, bool FPE>
struct b_dual_epi {
  static constexpr int kRed = 0;
  const TX *y, *lo, *up, *ya;
  TX *ybar, *yout, *yhat;
  double* rowbuf;
  inst_ctx ctx;
  int it_off;
  struct pre_t {
    TX y, lo, up, ya;
    int b;
  };
  __device__ bool skip_range(int r0, int r1) const { return ctx.all_frozen(r0, r1); }
  __device__ __forceinline__ pre_t load(int i) const
  {
    return pre_t{y[i], lo[i], up[i], HALPERN ? ya[i] : TX(0), ctx.inst[i]};
  }
  __device__ __forceinline__ void operator()(int i, double acc, const pre_t& p, red_t<0>&) const
  {
    if (!ctx.active[p.b]) return;
    const double d2 =
      dual_row_step<TX, MAJOR, HALPERN>(i, acc, p, ctx.sc + p.b, it_off, ybar, yout, yhat);
    if constexpr (FPE) rowbuf[i] = d2;
  }
};

// rowbuf[j] = (A^T y_bar - A^T y)_j (x_bar - x)_j ; rowbuf[stride + j] = (x_bar - x)_j^2.
template <typename TX>
struct b_fpe_epi {
  static constexpr int kRed = 0;
  const TX *aty, *xbar, *x;
  double* rowbuf;
  size_t stride;
  inst_ctx ctx;
  struct pre_t {
    TX aty, xbar, x;
    int b;
  };
  __device__ bool skip_range(int r0, int r1) const { return ctx.all_frozen(r0, r1); }
  __device__ __forceinline__ pre_t load(int j) const
  {
    return pre_t{aty[j], xbar[j], x[j], ctx.inst[j]};
  }
  __device__ __forceinline__ void operator()(int j, double acc, const pre_t& p, red_t<0>&) const
  {
    if (!ctx.active[p.b]) return;
    const double d  = acc - (double)p.aty;
    const double dx = (double)p.xbar - (double)p.x;
    rowbuf[j]          = d * dx;
    rowbuf[stride + j] = dx * dx;
  }
};

// Unscaled termination terms of row i of A: rp^2 and the dual-objective bound term.
struct b_term_primal_epi {
  static constexpr int kRed = 0;
  const double *lc, *uc, *y;
  double* rowbuf;
  size_t stride;
  inst_ctx ctx;
  struct pre_t {
    double l, u, y;
    int b;
  };
  __device__ bool skip_range(int r0, int r1) const { return ctx.all_frozen(r0, r1); }
  __device__ __forceinline__ pre_t load(int i) const
  {
    return pre_t{lc[i], uc[i], y[i], ctx.inst[i]};
  }
  __device__ __forceinline__ void operator()(int i, double ax, const pre_t& p, red_t<0>&) const
  {
    if (!ctx.active[p.b]) return;
    const double cl = fmax(p.l, fmin(ax, p.u));
    const double rp = ax - cl;
    rowbuf[i]          = rp * rp;
    rowbuf[stride + i] = fmax(p.y, 0.0) * finite_or_zero(p.l) + fmin(p.y, 0.0) * finite_or_zero(p.u);
  }
};

// Unscaled termination terms of row j of A^T: rd^2, c.x, s.x.
struct b_term_dual_epi {
  static constexpr int kRed = 0;
  const double *c, *x, *s;
  double* rowbuf;
  size_t stride;
  inst_ctx ctx;
  struct pre_t {
    double c, x, s;
    int b;
  };
  __device__ bool skip_range(int r0, int r1) const { return ctx.all_frozen(r0, r1); }
  __device__ __forceinline__ pre_t load(int j) const
  {
    return pre_t{c[j], x[j], s[j], ctx.inst[j]};
  }
  __device__ __forceinline__ void operator()(int j, double aty, const pre_t& p, red_t<0>&) const
  {
    if (!ctx.active[p.b]) return;
    const double rd        = (p.c - aty) - p.s;
    rowbuf[j]              = rd * rd;
    rowbuf[stride + j]     = p.c * p.x;
    rowbuf[2 * stride + j] = p.s * p.x;
  }
};

// Rows of an instance are processed in chunks of at most kChunkRows (each inside one instance), so
// a large instance does not serialise a kernel on one block.
constexpr int kChunkRows = 2048;

// Per-instance sums of row-buffer planes, for instances of any size: block c sums the K planes over its
// chunk (instance chunks[c].x, rows [chunks[c].y, chunks[c].z)) into part[c K + q]; then one
// thread per instance adds its chunks in chunk order.
template <int K>
__global__ void __launch_bounds__(kBlock) chunk_reduce_kernel(const double* rowbuf, size_t stride,
                                                              const int4* chunks, const int* want,
                                                              double* part)
{
  const int4 ch = chunks[blockIdx.x];
  if (want && !want[ch.x]) return;
  __shared__ double sm[kBlock];
  for (int q = 0; q < K; ++q) {
    const double* v = rowbuf + (size_t)q * stride;
    ksum acc;
    for (int i = ch.y + threadIdx.x; i < ch.z; i += kBlock) acc.add(v[i]);
    sm[threadIdx.x] = acc.value();
    __syncthreads();
    for (int h = kBlock / 2; h > 0; h >>= 1) {
      if (threadIdx.x < h) sm[threadIdx.x] += sm[threadIdx.x + h];
      __syncthreads();
    }
    if (threadIdx.x == 0) part[(size_t)blockIdx.x * K + q] = sm[0];
    __syncthreads();
  }
}

template <int K>
__global__ void instance_reduce_kernel(const double* part, const int* chunk_off, int count,
                                       const int* want, double* out)
{
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < count; b += gridDim.x * blockDim.x) {
    if (want && !want[b]) continue;
    for (int q = 0; q < K; ++q) {
      double t = 0.0;
      for (int c = chunk_off[b]; c < chunk_off[b + 1]; ++c) t += part[(size_t)c * K + q];
      out[(size_t)b * K + q] = t;
    }
  }
}

// Both termination sweeps of a check in one launch (blocks [0, gp) the rows of A, the others the rows
// of A^T; each writes planes of its own), and the per-instance sums of both in another: block c sums
// the planes of its chunk (chunks of rows, then chunks of columns), and the block that finishes last of
// its instance and side adds the instance's chunks in order into the pinned host buffer that the
// host reads once the launch's event has completed (2 values per instance, then 3).
__global__ void __launch_bounds__(kBlock, kCheckBlocks)
  b_term_kernel(const dev_sell<double> A, const dev_sell<double> AT, const double* __restrict__ xu,
                const double* __restrict__ yu, b_term_primal_epi ep, b_term_dual_epi ed, int gp)
{
  if ((int)blockIdx.x < gp)
    sell_map_block(A, xu, ep, nullptr, (int)blockIdx.x);
  else
    sell_map_block(AT, yu, ed, nullptr, (int)blockIdx.x - gp);
}

// Fixed-order block sum of per-thread values (compensated per thread, then a fixed tree).
__device__ __forceinline__ double block_sum(const ksum& acc, double* sm)
{
  sm[threadIdx.x] = acc.value();
  __syncthreads();
  for (int h = kBlock / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h) sm[threadIdx.x] += sm[threadIdx.x + h];
    __syncthreads();
  }
  const double v = sm[0];
  __syncthreads();
  return v;
}

struct b_side {  // one side (rows or columns) of a check's sums
  const int4* chunks;
  const int* offsets;
  int count;            // chunks
  const double* planes;
  double* part;
  unsigned* arrived;    // per instance; 0 before and after
  double* host;
};
template <int K>
__device__ __forceinline__ void b_term_side(const b_side& S, int c, size_t stride, const int* want)
{
  const int4 ch = S.chunks[c];
  if (!want[ch.x]) return;
  __shared__ double sm[kBlock];
  ksum acc[K];
  for (int i = ch.y + threadIdx.x; i < ch.z; i += kBlock)
#pragma unroll
    for (int q = 0; q < K; ++q) acc[q].add(S.planes[q * stride + i]);
  double t[K];
#pragma unroll
  for (int q = 0; q < K; ++q) t[q] = block_sum(acc[q], sm);
  if (threadIdx.x != 0) return;
#pragma unroll
  for (int q = 0; q < K; ++q) S.part[(size_t)c * K + q] = t[q];
  const int c0 = S.offsets[ch.x], c1 = S.offsets[ch.x + 1];
  __threadfence();
  if (atomicAdd(S.arrived + ch.x, 1u) != (unsigned)(c1 - c0 - 1)) return;
  __threadfence();
  double sum[K] = {};
  for (int d = c0; d < c1; ++d)
#pragma unroll
    for (int q = 0; q < K; ++q) sum[q] += __ldcg(S.part + (size_t)d * K + q);
#pragma unroll
  for (int q = 0; q < K; ++q) S.host[(size_t)ch.x * K + q] = sum[q];
  S.arrived[ch.x] = 0;
}
__global__ void __launch_bounds__(kBlock) b_term_sums_kernel(b_side rows, b_side cols, size_t stride,
                                                             const int* want)
{
  if ((int)blockIdx.x < rows.count)
    b_term_side<2>(rows, (int)blockIdx.x, stride, want);
  else
    b_term_side<3>(cols, (int)blockIdx.x - rows.count, stride, want);
}

// Elementwise fills of the row buffer.
template <typename TA>
__global__ void sq_diff_kernel(const TA* a, const TA* b, int n, double* out)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double d = b ? (double)a[i] - (double)b[i] : (double)a[i];
    out[i]         = d * d;
  }
}
__global__ void bound_terms_kernel(const double* lo, const double* up, int n, double* out)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double l = lo[i], u = up[i];
    double s       = 0.0;
    if (isfinite(l) && l != u) s += l * l;
    if (isfinite(u)) s += u * u;
    out[i] = s;
  }
}

// Instance ranges in the internal order, where each instance's items are contiguous inside
// [0, n_long) and inside [n_long, count): r[b] = {long_lo, long_hi, short_lo, short_hi}.  Segment
// starts and ends are found where the instance id changes; an id out of [0, B) or a decrease
// inside a part (instances not contiguous) is counted in bad[0].  r must be zeroed first.
__global__ void instance_ranges_kernel(const int* inst, int count, int n_long, int B, int4* r,
                                       int* bad)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const int b = inst[i];
    if (b < 0 || b >= B) {
      atomicAdd(bad, 1);
      continue;
    }
    const bool is_long = i < n_long;
    const bool first   = i == 0 || i == n_long;
    const bool last    = i == count - 1 || i == n_long - 1;
    const int prev     = first ? -1 : inst[i - 1];
    const int next     = last ? -1 : inst[i + 1];
    if (!first && prev > b) atomicAdd(bad, 1);
    if (first || prev != b) {
      if (is_long)
        r[b].x = i;
      else
        r[b].z = i;
    }
    if (last || next != b) {
      if (is_long)
        r[b].y = i + 1;
      else
        r[b].w = i + 1;
    }
  }
}

__global__ void gather_int_kernel(const int* src, const int* perm, int count, int* dst)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
    dst[i] = src[perm[i]];
}
__global__ void scale_by_inst_kernel(double* v, const int* inst, const double* f, int count)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
    v[i] *= f[inst[i]];
}
// dst[perm[i]] = f[inst[i]] * src[i]
__global__ void scatter_by_inst_kernel(const double* src, const int* perm, const int* inst,
                                       const double* f, int count, double* dst)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
    dst[perm[i]] = (f ? f[inst[i]] : 1.0) * src[i];
}

// Bound / objective rescaling with each instance's beta and gamma.
template <typename TX>
__global__ void b_rescale_vectors_kernel(const double* cs, const double* ls, const double* us,
                                         const double* lcs, const double* ucs, const double* beta,
                                         const double* gamma, const int* cinst, const int* rinst,
                                         int n, int m, TX* c_out, TX* l_out, TX* u_out, TX* lc_out,
                                         TX* uc_out)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += gridDim.x * blockDim.x) {
    if (i < n) {
      const int b = cinst[i];
      c_out[i]    = (TX)(cs[i] * gamma[b]);
      l_out[i]    = (TX)(ls[i] * beta[b]);
      u_out[i]    = (TX)(us[i] * beta[b]);
    } else {
      const int r = i - n, b = rinst[r];
      lc_out[r]   = (TX)(lcs[r] * beta[b]);
      uc_out[r]   = (TX)(ucs[r] * beta[b]);
    }
  }
}

template <typename TX>
__global__ void b_unscale_kernel(const TX* xhat, const TX* yhat, const TX* slack, const double* dc,
                                 const double* dr, const double* beta, const double* gamma,
                                 const int* cinst, const int* rinst, const int* active, int n,
                                 int m, double* xu, double* yu, double* su)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += gridDim.x * blockDim.x) {
    if (i < n) {
      const int b = cinst[i];
      if (!active[b]) continue;
      const double ib = 1.0 / beta[b], ig = 1.0 / gamma[b];
      const double d  = dc[i];
      xu[i]           = ((double)xhat[i] * d) * ib;
      const double s  = (double)slack[i];
      su[i]           = (d != 0.0 ? s / d : s) * ig;
    } else {
      const int r = i - n, b = rinst[r];
      if (!active[b]) continue;
      yu[r] = ((double)yhat[r] * dr[r]) * (1.0 / gamma[b]);
    }
  }
}

template <typename TX>
__global__ void b_halpern_kernel(TX* x, const TX* xbar, const TX* xa, int n, TX* y, const TX* ybar,
                                 const TX* ya, int m, const int* cinst, const int* rinst,
                                 const int* active, const pdlp_scalars* sc)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += gridDim.x * blockDim.x) {
    if (i < n) {
      const int b = cinst[i];
      if (!active[b]) continue;
      const double w = halpern_weight(sc + b, 0);
      x[i]           = (TX)halpern_mix(w, (double)xbar[i], (double)xa[i]);
    } else {
      const int r = i - n, b = rinst[r];
      if (!active[b]) continue;
      const double w = halpern_weight(sc + b, 0);
      y[r]           = (TX)halpern_mix(w, (double)ybar[r], (double)ya[r]);
    }
  }
}

// Restart to the current average: x, x_anchor <- x_hat (and y) for flagged instances.
template <typename TX>
__global__ void b_restart_kernel(TX* x, TX* xa, const TX* xhat, int n, TX* y, TX* ya,
                                 const TX* yhat, int m, const int* cinst, const int* rinst,
                                 const int* flag)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += gridDim.x * blockDim.x) {
    if (i < n) {
      if (!flag[cinst[i]]) continue;
      x[i]  = xhat[i];
      xa[i] = xhat[i];
    } else {
      const int r = i - n;
      if (!flag[rinst[r]]) continue;
      y[r]  = yhat[r];
      ya[r] = yhat[r];
    }
  }
}

// Warm start: a = b = c = v / d (v / d = v where d = 0) times the instance's factor f[inst].
template <typename TX>
__global__ void b_scale_initial_kernel(const double* v, const double* d, const int* inst,
                                       const double* f, int n, TX* a, TX* b, TX* c)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double s = d[i] != 0.0 ? v[i] / d[i] : v[i];
    const TX w     = (TX)(s * f[inst[i]]);
    a[i]           = w;
    b[i]           = w;
    c[i]           = w;
  }
}

__global__ void b_advance_kernel(pdlp_scalars* sc, const int* active, int count, int steps)
{
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < count; b += gridDim.x * blockDim.x)
    if (active[b]) sc[b].t0 += steps;
}

// Golub-Kahan-Lanczos bidiagonalisation per instance (the step size), the single engine's
// run on every instance at once: u and v hold the unnormalised Lanczos vectors, st[b] their
// norms (and the row chunks of the running sum that have been added), and rowbuf the squares of
// the new vector for the per-instance norms.
struct b_gk_state {
  double beta;
  double alpha;
  unsigned arrived;
  unsigned pad;
};

// Row j of A^T applied to u:  p_j = (A^T u)_j / beta - beta v_j / alpha  (written over v_j).
struct b_gk_primal_epi {
  static constexpr int kRed = 0;
  double* v;
  double* rowbuf;
  const b_gk_state* st;
  inst_ctx ctx;
  struct pre_t {
    double v;
    int b;
  };
  __device__ bool skip_range(int r0, int r1) const { return ctx.all_frozen(r0, r1); }
  __device__ __forceinline__ pre_t load(int j) const { return pre_t{v[j], ctx.inst[j]}; }
  __device__ __forceinline__ void operator()(int j, double acc, const pre_t& p, red_t<0>&) const
  {
    if (!ctx.active[p.b]) return;
    const double pj = gk_next_v(acc, p.v, st[p.b].beta, st[p.b].alpha);
    v[j]            = pj;
    rowbuf[j]       = pj * pj;
  }
};

// Row i of A applied to v:  q_i = (A v)_i / alpha - alpha u_i / beta  (written over u_i).
struct b_gk_dual_epi {
  static constexpr int kRed = 0;
  double* u;
  double* rowbuf;
  const b_gk_state* st;
  inst_ctx ctx;
  struct pre_t {
    double u;
    int b;
  };
  __device__ bool skip_range(int r0, int r1) const { return ctx.all_frozen(r0, r1); }
  __device__ __forceinline__ pre_t load(int i) const { return pre_t{u[i], ctx.inst[i]}; }
  __device__ __forceinline__ void operator()(int i, double acc, const pre_t& p, red_t<0>&) const
  {
    if (!ctx.active[p.b]) return;
    const double qi = gk_next_u(acc, p.u, st[p.b].alpha, st[p.b].beta);
    u[i]            = qi;
    rowbuf[i]       = qi * qi;
  }
};

// The norm of each iterating instance's new vector: block c sums its chunk of `v` (the squares in
// the row buffer, or with SQUARE the vector itself), and the block that finishes last of its
// instance adds the instance's chunks in chunk order.  FIELD 0 sets alpha (hist[k * count + b]),
// FIELD 1 sets beta (hist[(k + 1) * count + b]).
template <int FIELD, bool SQUARE = false>
__global__ void __launch_bounds__(kBlock)
  b_gk_norm_kernel(const int4* chunks, const int* chunk_off, int count, const int* active,
                   const double* v, double* part, b_gk_state* st, double* hist, int k)
{
  const int4 ch = chunks[blockIdx.x];
  const int b   = ch.x;
  if (!active[b]) return;
  __shared__ double sm[kBlock];
  ksum acc;
  for (int i = ch.y + threadIdx.x; i < ch.z; i += kBlock) acc.add(SQUARE ? v[i] * v[i] : v[i]);
  const double t = block_sum(acc, sm);
  if (threadIdx.x != 0) return;
  const int c0 = chunk_off[b], c1 = chunk_off[b + 1];
  part[blockIdx.x] = t;
  __threadfence();
  if (atomicAdd(&st[b].arrived, 1u) != (unsigned)(c1 - c0 - 1)) return;
  __threadfence();
  double sum = 0.0;
  for (int c = c0; c < c1; ++c) sum += __ldcg(part + c);
  const double norm = sqrt(sum);
  if (FIELD == 0) {
    st[b].alpha                 = norm;
    hist[(size_t)k * count + b] = norm;
  } else {
    st[b].beta                        = norm;
    hist[(size_t)(k + 1) * count + b] = norm;
  }
  st[b].arrived = 0;
}

// ------------------------------------------------------------------------------------------------
// Host side

struct inst_conv {
  double l2_primal = 0, l2_dual = 0, primal_obj = 0, dual_obj = 0, gap = 0, abs_obj = 0;
};

// Timing decisions of batch solves, remembered for the life of the process as those of single
// solves are: per batch shape (rows, columns, non-zeros, instances), device, iterate precision and
// the parameter that restricts the decision, and for the form of the plain iterations per set of
// active instances (a hash of their indices; 0 when all are active).  A later solve of the same
// batch reuses them instead of timing again.
using batch_key = std::tuple<int, int, int64_t, int, int, int, int, uint64_t>;
struct batch_form_choice {
  int form;
  double us[2];  // graphs, persistent kernel: microseconds per iteration when it was chosen
};
struct batch_shape_choice {
  int wpb_primal, wpb_dual;
  double ms[2][3];
};
std::mutex& batch_tune_mutex()
{
  static std::mutex mu;
  return mu;
}
std::map<batch_key, batch_form_choice>& batch_form_cache()
{
  static std::map<batch_key, batch_form_choice> c;
  return c;
}
std::map<batch_key, batch_shape_choice>& batch_shape_cache()
{
  static std::map<batch_key, batch_shape_choice> c;
  return c;
}
// FNV-1a hash of the indices of the active instances (0 when every instance is active).
uint64_t active_set_hash(const std::vector<int>& act)
{
  if (std::all_of(act.begin(), act.end(), [](int a) { return a != 0; })) return 0;
  uint64_t h = 1469598103934665603ull;
  for (size_t b = 0; b < act.size(); ++b)
    if (act[b]) {
      h ^= (uint64_t)b + 1;
      h *= 1099511628211ull;
    }
  return h == 0 ? 1 : h;
}

template <typename TX>
class batch_engine {
 public:
  batch_engine(const batch_device_input& in, const pdlp_params& p, cudaStream_t s)
    : in_(in), p_(p), s_(s), B_(in.count)
  {
    int dev = 0;
    B200_CUDA_CHECK(cudaGetDevice(&dev));
    B200_CUDA_CHECK(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, dev));
    B200_CUDA_CHECK(cudaMallocHost(&hbuf_, sizeof(double) * 8 * (size_t)std::max(B_, 1)));
    B200_CUDA_CHECK(cudaMallocHost(&hstatus_, sizeof(int)));
    B200_CUDA_CHECK(cudaStreamCreateWithFlags(&es_, cudaStreamNonBlocking));
    B200_CUDA_CHECK(cudaEventCreateWithFlags(&kept_, cudaEventDisableTiming));
    B200_CUDA_CHECK(cudaEventCreateWithFlags(&checked_, cudaEventDisableTiming));
  }
  batch_engine(const batch_engine&)            = delete;
  batch_engine& operator=(const batch_engine&) = delete;
  ~batch_engine()
  {
    // A check may still read buffers that are released, in the order of s_, after this; and no graph
    // is destroyed while it runs.
    if (es_) cudaStreamSynchronize(es_);
    if (!graphs_.empty()) cudaStreamSynchronize(s_);
    if (kept_) cudaEventDestroy(kept_);
    if (checked_) cudaEventDestroy(checked_);
    if (es_) cudaStreamDestroy(es_);
    for (auto& kv : graphs_) cudaGraphExecDestroy(kv.second);
    cudaFreeHost(hbuf_);
    cudaFreeHost(hstatus_);
  }

  std::vector<pdlp_result> run(double* x_out, double* y_out, double* rc_out)
  {
    alloc_scope scope(s_);
    t_start_ = now_s();
    results_.assign(B_, pdlp_result{});
    setup();
    tune_sweep_shape();
    init_plain_form(B_);
    t_loop_ = now_s();
    loop();
    trace("batch: loop");
    write_outputs(x_out, y_out, rc_out);
    const double t = now_s();
    for (int b = 0; b < B_; ++b) {
      results_[b].setup_time      = t_loop_ - t_start_;
      results_[b].loop_time       = results_[b].solve_time - (t_loop_ - t_start_);
      results_[b].kernel_launches = launches_;
      results_[b].power_iterations = power_iters_[b];
      results_[b].plain_form          = first_form_;
      results_[b].persistent_blocks   = first_blocks_;
      results_[b].us_plain_graphs     = first_us_[0];
      results_[b].us_plain_persistent = first_us_[1];
      results_[b].wpb_primal          = wpb_primal_;
      results_[b].wpb_dual            = wpb_dual_;
      std::memcpy(results_[b].wpb_ms, wpb_ms_, sizeof(wpb_ms_));
    }
    (void)t;
    return results_;
  }

 private:
  // ---------------------------------------------------------------- setup
  void setup()
  {
    const int m = in_.m, n = in_.n;
    layout_params lp;
    lp.row_inst = in_.row_inst;
    lp.col_inst = in_.col_inst;
    trace("batch: start");
    build_device_layout(m, n, in_.row_off, in_.col_idx, in_.val, s_, L_, lp);
    B200_CUDA_CHECK(cudaStreamSynchronize(s_));
    trace("batch: layout");
    vgrid_ = sms_ * 4;
    const int g = std::max({sell_grid(bview(L_.A, L_.A.val.data())),
                            sell_grid(bview(L_.AT, L_.AT.val.data())), vgrid_});
    partials_.resize((size_t)g * 4);
    stride_ = (size_t)std::max(m, n);
    rowbuf_.resize(3 * stride_);
    segout_.resize((size_t)B_ * 8);

    // Instance of every internal row / column, and each instance's ranges.
    rinst_.resize(m);
    cinst_.resize(n);
    gather_int_kernel<<<vgrid_, kBlock, 0, s_>>>(in_.row_inst, L_.row_new2old.data(), m,
                                                 rinst_.data());
    gather_int_kernel<<<vgrid_, kBlock, 0, s_>>>(in_.col_inst, L_.col_new2old.data(), n,
                                                 cinst_.data());
    B200_LAUNCH_CHECK();
    rranges_ = ranges_of(rinst_, m, L_.A.n_long);
    cranges_ = ranges_of(cinst_, n, L_.AT.n_long);
    trace("batch: instance ranges");
    rr_d_.resize(B_);
    cr_d_.resize(B_);
    rr_d_.upload(rranges_.data(), B_, s_);
    cr_d_.upload(cranges_.data(), B_, s_);
    build_chunks(rranges_, rows_);
    build_chunks(cranges_, cols_);
    tplanes_.resize(5 * stride_);
    tpart_.resize(2 * (size_t)rows_.count + 3 * (size_t)cols_.count + 1);
    tarrived_.resize(2 * (size_t)B_);
    tarrived_.zero(s_);

    // Per-instance sign (maximisation) and objective scale / offset.
    std::vector<double> sgn(B_);
    obj_scale_.resize(B_);
    obj_offset_.resize(B_);
    for (int b = 0; b < B_; ++b) {
      const bool mx  = in_.maximize[b] != 0;
      sgn[b]         = mx ? -1.0 : 1.0;
      obj_scale_[b]  = mx ? -1.0 : 1.0;
      obj_offset_[b] = mx ? -in_.obj_offset[b] : in_.obj_offset[b];
    }
    sgn_d_.resize(B_);
    sgn_d_.upload(sgn.data(), B_, s_);

    c64_.resize(n);
    l64_.resize(n);
    u64_.resize(n);
    lc64_.resize(m);
    uc64_.resize(m);
    permute_gather(in_.c, L_.col_new2old.data(), n, 1.0, c64_.data(), s_);
    scale_by_inst_kernel<<<vgrid_, kBlock, 0, s_>>>(c64_.data(), cinst_.data(), sgn_d_.data(), n);
    permute_gather(in_.var_lo, L_.col_new2old.data(), n, 1.0, l64_.data(), s_);
    permute_gather(in_.var_up, L_.col_new2old.data(), n, 1.0, u64_.data(), s_);
    permute_gather(in_.con_lo, L_.row_new2old.data(), m, 1.0, lc64_.data(), s_);
    permute_gather(in_.con_up, L_.row_new2old.data(), m, 1.0, uc64_.data(), s_);

    // Ruiz (10 passes) then Pock-Chambolle (alpha = 1); row / column operations, so the batch
    // scales every instance exactly as a single solve would (reference initial_scaling.cu:152-365).
    const auto A64 = bview(L_.A, L_.A.val.data()), AT64 = bview(L_.AT, L_.AT.val.data());
    dr_.resize(m);
    dc_.resize(n);
    fill(dr_.data(), m, 1.0);
    fill(dc_.data(), n, 1.0);
    dbuf<double> rtmp(m), ctmp(n);
    launches_ += scale_passes(A64, AT64, kRuizIterations, kPcAlpha, dr_, dc_, rtmp, ctmp, s_);
    As_.resize(L_.A.stored());
    ATs_.resize(L_.AT.stored());
    scale_values_kernel<TX, false><<<sell_grid(A64), kBlock, 0, s_>>>(A64, dr_.data(), dc_.data(),
                                                                     As_.data());
    scale_values_kernel<TX, true><<<sell_grid(AT64), kBlock, 0, s_>>>(AT64, dr_.data(),
                                                                     dc_.data(), ATs_.data());
    B200_LAUNCH_CHECK();

    // All instances active from here on (the power iteration has its own flags).
    active_h_.assign(B_, 1);
    active_d_.resize(B_);
    active_d_.upload(active_h_.data(), B_, s_);
    B200_CUDA_CHECK(cudaStreamSynchronize(s_));
    trace("batch: ranges + scaling");
    prepare_vectors();
    trace("batch: vectors");
    // Step size from the largest singular value of each scaled instance: the power iteration
    // (reference pdlp.cu:2620-2731), or Golub-Kahan-Lanczos in mixed precision, as single solves.
    if ((int)in_.initial_step.size() == B_) {
      eta_ = in_.initial_step;
      power_iters_.assign(B_, 0);
    } else if (p_.precision == 1)
      lanczos_step_size();
    else
      power_iteration();
    trace("batch: step size");

    xu_.resize(n);
    su_.resize(n);
    yu_.resize(m);
    xu_.zero(s_);
    su_.zero(s_);
    yu_.zero(s_);
    sc_d_.resize(B_);
    if ((int)in_.initial_weight.size() == B_)
      omega_ = in_.initial_weight;
    else
      omega_.assign(B_, 1.0);
    best_omega_ = omega_;
    restarts_.assign(B_, 0);
    for (auto* b : {&x_, &xhat_, &slack_, &xbar_, &xa_, &aty_}) {
      b->resize(n);
      b->zero(s_);
    }
    for (auto* b : {&y_, &yhat_, &ybar_, &ya_}) {
      b->resize(m);
      b->zero(s_);
    }
    // Warm start: iterate, anchor and x_hat from the initial solution in the scaled space (the
    // single engine's load_initial_solution, per instance).
    if (in_.initial_primal) {
      dbuf<double> v(n);
      permute_gather(in_.initial_primal, L_.col_new2old.data(), n, 1.0, v.data(), s_);
      b_scale_initial_kernel<TX><<<vgrid_, kBlock, 0, s_>>>(v.data(), dc_.data(), cinst_.data(),
                                                            beta_d_.data(), n, x_.data(),
                                                            xhat_.data(), xa_.data());
      B200_CUDA_CHECK(cudaStreamSynchronize(s_));
    }
    if (in_.initial_dual) {
      dbuf<double> v(m);
      permute_gather(in_.initial_dual, L_.row_new2old.data(), m, 1.0, v.data(), s_);
      b_scale_initial_kernel<TX><<<vgrid_, kBlock, 0, s_>>>(v.data(), dr_.data(), rinst_.data(),
                                                            gamma_d_.data(), m, y_.data(),
                                                            yhat_.data(), ya_.data());
      B200_CUDA_CHECK(cudaStreamSynchronize(s_));
    }
    clamp_kernel<TX><<<vgrid_, kBlock, 0, s_>>>(x_.data(), ls_.data(), us_.data(), n);
    launches_ += 1;
    B200_LAUNCH_CHECK();
    B200_CUDA_CHECK(cudaStreamSynchronize(s_));
  }

  // Ranges {long_lo, long_hi, short_lo, short_hi} of every instance in an internal order whose
  // instance ids are sorted inside [0, n_long) and inside [n_long, count).
  std::vector<int4> ranges_of(const dbuf<int>& inst, int count, int n_long)
  {
    dbuf<int4> r(B_);
    dbuf<int> bad(1);
    r.zero(s_);
    bad.zero(s_);
    if (count > 0)
      instance_ranges_kernel<<<vgrid_, kBlock, 0, s_>>>(inst.data(), count, n_long, B_, r.data(),
                                                        bad.data());
    B200_LAUNCH_CHECK();
    std::vector<int4> h(B_);
    int hbad = 0;
    r.download(h.data(), B_, s_);
    bad.download(&hbad, 1, s_);
    B200_CUDA_CHECK(cudaStreamSynchronize(s_));
    if (hbad) throw std::runtime_error("batch layout: instance ids out of range or not contiguous");
    return h;
  }

  void fill(double* p, int n, double v)
  {
    fill_kernel<<<vgrid_, kBlock, 0, s_>>>(p, n, v);
    ++launches_;
    B200_LAUNCH_CHECK();
  }

  // Per-instance sums of K planes of the row buffer over rows (ROWS) or columns; result in
  // segout_ + offset, optionally only for active instances.
  // Row chunks of every instance (rows of A, or of A^T for the columns), see kChunkRows.
  struct chunk_table {
    dbuf<int4> chunks;
    dbuf<int> offsets;
    int count = 0;
  };
  void build_chunks(const std::vector<int4>& ranges, chunk_table& t)
  {
    std::vector<int4> chunks;
    std::vector<int> off(B_ + 1, 0);
    for (int b = 0; b < B_; ++b) {
      off[b]       = (int)chunks.size();
      const int4 r = ranges[b];
      for (int lo = r.x; lo < r.y; lo += kChunkRows)
        chunks.push_back(int4{b, lo, std::min(lo + kChunkRows, r.y), 0});
      for (int lo = r.z; lo < r.w; lo += kChunkRows)
        chunks.push_back(int4{b, lo, std::min(lo + kChunkRows, r.w), 0});
    }
    off[B_] = (int)chunks.size();
    t.count = (int)chunks.size();
    t.chunks.resize(std::max(t.count, 1));
    t.offsets.resize(B_ + 1);
    if (t.count > 0) t.chunks.upload(chunks.data(), t.count, s_);
    t.offsets.upload(off.data(), B_ + 1, s_);
    B200_CUDA_CHECK(cudaStreamSynchronize(s_));
  }

  // Per-instance sums of K planes of the row buffer over rows (ROWS) or columns; result in
  // segout_ + offset, optionally only for active instances.
  template <int K>
  void seg_reduce(bool rows, size_t offset, bool only_active)
  {
    const chunk_table& t = rows ? rows_ : cols_;
    const int* want      = only_active ? active_d_.data() : nullptr;
    if (chunk_part_.size() < (size_t)std::max(rows_.count, cols_.count) * 3)
      chunk_part_.resize((size_t)std::max({rows_.count, cols_.count, 1}) * 3);
    if (t.count > 0)
      chunk_reduce_kernel<K><<<t.count, kBlock, 0, s_>>>(rowbuf_.data(), stride_, t.chunks.data(),
                                                         want, chunk_part_.data());
    instance_reduce_kernel<K><<<ceil_div(B_, kBlock), kBlock, 0, s_>>>(
      chunk_part_.data(), t.offsets.data(), B_, want, segout_.data() + offset);
    launches_ += 2;
  }
  void fetch(size_t offset, size_t count, double* dst)
  {
    B200_CUDA_CHECK(cudaMemcpyAsync(dst, segout_.data() + offset, count * sizeof(double),
                                    cudaMemcpyDeviceToHost, s_));
    if (persist_used_)
      B200_CUDA_CHECK(cudaMemcpyAsync(hstatus_, &pctl_.data()->status, sizeof(int),
                                      cudaMemcpyDeviceToHost, s_));
    B200_CUDA_CHECK(cudaStreamSynchronize(s_));
    if (persist_used_) {
      persist_used_ = false;
      check_status();
    }
    collect_form_timing();
  }
  void check_status() const
  {
    if (*hstatus_ != 0)
      throw cuda_error(*hstatus_ == kBarrierTimedOut
                         ? "persistent batch iterations: a grid barrier passed its deadline"
                         : "persistent batch iterations: a grid barrier passed its poll limit");
  }

  void prepare_vectors()
  {
    const int m = in_.m, n = in_.n;
    std::vector<double> h(4 * (size_t)B_);
    sq_diff_kernel<double><<<vgrid_, kBlock, 0, s_>>>(c64_.data(), nullptr, n, rowbuf_.data());
    seg_reduce<1>(false, 0, false);
    bound_terms_kernel<<<vgrid_, kBlock, 0, s_>>>(lc64_.data(), uc64_.data(), m, rowbuf_.data());
    seg_reduce<1>(true, B_, false);
    dbuf<double> cs(n), ls(n), us(n), lcs(m), ucs(m);
    scale_vectors_kernel<<<vgrid_, kBlock, 0, s_>>>(c64_.data(), l64_.data(), u64_.data(),
                                                    lc64_.data(), uc64_.data(), dc_.data(),
                                                    dr_.data(), n, m, cs.data(), ls.data(),
                                                    us.data(), lcs.data(), ucs.data());
    sq_diff_kernel<double><<<vgrid_, kBlock, 0, s_>>>(cs.data(), nullptr, n, rowbuf_.data());
    seg_reduce<1>(false, 2 * (size_t)B_, false);
    bound_terms_kernel<<<vgrid_, kBlock, 0, s_>>>(lcs.data(), ucs.data(), m, rowbuf_.data());
    seg_reduce<1>(true, 3 * (size_t)B_, false);
    launches_ += 5;
    B200_LAUNCH_CHECK();
    fetch(0, 4 * (size_t)B_, h.data());
    c_norm_.resize(B_);
    b_norm_.resize(B_);
    std::vector<double> beta(B_), gamma(B_);
    for (int b = 0; b < B_; ++b) {
      c_norm_[b] = std::sqrt(h[b]);
      b_norm_[b] = std::sqrt(h[B_ + b]);
      gamma[b]   = 1.0 / (std::sqrt(h[2 * B_ + b]) + 1.0);
      beta[b]    = 1.0 / (std::sqrt(h[3 * B_ + b]) + 1.0);
    }
    beta_d_.resize(B_);
    gamma_d_.resize(B_);
    beta_d_.upload(beta.data(), B_, s_);
    gamma_d_.upload(gamma.data(), B_, s_);
    beta_  = beta;
    gamma_ = gamma;
    cs_.resize(n);
    ls_.resize(n);
    us_.resize(n);
    lcs_.resize(m);
    ucs_.resize(m);
    b_rescale_vectors_kernel<TX><<<vgrid_, kBlock, 0, s_>>>(
      cs.data(), ls.data(), us.data(), lcs.data(), ucs.data(), beta_d_.data(), gamma_d_.data(),
      cinst_.data(), rinst_.data(), n, m, cs_.data(), ls_.data(), us_.data(), lcs_.data(),
      ucs_.data());
    ++launches_;
    B200_LAUNCH_CHECK();
    B200_CUDA_CHECK(cudaStreamSynchronize(s_));
  }

  // The reference's power iteration of every instance (pdlp.cu:2620-2731) in the Krylov space of
  // its start vector, as in single solves.  On 64 LPs of 200 to 20 000 rows, whose iterations take
  // up to 2 800 products with A A^T, the step sizes took 164 of 264 ms with the iteration itself.
  void power_iteration()
  {
    std::vector<krylov_power_iteration> power(B_);
    bidiagonalise(kKrylovMaxSteps, [&](int b, int k, const double* a, const double* bb) {
      const bool done = power[b].advance(a, bb, k);
      power_iters_[b] = power[b].iterations();
      return done;
    });
    for (int b = 0; b < B_; ++b) eta_[b] = kStepScaling / std::sqrt(power[b].sigma2());
  }

  // The largest singular value of every instance (the single engine's lanczos_step_size): an
  // instance stops when its estimate moved by at most kLanczosTol (relative) over a chunk of
  // steps, or its recurrence broke down.
  void lanczos_step_size()
  {
    std::vector<double> prev(B_, -1.0), sigma2(B_, 0.0);
    bidiagonalise(kLanczosMaxSteps, [&](int b, int k, const double* a, const double* bb) {
      bool breakdown = false;
      int used       = k;
      for (int j = 0; j < k; ++j)
        if (!(a[j] > 0.0) || !(bb[j] > 0.0) || !std::isfinite(a[j]) || !std::isfinite(bb[j])) {
          used      = j + 1;
          breakdown = true;
          break;
        }
      sigma2[b]       = largest_bidiagonal_sigma2(a, bb, used);
      power_iters_[b] = used;
      const bool done = breakdown || (prev[b] > 0.0 && std::fabs(sigma2[b] - prev[b]) <=
                                                         kLanczosTol * sigma2[b]);
      prev[b] = sigma2[b];
      return done;
    });
    for (int b = 0; b < B_; ++b) eta_[b] = kStepScaling / std::sqrt(sigma2[b]);
  }

  // Golub-Kahan bidiagonalisation of every instance, in chunks of kLanczosChunk steps: after each,
  // test(instance, steps, diagonal, subdiagonal) tells which instances are done, and the sweeps
  // shrink to the others once these are at most half of those listed.
  template <class Test>
  void bidiagonalise(int max_steps, Test&& test)
  {
    const int m = in_.m, n = in_.n;
    // Every instance starts from the first m_b values of the std::mt19937(1) normal sequence.
    std::vector<double> z0(m);
    int max_rows = 0;
    for (int b = 0; b < B_; ++b) max_rows = std::max(max_rows, in_.row_start[b + 1] - in_.row_start[b]);
    const auto seq = power_start_sequence(max_rows);
    for (int b = 0; b < B_; ++b)
      std::copy(seq->begin(), seq->begin() + (in_.row_start[b + 1] - in_.row_start[b]),
                z0.begin() + in_.row_start[b]);
    dbuf<double> u(m), v(n), tmp(m);
    // The coefficients of one chunk, a row of B_ a step; row 0 of betas is the norm of the start.
    dbuf<double> alphas((size_t)B_ * kLanczosChunk), betas((size_t)B_ * (kLanczosChunk + 1));
    dbuf<b_gk_state> st(B_);
    tmp.upload(z0.data(), m, s_);
    permute_gather(tmp.data(), L_.row_new2old.data(), m, 1.0, u.data(), s_);
    v.zero(s_);
    st.zero(s_);
    dbuf<int> pact(B_);
    std::vector<int> pact_h(B_, 1);
    pact.upload(pact_h.data(), B_, s_);
    const inst_ctx rctx{rinst_.data(), pact.data(), nullptr};
    const inst_ctx cctx{cinst_.data(), pact.data(), nullptr};
    dbuf<double> part(std::max({rows_.count, cols_.count, 1}));
    // beta_0 = |z0| per instance
    b_gk_norm_kernel<1, true><<<rows_.count, kBlock, 0, s_>>>(
      rows_.chunks.data(), rows_.offsets.data(), B_, pact.data(), u.data(), part.data(), st.data(),
      betas.data(), -1);
    ++launches_;
    B200_LAUNCH_CHECK();
    auto step = [&](int k) {
      const auto As  = wview<TX>(true, As_.data());
      const auto ATs = wview<TX>(false, ATs_.data());
      sell_map_kernel<TX, double, b_gk_primal_epi><<<sell_grid(ATs), kBlock, 0, s_>>>(
        ATs, u.data(), b_gk_primal_epi{v.data(), rowbuf_.data(), st.data(), cctx},
        partials_.data());
      b_gk_norm_kernel<0><<<cols_.count, kBlock, 0, s_>>>(
        cols_.chunks.data(), cols_.offsets.data(), B_, pact.data(), rowbuf_.data(), part.data(),
        st.data(), alphas.data(), k);
      sell_map_kernel<TX, double, b_gk_dual_epi><<<sell_grid(As), kBlock, 0, s_>>>(
        As, v.data(), b_gk_dual_epi{u.data(), rowbuf_.data(), st.data(), rctx},
        partials_.data());
      b_gk_norm_kernel<1><<<rows_.count, kBlock, 0, s_>>>(
        rows_.chunks.data(), rows_.offsets.data(), B_, pact.data(), rowbuf_.data(), part.data(),
        st.data(), betas.data(), k);
    };
    // On the host, each instance's own from its first step to its last.
    std::vector<double> ha((size_t)B_ * kLanczosChunk), hb((size_t)B_ * kLanczosChunk);
    std::vector<std::vector<double>> diag(B_), sub(B_);
    std::vector<char> done(B_, 0);
    eta_.assign(B_, 0.0);
    power_iters_.assign(B_, 0);
    int left = B_, listed = B_, k = 0;
    while (left > 0 && k < max_steps) {
      const int c = std::min(kLanczosChunk, max_steps - k);
      for (int i = 0; i < c; ++i) step(i);
      launches_ += 4.0 * c;
      B200_LAUNCH_CHECK();
      alphas.download(ha.data(), (size_t)c * B_, s_);
      B200_CUDA_CHECK(cudaMemcpyAsync(hb.data(), betas.data() + B_, (size_t)c * B_ * sizeof(double),
                                      cudaMemcpyDeviceToHost, s_));
      B200_CUDA_CHECK(cudaStreamSynchronize(s_));
      k += c;
      // Each instance's test (the host's share of the step) is independent of the others:
      // instances are split over host threads, each writing only its own entries, so the results
      // do not depend on the split.
      parallel_ranges(B_, [&](int b0, int b1) {
        for (int b = b0; b < b1; ++b) {
          if (!pact_h[b]) continue;
          for (int j = 0; j < c; ++j) {
            diag[b].push_back(ha[(size_t)j * B_ + b]);
            sub[b].push_back(hb[(size_t)j * B_ + b]);
          }
          done[b] = test(b, k, diag[b].data(), sub[b].data());
          if (done[b]) {
            diag[b] = {};
            sub[b]  = {};
          }
        }
      });
      for (int b = 0; b < B_; ++b)
        if (pact_h[b] && done[b]) {
          pact_h[b] = 0;
          --left;
        }
      if (left == 0) break;
      pact.upload(pact_h.data(), B_, s_);
      if (2 * left <= listed) {
        rebuild_work(pact_h);
        listed = left;
        char what[96];
        std::snprintf(what, sizeof what, "batch: bidiagonal to %d steps, %d instances left", k,
                      left);
        trace(what);
      }
    }
    clear_work();
  }

  // ---------------------------------------------------------------- work lists
  // Sweeps over A (rows = constraints) and A^T (rows = variables), restricted to the listed long
  // rows and slices once some instances have finished.
  template <typename T>
  dev_sell<T> wview(bool of_A, const T* vals) const
  {
    dev_sell<T> v = bview<T>(of_A ? L_.A : L_.AT, vals);
    if (lists_on_) {
      const work_list& w = of_A ? wa_ : wt_;
      v.long_list        = w.longs.data();
      v.slice_list       = w.slices.data();
      v.work_long        = w.n_long;
      v.work_slices      = w.n_slices;
    }
    return v;
  }

  struct work_list {
    dbuf<int> longs, slices;
    int n_long = 0, n_slices = 0;
  };

  void build_list(const std::vector<int4>& ranges, int n_long_rows, const std::vector<int>& act,
                  work_list& w)
  {
    std::vector<int> longs, slices;
    for (int b = 0; b < B_; ++b) {
      if (!act[b]) continue;
      const int4 r = ranges[b];
      for (int i = r.x; i < r.y; ++i) longs.push_back(i);
      if (r.z < r.w) {
        const int first = (r.z - n_long_rows) / kWarp, last = (r.w - 1 - n_long_rows) / kWarp;
        for (int q = first; q <= last; ++q)
          if (slices.empty() || slices.back() < q) slices.push_back(q);
      }
    }
    w.n_long   = (int)longs.size();
    w.n_slices = (int)slices.size();
    w.longs.resize(std::max<size_t>(longs.size(), 1));
    w.slices.resize(std::max<size_t>(slices.size(), 1));
    if (!longs.empty()) w.longs.upload(longs.data(), longs.size(), s_);
    if (!slices.empty()) w.slices.upload(slices.data(), slices.size(), s_);
  }

  // Restricts the sweeps to the instances flagged in `act`; cached graphs are dropped because
  // they hold the previous lists.
  void rebuild_work(const std::vector<int>& act)
  {
    build_list(rranges_, L_.A.n_long, act, wa_);
    build_list(cranges_, L_.AT.n_long, act, wt_);
    B200_CUDA_CHECK(cudaStreamSynchronize(s_));
    lists_on_ = true;
    drop_graphs();
    init_plain_form((int)std::count(act.begin(), act.end(), 1), active_set_hash(act));
  }
  void clear_work()
  {
    lists_on_ = false;
    drop_graphs();
    init_plain_form(B_);
  }
  void drop_graphs()
  {
    for (auto& kv : graphs_) cudaGraphExecDestroy(kv.second);
    graphs_.clear();
  }

  // ---------------------------------------------------------------- iterations
  inst_ctx ctx_rows() const { return inst_ctx{rinst_.data(), active_d_.data(), sc_d_.data()}; }
  inst_ctx ctx_cols() const { return inst_ctx{cinst_.data(), active_d_.data(), sc_d_.data()}; }

  // The plain sweeps run with the tuned number of warps per block (tune_sweep_shape).
  template <bool MAJOR, bool HALPERN, bool SAVE_ATY>
  void launch_primal(int it_off, int wpb = 0)
  {
    const auto A = wview<TX>(false, ATs_.data());
    b_primal_epi<TX, MAJOR, HALPERN, SAVE_ATY> e{x_.data(),    cs_.data(),   ls_.data(),
                                                 us_.data(),   xa_.data(),   xbar_.data(),
                                                 x_.data(),    xhat_.data(), slack_.data(),
                                                 aty_.data(),  ctx_cols(),   it_off};
    if constexpr (!MAJOR && HALPERN && !SAVE_ATY)
      launch_sell_wpb(wpb ? wpb : wpb_primal_, A, y_.data(), e, partials_.data(), s_);
    else
      sell_map_kernel<TX, TX, decltype(e)><<<sell_grid(A), kBlock, 0, s_>>>(A, y_.data(), e,
                                                                           partials_.data());
    ++launches_;
  }
  template <bool MAJOR, bool HALPERN, bool FPE>
  void launch_dual(int it_off, int wpb = 0)
  {
    const auto A = wview<TX>(true, As_.data());
    b_dual_epi<TX, MAJOR, HALPERN, FPE> e{y_.data(),     lcs_.data(),  ucs_.data(),
                                          ya_.data(),    ybar_.data(), y_.data(),
                                          yhat_.data(),  rowbuf_.data(), ctx_rows(), it_off};
    if constexpr (!MAJOR && HALPERN && !FPE)
      launch_sell_wpb(wpb ? wpb : wpb_dual_, A, xbar_.data(), e, partials_.data(), s_);
    else
      sell_map_kernel<TX, TX, decltype(e)><<<sell_grid(A), kBlock, 0, s_>>>(A, xbar_.data(), e,
                                                                           partials_.data());
    ++launches_;
  }

  // Block shape of the plain sweeps over all instances (pdlp_sweep_warps_per_block = 0): 4, 8 and
  // 16 warps per block, a warm-up launch and about 1 ms of launches each; another shape replaces 8
  // warps when it is at least 3 % faster.  The iterates the timed sweeps move are restored (x, y) or
  // cleared (x_bar, y_bar) afterwards.
  void tune_sweep_shape()
  {
    wpb_primal_ = wpb_dual_ = p_.sweep_wpb ? p_.sweep_wpb : kWarpsPerBlock;
    if (p_.sweep_wpb) return;
    const batch_key key = tune_key(0, 0);
    {
      std::lock_guard<std::mutex> lock(batch_tune_mutex());
      auto it = batch_shape_cache().find(key);
      if (it != batch_shape_cache().end()) {
        wpb_primal_ = it->second.wpb_primal;
        wpb_dual_   = it->second.wpb_dual;
        std::memcpy(wpb_ms_, it->second.ms, sizeof(wpb_ms_));
        return;
      }
    }
    const int m = in_.m, n = in_.n;
    upload_scalars(std::vector<long>(B_, 0));
    dbuf<TX> x0(n), y0(m);
    B200_CUDA_CHECK(cudaMemcpyAsync(x0.data(), x_.data(), n * sizeof(TX),
                                    cudaMemcpyDeviceToDevice, s_));
    B200_CUDA_CHECK(cudaMemcpyAsync(y0.data(), y_.data(), m * sizeof(TX),
                                    cudaMemcpyDeviceToDevice, s_));
    cudaEvent_t e0, e1;
    B200_CUDA_CHECK(cudaEventCreate(&e0));
    B200_CUDA_CHECK(cudaEventCreate(&e1));
    // One warm-up launch, then enough launches for about a millisecond of timed work (at least 3).
    auto time_of = [&](auto&& launch) {
      B200_CUDA_CHECK(cudaEventRecord(e0, s_));
      launch();
      B200_CUDA_CHECK(cudaEventRecord(e1, s_));
      B200_CUDA_CHECK(cudaEventSynchronize(e1));
      float ms = 0.f;
      B200_CUDA_CHECK(cudaEventElapsedTime(&ms, e0, e1));
      const int reps = std::max(3, std::min(200, (int)std::ceil(1.0 / std::max(ms, 1e-3f))));
      B200_CUDA_CHECK(cudaEventRecord(e0, s_));
      for (int i = 0; i < reps; ++i) launch();
      B200_CUDA_CHECK(cudaEventRecord(e1, s_));
      B200_CUDA_CHECK(cudaEventSynchronize(e1));
      B200_CUDA_CHECK(cudaEventElapsedTime(&ms, e0, e1));
      return (double)ms / reps;
    };
    static constexpr int kShapes[3] = {4, 8, 16};
    for (int q = 0; q < 3; ++q) {
      wpb_ms_[0][q] = time_of([&] { launch_primal<false, true, false>(0, kShapes[q]); });
      wpb_ms_[1][q] = time_of([&] { launch_dual<false, true, false>(0, kShapes[q]); });
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    // Another shape replaces the default 8 warps only when it is at least 3 % faster.
    auto best = [&](const double* t) {
      int b = 1;
      for (int q = 0; q < 3; ++q)
        if (t[q] > 0 && t[q] < 0.97 * t[1] && t[q] < t[b]) b = q;
      return kShapes[b];
    };
    wpb_primal_ = best(wpb_ms_[0]);
    wpb_dual_   = best(wpb_ms_[1]);
    {
      std::lock_guard<std::mutex> lock(batch_tune_mutex());
      batch_shape_choice c{wpb_primal_, wpb_dual_, {}};
      std::memcpy(c.ms, wpb_ms_, sizeof(wpb_ms_));
      batch_shape_cache()[key] = c;
    }
    B200_CUDA_CHECK(cudaMemcpyAsync(x_.data(), x0.data(), n * sizeof(TX),
                                    cudaMemcpyDeviceToDevice, s_));
    B200_CUDA_CHECK(cudaMemcpyAsync(y_.data(), y0.data(), m * sizeof(TX),
                                    cudaMemcpyDeviceToDevice, s_));
    xbar_.zero(s_);
    ybar_.zero(s_);
    B200_CUDA_CHECK(cudaStreamSynchronize(s_));
    if (std::getenv("CUOPT_B200_TRACE"))
      std::fprintf(stderr,
                   "[cuopt_b200] batch sweep block shape: primal %.4f/%.4f/%.4f ms -> %d warps; "
                   "dual %.4f/%.4f/%.4f ms -> %d warps (4/8/16 warps per block)\n",
                   wpb_ms_[0][0], wpb_ms_[0][1], wpb_ms_[0][2], wpb_primal_, wpb_ms_[1][0],
                   wpb_ms_[1][1], wpb_ms_[1][2], wpb_dual_);
  }
  void advance(int steps)
  {
    b_advance_kernel<<<ceil_div(B_, kBlock), kBlock, 0, s_>>>(sc_d_.data(), active_d_.data(), B_,
                                                             steps);
    ++launches_;
  }
  void plain_iterations(int L)
  {
    for (int i = 0; i < L; ++i) {
      launch_primal<false, true, false>(i);
      launch_dual<false, true, false>(i);
    }
    advance(L);
  }
  // ---------------------------------------------------------------- persistent plain iterations
  // The same choice as for single solves (plain_form.hpp), made again for every work list: the
  // sweeps shrink as instances finish, and the cost of kernel boundaries grows relative to them.
  using persist_pe = b_primal_epi<TX, false, true, false>;
  using persist_de = b_dual_epi<TX, false, true, false>;
  static const void* persistent_fn()
  {
    return (const void*)persistent_plain_kernel<TX, persist_pe, persist_de, advance_active>;
  }
  batch_key tune_key(int param, uint64_t set_hash) const
  {
    int dev = 0;
    B200_CUDA_CHECK(cudaGetDevice(&dev));
    return batch_key{in_.m, in_.n, L_.nnz, B_, dev, (int)sizeof(TX), param, set_hash};
  }
  void init_plain_form(int n_active, uint64_t set_hash = 0)
  {
    int dev = 0, coop = 0, per_sm = 0;
    B200_CUDA_CHECK(cudaGetDevice(&dev));
    B200_CUDA_CHECK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    B200_CUDA_CHECK(
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, persistent_fn(), kBlock, 0));
    const int need = std::max(sell_grid(wview<TX>(false, ATs_.data())),
                              sell_grid(wview<TX>(true, As_.data())));
    persist_grid_  = std::min(need, per_sm * sms_);
    if (pctl_.size() == 0) {
      pctl_.resize(1);
      pctl_.zero(s_);
    }
    form_active_ = n_active;
    if (cycle_open_) form_.end(s_, cycle_form_, 0, true);  // a cycle cut short is not counted
    cycle_open_ = false;
    ++form_epochs_;
    const bool avail[plain_form_tuner::kForms] = {true, coop && persist_grid_ > 0, false};
    form_key_   = tune_key(p_.persistent, set_hash);
    int known   = -1;
    known_us_[0] = known_us_[1] = 0.0;
    if (p_.persistent < 0) {
      std::lock_guard<std::mutex> lock(batch_tune_mutex());
      auto it = batch_form_cache().find(form_key_);
      if (it != batch_form_cache().end()) {
        known        = it->second.form;
        known_us_[0] = it->second.us[0];
        known_us_[1] = it->second.us[1];
      }
    }
    form_.reset(p_.persistent, known, avail);
    if (n_active == B_ && form_.decided()) {  // forced, remembered, or the only form available
      first_form_   = form_.chosen();
      first_blocks_ = persist_grid_;
      first_us_[0]  = known_us_[0];
      first_us_[1]  = known_us_[1];
    }
  }
  void trace_form()
  {
    if (form_active_ == B_ && first_form_ < 0) {
      first_form_    = form_.chosen();
      first_us_[0]   = form_.us_per_iteration(0);
      first_us_[1]   = form_.us_per_iteration(1);
      first_blocks_  = persist_grid_;
    }
    if (std::getenv("CUOPT_B200_TRACE"))
      std::fprintf(stderr,
                   "[cuopt_b200] batch plain iterations (%d instances): graphs %.2f us, "
                   "persistent (%d blocks) %.2f us per iteration -> %s\n",
                   form_active_, form_.us_per_iteration(0), persist_grid_,
                   form_.us_per_iteration(1), form_.chosen() ? "persistent" : "graphs");
  }
  void collect_form_timing()
  {
    const bool before = form_.decided();
    form_.collect();
    if (!before && form_.decided()) {
      trace_form();
      std::lock_guard<std::mutex> lock(batch_tune_mutex());
      batch_form_cache()[form_key_] =
        batch_form_choice{form_.chosen(), {form_.us_per_iteration(0), form_.us_per_iteration(1)}};
    }
  }
  // Returns true for the first launch of the engine (which may include loading the kernel).
  bool launch_persistent(int L)
  {
    const auto AT = wview<TX>(false, ATs_.data()), A = wview<TX>(true, As_.data());
    persist_pe pe{x_.data(),   cs_.data(),   ls_.data(),    us_.data(),  xa_.data(),
                  xbar_.data(), x_.data(),   xhat_.data(),  slack_.data(), aty_.data(),
                  ctx_cols(),  0};
    persist_de de{y_.data(),    lcs_.data(),  ucs_.data(),    ya_.data(), ybar_.data(),
                  y_.data(),    yhat_.data(), rowbuf_.data(), ctx_rows(), 0};
    advance_active adv{sc_d_.data(), active_d_.data(), B_};
    int gp = sell_grid(AT), gd = sell_grid(A);
    const TX* y    = y_.data();
    const TX* xb   = xbar_.data();
    persist_ctl* c = pctl_.data();
    unsigned long long budget = kPersistBudgetNs;
    B200_CUDA_CHECK(cudaMemsetAsync(&c->arrivals, 0, sizeof(unsigned), s_));
    void* args[] = {(void*)&AT, (void*)&A, (void*)&y, (void*)&xb, (void*)&pe, (void*)&de,
                    (void*)&adv, (void*)&L, (void*)&gp, (void*)&gd, (void*)&c, (void*)&budget};
    B200_CUDA_CHECK(cudaLaunchCooperativeKernel(persistent_fn(), dim3(persist_grid_),
                                                dim3(kBlock), args, 0, s_));
    ++launches_;
    persist_used_ = true;
    return persist_launches_++ == 0;
  }

  // A timing cycle runs from the first plain run after a termination check to the next check:
  // all its plain runs use one form, and its events bracket everything the GPU does in between
  // (major steps, fixed-point errors and every launch boundary), so the forms are compared on
  // what they cost the loop.
  void run_plain(long R, long k)
  {
    if (!cycle_open_) {
      cycle_form_     = form_.next();
      cycle_k0_       = k;
      cycle_one_time_ = false;
      cycle_open_     = true;
      form_.begin(s_);
    }
    cycle_one_time_ |= cycle_form_ == 1 ? launch_persistent((int)R) : run_graphs(R);
  }
  void close_cycle(long k)
  {
    if (!cycle_open_) return;
    cycle_open_ = false;
    form_.end(s_, cycle_form_, k - cycle_k0_, cycle_one_time_);
  }

  // Returns true when a graph had to be captured and instantiated first.
  bool run_graphs(long R)
  {
    bool built = false;
    for (int L = 128; L >= 1; L >>= 1) {
      while (R >= L) {
        auto it = graphs_.find(L);
        if (it == graphs_.end()) {
          cudaGraph_t g;
          cudaGraphExec_t e;
          B200_CUDA_CHECK(cudaStreamBeginCapture(s_, cudaStreamCaptureModeThreadLocal));
          const double before = launches_;
          plain_iterations(L);
          launches_ = before;
          B200_CUDA_CHECK(cudaStreamEndCapture(s_, &g));
          B200_CUDA_CHECK(cudaGraphInstantiate(&e, g, 0));
          cudaGraphDestroy(g);
          it = graphs_.emplace(L, e).first;
          built = true;
        }
        B200_CUDA_CHECK(cudaGraphLaunch(it->second, s_));
        launches_ += 2.0 * L + 1.0;
        R -= L;
      }
    }
    return built;
  }

  void upload_scalars(const std::vector<long>& since)
  {
    std::vector<pdlp_scalars> h(B_);
    for (int b = 0; b < B_; ++b)
      h[b] = pdlp_scalars{eta_[b] / omega_[b], eta_[b] * omega_[b], eta_[b], omega_[b],
                          (long long)since[b]};
    sc_d_.upload(h.data(), B_, s_);
    active_d_.upload(active_h_.data(), B_, s_);
  }

  // Unscaled residuals / objectives of every active instance (x_hat, y_hat, slack of the last
  // major step), like the single-LP evaluation; where the iterations do not fill the GPU, on a stream
  // of its own beside the plain iterations that follow, which do not write what it reads.
  void post_check()
  {
    const int m = in_.m, n = in_.n;
    if (cs_check_ != s_) B200_CUDA_CHECK(cudaStreamWaitEvent(cs_check_, kept_, 0));
    b_unscale_kernel<TX><<<vgrid_, kBlock, 0, cs_check_>>>(
      xhat_.data(), yhat_.data(), slack_.data(), dc_.data(), dr_.data(), beta_d_.data(),
      gamma_d_.data(), cinst_.data(), rinst_.data(), active_d_.data(), n, m, xu_.data(), yu_.data(),
      su_.data());
    const auto A = wview<double>(true, L_.A.val.data()), AT = wview<double>(false, L_.AT.val.data());
    const int gp = sell_grid(A), gd = sell_grid(AT);
    double* col_planes = tplanes_.data() + 2 * stride_;
    b_term_kernel<<<gp + gd, kBlock, 0, cs_check_>>>(
      A, AT, xu_.data(), yu_.data(),
      b_term_primal_epi{lc64_.data(), uc64_.data(), yu_.data(), tplanes_.data(), stride_,
                        ctx_rows()},
      b_term_dual_epi{c64_.data(), xu_.data(), su_.data(), col_planes, stride_, ctx_cols()}, gp);
    const b_side rows{rows_.chunks.data(), rows_.offsets.data(), rows_.count, tplanes_.data(),
                      tpart_.data(), tarrived_.data(), hbuf_};
    const b_side cols{cols_.chunks.data(), cols_.offsets.data(), cols_.count, col_planes,
                      tpart_.data() + 2 * (size_t)rows_.count, tarrived_.data() + B_,
                      hbuf_ + 2 * (size_t)B_};
    // Instances without rows or columns have no chunk that would write their sums.
    for (int b = 0; b < B_; ++b) {
      const int4 r = rranges_[b], c = cranges_[b];
      if (r.x == r.y && r.z == r.w) std::fill_n(hbuf_ + 2 * (size_t)b, 2, 0.0);
      if (c.x == c.y && c.z == c.w) std::fill_n(hbuf_ + 2 * (size_t)B_ + 3 * (size_t)b, 3, 0.0);
    }
    if (rows_.count + cols_.count > 0)
      b_term_sums_kernel<<<rows_.count + cols_.count, kBlock, 0, cs_check_>>>(rows, cols, stride_,
                                                                       active_d_.data());
    launches_ += 3;
    if (persist_used_)
      B200_CUDA_CHECK(cudaMemcpyAsync(hstatus_, &pctl_.data()->status, sizeof(int),
                                      cudaMemcpyDeviceToHost, cs_check_));
    status_posted_ = persist_used_;
    persist_used_  = false;
    B200_LAUNCH_CHECK();
    B200_CUDA_CHECK(cudaEventRecord(checked_, cs_check_));
  }
  std::vector<inst_conv> wait_check()
  {
    B200_CUDA_CHECK(cudaEventSynchronize(checked_));
    if (status_posted_) check_status();
    collect_form_timing();
    std::vector<inst_conv> cv(B_);
    for (int b = 0; b < B_; ++b) {
      if (!active_h_[b]) continue;
      const double* pr = hbuf_ + 2 * b;
      const double* du = hbuf_ + 2 * B_ + 3 * b;
      inst_conv& c     = cv[b];
      c.l2_primal      = std::sqrt(pr[0]);
      c.l2_dual        = std::sqrt(du[0]);
      c.primal_obj     = du[1];
      c.dual_obj       = du[2] + pr[1];
      if (obj_scale_[b] != 1.0 || obj_offset_[b] != 0.0) {
        c.primal_obj = obj_scale_[b] * (c.primal_obj + obj_offset_[b]);
        c.dual_obj   = obj_scale_[b] * (c.dual_obj + obj_offset_[b]);
      }
      c.gap     = std::fabs(c.primal_obj - c.dual_obj);
      c.abs_obj = std::fabs(c.primal_obj) + std::fabs(c.dual_obj);
    }
    return cv;
  }

  void finish(int b, int status, const inst_conv& c, long k)
  {
    pdlp_result& r   = results_[b];
    r.status         = status;
    r.iterations     = k;
    r.primal_obj     = c.primal_obj;
    r.dual_obj       = c.dual_obj;
    r.l2_primal      = c.l2_primal;
    r.l2_dual        = c.l2_dual;
    r.rel_primal     = c.l2_primal / (1.0 + b_norm_[b]);
    r.rel_dual       = c.l2_dual / (1.0 + c_norm_[b]);
    r.gap            = c.gap;
    r.rel_gap        = c.gap / (1.0 + c.abs_obj);
    r.step_size      = eta_[b];
    r.primal_weight  = omega_[b];
    r.restarts       = restarts_[b];
    r.solve_time     = now_s() - t_start_;
    active_h_[b]     = 0;
  }

  // Same schedule and per-instance decisions as engine::loop of the single-LP solver.
  void loop()
  {
    const int m = in_.m, n = in_.n;
    const double qnan = std::numeric_limits<double>::quiet_NaN();
    const double inf  = std::numeric_limits<double>::infinity();
    std::vector<double> fpe(B_, qnan), fpe0(B_, qnan), last_trial(B_, inf);
    std::vector<double> pid_sum(B_, 0.0), pid_last(B_, 0.0), best_gap(B_, inf);
    std::vector<long> since(B_, 0);
    std::vector<int> restarted(B_, 0);
    // Stall test of mixed precision (per instance; see kStallWindow).
    std::vector<double> stall_ref(B_, std::numeric_limits<double>::infinity());
    std::vector<long> stall_k(B_, 0);
    int n_active = B_, listed = B_;
    upload_scalars(since);
    B200_CUDA_CHECK(cudaEventRecord(kept_, s_));
    // As in the single engine: a check takes about 40 us until the host has read it.  Its stream follows
    // the time of an iteration here: by what fits in L2, as for single LPs, 16 FP64 LPs of 500 to 5000
    // rows took 27.2 ms instead of 25.7, 48 mixed ones of 200 to 3000 rows 26.0 instead of 27.0, and
    // others the same.
    const double est_us = 9.0 + 2.0 * (double)L_.nnz / 2.5e5;
    const bool small    = est_us <= 16.0;
    const long ahead    = small ? 8 : std::max(1L, (long)std::ceil(40.0 / est_us));
    cs_check_           = small ? es_ : s_;
    std::vector<inst_conv> cv;
    // Reads the outstanding check; false when no instance is left.  Instances that end are taken out
    // of the iterations from here on (their solution is the check's, which is not written again).
    auto resolve = [&]() {
      const long kc = posted_;
      posted_       = -1;
      cv            = wait_check();
      const bool out_of_time = now_s() - t_start_ >= p_.time_limit;
      const int before       = n_active;
      for (int b = 0; b < B_; ++b) {
        if (!active_h_[b]) continue;
        const inst_conv& c   = cv[b];
        const bool primal_ok = c.l2_primal <= p_.abs_primal + p_.rel_primal * b_norm_[b];
        const bool optimal   = c.l2_dual <= p_.abs_dual + p_.rel_dual * c_norm_[b] && primal_ok &&
                             c.gap <= p_.abs_gap + p_.rel_gap * c.abs_obj;
        if (kc > 1 && optimal)
          finish(b, kOptimal, c, kc);
        else if (out_of_time)
          finish(b, kTimeLimit, c, kc);
        else if (kc >= p_.iteration_limit)
          finish(b, kIterationLimit, c, kc);
        else if (!std::isfinite(c.l2_primal) || !std::isfinite(c.l2_dual))
          finish(b, kNumericalError, c, kc);
        else if (std::is_same_v<TX, float>) {
          const double q = termination_distance(
            c.l2_primal, p_.abs_primal + p_.rel_primal * b_norm_[b], c.l2_dual,
            p_.abs_dual + p_.rel_dual * c_norm_[b], c.gap, p_.abs_gap + p_.rel_gap * c.abs_obj);
          if (q <= 0.5 * stall_ref[b]) {
            stall_ref[b] = q;
            stall_k[b]   = kc;
          } else if (kc - stall_k[b] >= kStallWindow)
            finish(b, kStalled, c, kc);
        }
      }
      n_active = (int)std::count(active_h_.begin(), active_h_.end(), 1);
      if (n_active == 0) return false;
      if (n_active < before) active_d_.upload(active_h_.data(), B_, s_);
      if (2 * n_active <= listed) {
        B200_CUDA_CHECK(cudaStreamSynchronize(s_));  // no graph is destroyed while it runs
        rebuild_work(active_h_);
        listed = n_active;
        char what[96];
        std::snprintf(what, sizeof what, "batch: loop to %ld its, %d instances left", kc, n_active);
        trace(what);
      }
      return true;
    };

    for (long k = 0;;) {
      const bool major = (k % kMajor == 0 && k > 0) || k <= 0;
      const bool cond  = (k % conditional_major(k)) == 0;
      std::fill(restarted.begin(), restarted.end(), 0);
      bool any_restart = false;
      if (major || cond) {
        close_cycle(k);
        post_check();
        posted_ = k;
        if (major && !resolve()) break;

        if (major) {
          // Restart distances of every active instance.
          sq_diff_kernel<TX><<<vgrid_, kBlock, 0, s_>>>(xa_.data(), xhat_.data(), n,
                                                        rowbuf_.data());
          seg_reduce<1>(false, 0, true);
          sq_diff_kernel<TX><<<vgrid_, kBlock, 0, s_>>>(ya_.data(), yhat_.data(), m,
                                                        rowbuf_.data());
          seg_reduce<1>(true, B_, true);
          launches_ += 2;
          fetch(0, 2 * (size_t)B_, hbuf_);
          for (int b = 0; b < B_; ++b) {
            if (!active_h_[b]) continue;
            // should_cupdlpx_restart (reference pdlp_restart_strategy.cu:689-754)
            bool restart = false;
            if (k == kMajor)
              restart = true;
            else if (k > kMajor) {
              if (fpe[b] <= kSufficientReduction * fpe0[b])
                restart = true;
              else if (fpe[b] <= kNecessaryReduction * fpe0[b] && fpe[b] > last_trial[b])
                restart = true;
              else if ((double)since[b] >= kArtificialRestart * (double)k)
                restart = true;
            }
            last_trial[b] = fpe[b];
            if (!restart) continue;
            // cupdlpx_restart + PID primal weight (reference pdlp_restart_strategy.cu:758-986)
            const inst_conv& c      = cv[b];
            const double rel_dual   = c.l2_dual / (1.0 + c_norm_[b]);
            const double rel_primal = c.l2_primal / (1.0 + b_norm_[b]);
            const double lp = std::sqrt(hbuf_[b]), ld = std::sqrt(hbuf_[B_ + b]);
            const double ratio = rel_primal == 0.0 ? inf : rel_dual / rel_primal;
            if (lp > 1e-16 && ld > 1e-16 && lp < 1e12 && ld < 1e12 && ratio > 1e-8 &&
                ratio < 1e8) {
              const double err  = std::log(ld) - std::log(lp) - std::log(omega_[b]);
              pid_sum[b]        = pid_sum[b] * kISmooth + err;
              const double derr = err - pid_last[b];
              omega_[b]   = std::exp(kKp * err + kKi * pid_sum[b] + kKd * derr) * omega_[b];
              pid_last[b] = err;
            } else {
              omega_[b]    = best_omega_[b];
              pid_sum[b]   = 0.0;
              pid_last[b]  = 0.0;
            }
            const double rgap = std::fabs(std::log10(ratio));
            if (rgap < best_gap[b]) {
              best_gap[b]    = rgap;
              best_omega_[b] = omega_[b];
            }
            since[b]      = 0;
            last_trial[b] = inf;
            restarted[b]  = 1;
            any_restart   = true;
            ++restarts_[b];
          }
          if (any_restart) {
            restart_flags_.resize(B_);
            restart_flags_.upload(restarted.data(), B_, s_);
            b_restart_kernel<TX><<<vgrid_, kBlock, 0, s_>>>(
              x_.data(), xa_.data(), xhat_.data(), n, y_.data(), ya_.data(), yhat_.data(), m,
              cinst_.data(), rinst_.data(), restart_flags_.data());
            ++launches_;
            upload_scalars(since);
          }
        }
        B200_LAUNCH_CHECK();
      }

      const bool mstep   = is_major_step(k);
      const bool fpe_all = ((k + 1) % kMajor == 0);
      if (!mstep && !fpe_all && !any_restart) {
        long R = 1;
        while (R < 255) {
          const long kk = k + R;
          if (is_check(kk) || is_major_step(kk) || ((kk + 1) % kMajor == 0)) break;
          ++R;
        }
        if (posted_ >= 0) R = std::min(R, ahead);
        run_plain(R, k);
        k += R;
        for (int b = 0; b < B_; ++b)
          if (active_h_[b]) since[b] += R;
        if (posted_ >= 0 && !resolve()) break;
        continue;
      }
      if (posted_ >= 0 && !resolve()) break;

      if (fpe_all || any_restart) {
        // Every active instance takes the fixed-point-error form of the step (the same update
        // with the Halpern step applied separately); only instances that need the error use it.
        if (mstep) {
          launch_primal<true, false, true>(0);
          launch_dual<true, false, true>(0);
          B200_CUDA_CHECK(cudaEventRecord(kept_, s_));
        } else {
          launch_primal<false, false, true>(0);
          launch_dual<false, false, true>(0);
        }
        seg_reduce<1>(true, 0, true);
        const auto AT = wview<TX>(false, ATs_.data());
        sell_map_kernel<TX, TX, b_fpe_epi<TX>><<<sell_grid(AT), kBlock, 0, s_>>>(
          AT, ybar_.data(),
          b_fpe_epi<TX>{aty_.data(), xbar_.data(), x_.data(), rowbuf_.data(), stride_, ctx_cols()},
          partials_.data());
        seg_reduce<2>(false, B_, true);
        b_halpern_kernel<TX><<<vgrid_, kBlock, 0, s_>>>(x_.data(), xbar_.data(), xa_.data(), n,
                                                        y_.data(), ybar_.data(), ya_.data(), m,
                                                        cinst_.data(), rinst_.data(),
                                                        active_d_.data(), sc_d_.data());
        advance(1);
        launches_ += 2;
        B200_LAUNCH_CHECK();
        fetch(0, 3 * (size_t)B_, hbuf_);
        for (int b = 0; b < B_; ++b) {
          if (!active_h_[b] || !(fpe_all || restarted[b])) continue;
          const double ndy = hbuf_[b], inter = hbuf_[B_ + 2 * b], ndx = hbuf_[B_ + 2 * b + 1];
          const double movement = ndx * omega_[b] + ndy / omega_[b];
          fpe[b]                = std::sqrt(movement + 2.0 * inter * eta_[b]);
          if (restarted[b]) fpe0[b] = fpe[b];
        }
      } else {
        launch_primal<true, true, false>(0);
        launch_dual<true, true, false>(0);
        B200_CUDA_CHECK(cudaEventRecord(kept_, s_));
        advance(1);
        B200_LAUNCH_CHECK();
      }
      ++k;
      for (int b = 0; b < B_; ++b)
        if (active_h_[b]) ++since[b];
    }
  }

  void write_outputs(double* x_out, double* y_out, double* rc_out)
  {
    const int m = in_.m, n = in_.n;
    B200_CUDA_CHECK(cudaStreamSynchronize(es_));
    if (x_out)
      scatter_by_inst_kernel<<<vgrid_, kBlock, 0, s_>>>(xu_.data(), L_.col_new2old.data(),
                                                        cinst_.data(), nullptr, n, x_out);
    if (rc_out)
      scatter_by_inst_kernel<<<vgrid_, kBlock, 0, s_>>>(su_.data(), L_.col_new2old.data(),
                                                        cinst_.data(), sgn_d_.data(), n, rc_out);
    if (y_out)
      scatter_by_inst_kernel<<<vgrid_, kBlock, 0, s_>>>(yu_.data(), L_.row_new2old.data(),
                                                        rinst_.data(), sgn_d_.data(), m, y_out);
    B200_LAUNCH_CHECK();
    B200_CUDA_CHECK(cudaStreamSynchronize(s_));
  }

  // ---------------------------------------------------------------- state
  const batch_device_input& in_;
  const pdlp_params& p_;
  cudaStream_t s_;
  int B_;
  int sms_ = 148, vgrid_ = 592;
  double* hbuf_ = nullptr;
  // Termination checks: their stream, the event of the last step that kept x_hat / y_hat / slack,
  // the event of the last check's end, the check that has been launched but not read yet, and
  // its planes and sums.
  cudaStream_t es_     = nullptr, cs_check_ = nullptr;  // cs_check_: es_, or s_ for large batches
  cudaEvent_t kept_    = nullptr;
  cudaEvent_t checked_ = nullptr;
  long posted_         = -1;
  bool status_posted_  = false;
  dbuf<double> tplanes_, tpart_;
  dbuf<unsigned> tarrived_;
  double t_start_ = 0, t_loop_ = 0;
  double launches_ = 0;
  size_t stride_ = 0;

  device_layout L_;
  dbuf<TX> As_, ATs_;
  dbuf<int> rinst_, cinst_, active_d_, restart_flags_;
  dbuf<int4> rr_d_, cr_d_;
  std::vector<int4> rranges_, cranges_;
  dbuf<double> c64_, l64_, u64_, lc64_, uc64_, dr_, dc_, sgn_d_, beta_d_, gamma_d_;
  dbuf<TX> cs_, ls_, us_, lcs_, ucs_;
  dbuf<TX> x_, xhat_, slack_, xbar_, xa_, aty_, y_, yhat_, ybar_, ya_;
  dbuf<double> xu_, yu_, su_, rowbuf_, segout_, partials_;
  dbuf<pdlp_scalars> sc_d_;

  std::vector<double> obj_scale_, obj_offset_, c_norm_, b_norm_, beta_, gamma_, eta_, omega_,
    best_omega_;
  std::vector<int> restarts_, power_iters_, active_h_;
  std::vector<pdlp_result> results_;
  std::map<int, cudaGraphExec_t> graphs_;
  work_list wa_, wt_;
  bool lists_on_ = false;
  chunk_table rows_, cols_;
  dbuf<double> chunk_part_;
  // Persistent plain iterations: control block, grid, the choice of form for the current work
  // list, and the choice made while every instance ran (reported in the results).
  dbuf<persist_ctl> pctl_;
  int* hstatus_      = nullptr;
  bool cycle_open_ = false, cycle_one_time_ = false;
  int cycle_form_  = 0;
  long cycle_k0_   = 0;
  int persist_grid_  = 0;
  bool persist_used_ = false;
  long persist_launches_ = 0;
  plain_form_tuner form_;
  int form_active_ = 0, form_epochs_ = 0;
  int first_form_ = -1, first_blocks_ = 0;
  double first_us_[2] = {0, 0};
  batch_key form_key_{};           // the current work list's form decision in batch_form_cache
  double known_us_[2] = {0, 0};    // its timings, when it was remembered from an earlier solve
  // Warps per block of the plain sweeps and the timings they were chosen by.
  int wpb_primal_ = kWarpsPerBlock, wpb_dual_ = kWarpsPerBlock;
  double wpb_ms_[2][3] = {{0, 0, 0}, {0, 0, 0}};
};


}  // namespace

std::vector<pdlp_result> pdlp_batch_solve_device(const batch_device_input& in,
                                                 const pdlp_params& p, cudaStream_t stream,
                                                 double* x_out, double* y_out, double* rc_out)
{
  if (in.count <= 0 || in.count > 65535)
    throw std::invalid_argument("batch size must be in [1, 65535]");
  configure_pool_once();
  joined_stream js(stream);
  if (p.precision == 1) {
    batch_engine<float> e(in, p, js.own);
    return e.run(x_out, y_out, rc_out);
  }
  batch_engine<double> e(in, p, js.own);
  return e.run(x_out, y_out, rc_out);
}

}  // namespace cuopt_b200
