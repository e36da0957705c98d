// Batched LSQR on sm_100a: many small sparse least-squares systems, one cluster each.
//
// The KKT adjoint and the vertex polish both need solves with the active-set matrix M = A_{R,F}
// (rows held at a bound x variables strictly inside their bounds) or its transpose.  These are
// non-symmetric and, on random sparse LPs, ill-conditioned (condition numbers 1e4 - 1e5 for the
// 5000 x 5000 bases of the 64-LP adjoint workload), where restarted GMRES and BiCGStab stall and
// LSQR converges in 7 000 - 11 000 iterations.  A batch of such systems would need two kernel
// boundaries and a reduction per system per iteration if each iteration were a grid-wide launch,
// so instead every system gets one thread-block cluster that runs its whole LSQR loop:
//   * every block of the cluster holds a copy of u (rows) and v (cols) in shared memory, gathers
//     from it, and sends each new entry to every block's copy with st.async, whose bytes count
//     towards the receiving block's mbarrier; x and w are kept by the block that owns their column;
//   * the operator and its transpose are stored as 32-row sliced ELL (lane t of a warp owns row t
//     of a slice and reads element k at base + 32 k + t), rows sorted by length; slice s belongs to
//     block s % C, whose share is copied into its shared memory (16-bit indices) where it fits, so
//     that an iteration reads no global memory;
//   * the two norms of an iteration are sums of per-slice sums, sent to every block with the vector
//     entries and added in the slices' order by every warp, so the scalar recurrence and the stopping
//     decision are uniform, and an iteration costs two products and two exchanges.  A warp sends the
//     sums of a slice after its gathers (a warp without slices sends zeros that nobody adds), so a
//     block that has all of one exchange knows that every warp is done reading the vector written
//     next, and has read the sums of the exchange before.  No sum depends on the number of blocks, and
//     every product that the compiler could fuse or not is written out: a system's result is the
//     same bits whatever cluster it runs in, that is, whatever else is in its batch;
//   * the x / w update of an iteration is applied in the next transpose product by the thread that
//     owns the row.
// One block per system, reading the operator from L2, took 33 us an iteration on the 5000 x 5000
// systems.  Systems whose vectors do not fit in clusters of 8 (some 25 000 rows and columns together)
// still run in one block each, with u, v, x and w in global memory.
// Each cluster stops at LSQR's tests or at its iteration limit: none waits for another, and a wait
// for an exchange is bounded (its end without one is reported as an error).
#include "common.cuh"
#include "lsqr.hpp"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <numeric>
#include <thread>

namespace cuopt_b200 {

namespace {

constexpr int kLsqrThreads = 512;
constexpr int kLsqrWarps   = kLsqrThreads / kWarp;
// Blocks of a cluster: 8 warps, so that a thread has the registers for eight elements in flight, its
// row's state and the remote addresses (with 16 warps some 500 bytes of it spilled).
constexpr int kClThreads = 256;
constexpr int kClWarps   = kClThreads / kWarp;
constexpr int kEquilibrationPasses = 10;
constexpr int kLsqrFailed = -1;       // flag of a system whose exchange did not complete

struct lsqr_desc {
  int rows, cols;           // u has `rows` entries, v / x / w have `cols`
  int slices_p, slices_q;   // slices of P (= Op, rows x cols) and Q (= Op^T, cols x rows)
  const int64_t* p_slice;   // slices_p + 1 element offsets
  const int* p_idx;
  const double* p_val;
  const int64_t* q_slice;   // slices_q + 1
  const int* q_idx;
  const double* q_val;
  const double* b;          // rows (sorted, equilibrated)
  double* z;                // cols (sorted, equilibrated)
  double* scratch;          // rows + 3 cols doubles (systems that run in one block each)
  int64_t share_p, share_q; // most elements of P and Q that one block of a cluster holds
  int max_iter;
  double tol;
};

struct lsqr_out {
  int iterations;
  int flag;
  double rnorm;
  double arnorm;
};

// Sum over the block of K per-thread values; every thread gets the same totals (fixed order).
template <int K, int WARPS = kLsqrWarps>
__device__ __forceinline__ void block_sums(const double (&v)[K], double* part, double (&out)[K])
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const double s = warp_sum(v[q]);
    if (lane == 0) part[warp * K + q] = s;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < K; ++q) {
    double s = 0.0;
    for (int w = 0; w < WARPS; ++w) s += part[w * K + q];
    out[q] = s;
  }
}

// acc_r = sum_k val[r, k] vec[idx[r, k]] for the rows of a sliced-ELL matrix; f(r, acc_r) for the
// rows this thread owns (row s * 32 + lane of slice s, slices dealt to warps round-robin).
template <class F>
__device__ __forceinline__ void slice_products(int slices, int rows, const int64_t* __restrict__ so,
                                               const int* __restrict__ idx,
                                               const double* __restrict__ val,
                                               const double* vec, F&& f)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int s = warp; s < slices; s += kLsqrWarps) {
    const int64_t base = so[s];
    const int len      = (int)((so[s + 1] - base) >> 5);
    const int* ip      = idx + base + lane;
    const double* vp   = val + base + lane;
    double acc         = 0.0;
    int k              = 0;
    for (; k + 2 <= len; k += 2) {
      const int i0 = ip[32 * k], i1 = ip[32 * k + 32];
      const double a0 = vp[32 * k], a1 = vp[32 * k + 32];
      acc += a0 * vec[i0];
      acc += a1 * vec[i1];
    }
    if (k < len) acc += vp[32 * k] * vec[ip[32 * k]];
    const int r = s * kWarp + lane;
    if (r < rows) f(r, acc);
  }
}

__global__ void __launch_bounds__(kLsqrThreads, 1) lsqr_kernel(const lsqr_desc* __restrict__ descs,
                                                            lsqr_out* __restrict__ outs)
{
  __shared__ double part_a[kLsqrWarps * 2], part_b[kLsqrWarps * 2];
  const lsqr_desc d = descs[blockIdx.x];
  double* u = d.scratch;
  double* v = u + d.rows;
  double* x = v + d.cols;
  double* w = x + d.cols;
  const int T = kLsqrThreads;

  // u = b, beta = |b|
  double t1[1] = {0.0}, r1[1];
  for (int r = threadIdx.x; r < d.rows; r += T) {
    const double bv = d.b[r];
    u[r]            = bv;
    t1[0] += bv * bv;
  }
  block_sums<1>(t1, part_a, r1);
  double beta        = sqrt(r1[0]);
  const double bnorm = beta;
  if (!(beta > 0.0) || !isfinite(beta)) {
    for (int j = threadIdx.x; j < d.cols; j += T) d.z[j] = 0.0;
    if (threadIdx.x == 0) outs[blockIdx.x] = lsqr_out{0, 0, beta, 0.0};
    return;
  }
  double us = 1.0 / beta;  // the normalised u is u * us
  // v = Op^T u / beta, alpha = |v|; x = w = 0 (w becomes v_1 in the first transpose product)
  t1[0] = 0.0;
  slice_products(d.slices_q, d.cols, d.q_slice, d.q_idx, d.q_val, u, [&](int j, double acc) {
    const double vj = acc * us;
    v[j]            = vj;
    x[j]            = 0.0;
    w[j]            = 0.0;
    t1[0] += vj * vj;
  });
  block_sums<1>(t1, part_b, r1);
  double alpha  = sqrt(r1[0]);
  double vs     = alpha > 0.0 ? 1.0 / alpha : 0.0;
  double rhobar = alpha, phibar = beta, anorm2 = 0.0, xnorm = 0.0;
  double c1 = 0.0, c2 = 0.0;  // pending update: x += c1 w; w = v - c2 w
  double rnorm = beta, arnorm = alpha * beta;
  int flag = 3, it = 0;
  if (!(alpha > 0.0)) {
    flag = 2;  // Op^T b = 0: z = 0 is the least-squares solution
  } else {
    for (it = 1; it <= d.max_iter; ++it) {
      // u <- Op v - alpha u  (normalised v = v * vs, normalised u = u * us)
      t1[0] = 0.0;
      slice_products(d.slices_p, d.rows, d.p_slice, d.p_idx, d.p_val, v, [&](int r, double acc) {
        const double un = acc * vs - alpha * (u[r] * us);
        u[r]            = un;
        t1[0] += un * un;
      });
      block_sums<1>(t1, part_a, r1);
      beta = sqrt(r1[0]);
      us   = beta > 0.0 ? 1.0 / beta : 0.0;
      anorm2 += alpha * alpha + beta * beta;
      // pending x / w update, then v <- Op^T u - beta v
      double t2[2] = {0.0, 0.0}, r2[2];
      slice_products(d.slices_q, d.cols, d.q_slice, d.q_idx, d.q_val, u, [&](int j, double acc) {
        const double vo = v[j] * vs;
        double wj       = w[j];
        const double xj = x[j] + c1 * wj;
        wj              = vo - c2 * wj;
        x[j]            = xj;
        w[j]            = wj;
        const double vn = acc * us - beta * vo;
        v[j]            = vn;
        t2[0] += vn * vn;
        t2[1] += xj * xj;
      });
      block_sums<2>(t2, part_b, r2);
      alpha = sqrt(r2[0]);
      vs    = alpha > 0.0 ? 1.0 / alpha : 0.0;
      xnorm = sqrt(r2[1]);
      // Plane rotation (no damping) and the new pending update.
      const double rho = sqrt(rhobar * rhobar + beta * beta);
      const double cs = rhobar / rho, sn = beta / rho;
      const double theta = sn * alpha;
      rhobar             = -cs * alpha;
      const double phi   = cs * phibar;
      phibar             = sn * phibar;
      c1                 = phi / rho;
      c2                 = theta / rho;
      rnorm              = phibar;
      arnorm             = alpha * fabs(sn * phi);
      const double anorm = sqrt(anorm2);
      if (rnorm <= d.tol * bnorm + d.tol * anorm * xnorm) {
        flag = 1;
        break;
      }
      if (arnorm <= d.tol * anorm * rnorm) {
        flag = 2;
        break;
      }
      if (!(alpha > 0.0) || !(beta > 0.0)) {  // exact breakdown: the Krylov space is exhausted
        flag = 1;
        break;
      }
    }
    if (it > d.max_iter) it = d.max_iter;
  }
  // The last pending x update, then the result.
  for (int j = threadIdx.x; j < d.cols; j += T) d.z[j] = x[j] + c1 * w[j];
  if (threadIdx.x == 0) outs[blockIdx.x] = lsqr_out{it, flag, rnorm, arnorm};
}

// Entries of the sums of one exchange: one per slice, and one for every warp of the cluster that has
// none (slice s is the first of warp s / C of block s % C).
B200_HD inline size_t sum_slots(int slices, int C)
{
  return slices > C * kClWarps ? slices : C * kClWarps;
}
// Shared memory of one block of a cluster of C for a system: u, v, the x and w of the block's
// columns, the per-slice sums of the two norms, and with `cached` the block's shares of P and Q:
// {start, length} per slice, values, 16-bit indices.
struct lsqr_smem {
  size_t v, x, w, part_a, part_b, tab[2], val[2], idx[2], bytes;
  static B200_HD size_t pad(size_t b) { return (b + 15) & ~(size_t)15; }
  B200_HD lsqr_smem(int rows, int cols, int slices_p, int slices_q, int64_t elems_p,
                    int64_t elems_q, int C, bool cached)
  {
    size_t at    = 16 + pad((size_t)rows * 8);  // two barriers, u
    auto take    = [&](size_t b) {
      const size_t here = at;
      at += pad(b);
      return here;
    };
    const size_t np = (size_t)(slices_p + C - 1) / C, nq = (size_t)(slices_q + C - 1) / C;
    v      = take((size_t)cols * 8);
    x      = take(nq * kWarp * 8);
    w      = take(nq * kWarp * 8);
    part_a = take(sum_slots(slices_p, C) * 8);
    part_b = take(sum_slots(slices_q, C) * 16);
    tab[0] = take(cached ? np * 8 : 0);
    tab[1] = take(cached ? nq * 8 : 0);
    val[0] = take(cached ? (size_t)elems_p * 8 : 0);
    val[1] = take(cached ? (size_t)elems_q * 8 : 0);
    idx[0] = take(cached ? (size_t)elems_p * 2 : 0);
    idx[1] = take(cached ? (size_t)elems_q * 2 : 0);
    bytes  = at;
  }
};

__device__ __forceinline__ unsigned lsqr_rank()
{
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void lsqr_barrier()
{
  __syncwarp();
  asm volatile(
    "barrier.cluster.arrive.release.aligned;\n"
    "barrier.cluster.wait.acquire.aligned;\n" ::
      : "memory");
}
__device__ __forceinline__ void send_bytes(unsigned to, unsigned bar, double v)
{
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(
                 to),
               "d"(v), "r"(bar)
               : "memory");
}
// Stores v at offset `off` of every block, counted by its barrier at offset `bar`.
template <int C>
__device__ __forceinline__ void send_all(const unsigned (&base)[C], unsigned off, unsigned bar, double v)
{
#pragma unroll
  for (int c = 0; c < C; ++c) send_bytes(base[c] + off, base[c] + bar, v);
}

// Warp sums of K values (as warp_sum, step by step together).
template <int K>
__device__ __forceinline__ void warp_sums(const double (&v)[K], double (&s)[K])
{
#pragma unroll
  for (int q = 0; q < K; ++q) s[q] = v[q];
#pragma unroll
  for (int o = kWarp / 2; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < K; ++q) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
}
// Sends the warp's sums of K per-thread values for slot `slot` of `slots` (planes of them) to every
// block (lane c to block c; `mine`: that block's base address); once all are in, cluster_totals adds
// those of the slices in one order everywhere.
template <int K, int C>
__device__ __forceinline__ void send_sums(const double (&v)[K], unsigned mine, unsigned part,
                                          unsigned bar, int slot, int slots)
{
  double s[K];
  warp_sums<K>(v, s);
  if ((threadIdx.x & 31) < C) {
#pragma unroll
    for (int q = 0; q < K; ++q) send_bytes(mine + part + 8u * (q * slots + slot), mine + bar, s[q]);
  }
}
template <int K>
__device__ __forceinline__ void cluster_totals(const double* part, int slices, int slots,
                                               double (&out)[K])
{
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < K; ++q) out[q] = 0.0;
  for (int i = lane; i < slices; i += 4 * kWarp) {  // four at a time, so that their loads overlap
    double e[K][4];
#pragma unroll
    for (int q = 0; q < K; ++q)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        e[q][j] = i + j * kWarp < slices ? part[q * slots + i + j * kWarp] : 0.0;
#pragma unroll
    for (int q = 0; q < K; ++q)
#pragma unroll
      for (int j = 0; j < 4; ++j) out[q] += e[q][j];
  }
  warp_sums<K>(out, out);
}

template <int C, bool CACHED>
__global__ void __launch_bounds__(kClThreads, 1)
  lsqr_cluster_kernel(const lsqr_desc* __restrict__ descs, lsqr_out* __restrict__ outs)
{
  extern __shared__ __align__(16) unsigned char dyn[];
  const unsigned rank = lsqr_rank();
  const int system    = (int)blockIdx.x / C;
  const lsqr_desc d   = descs[system];
  const lsqr_smem S(d.rows, d.cols, d.slices_p, d.slices_q, d.share_p, d.share_q, C, CACHED);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, T = kClThreads;
  auto at        = [&](size_t o) { return reinterpret_cast<double*>(dyn + o); };
  double *u = at(16), *v = at(S.v), *x = at(S.x), *w = at(S.w);
  double *part_a = at(S.part_a), *part_b = at(S.part_b);
  const int np = (d.slices_p + C - 1) / C, nq = (d.slices_q + C - 1) / C;

  if constexpr (CACHED) {
    for (int m = 0; m < 2; ++m) {
      const int n           = m == 0 ? np : nq, slices = m == 0 ? d.slices_p : d.slices_q;
      const int64_t* so     = m == 0 ? d.p_slice : d.q_slice;
      const int* gi         = m == 0 ? d.p_idx : d.q_idx;
      const double* gv      = m == 0 ? d.p_val : d.q_val;
      int2* tab             = reinterpret_cast<int2*>(dyn + S.tab[m]);
      double* val           = at(S.val[m]);
      unsigned short* idx   = reinterpret_cast<unsigned short*>(dyn + S.idx[m]);
      if (threadIdx.x == 0) {
        int start = 0;
        for (int i = 0; i < n; ++i) {
          const int s   = (int)rank + C * i;
          const int len = s < slices ? (int)(so[s + 1] - so[s]) : 0;
          tab[i]        = make_int2(start, len >> 5);
          start += len;
        }
      }
      __syncthreads();
      for (int i = warp; i < n; i += kClWarps) {
        const int s = (int)rank + C * i;
        if (s >= slices) break;
        const int64_t base = so[s];
        const int2 t       = tab[i];
        for (int k = lane; k < t.y * kWarp; k += kWarp) {
          val[t.x + k] = gv[base + k];
          idx[t.x + k] = (unsigned short)gi[base + k];
        }
      }
    }
  }
  const int slots_p = (int)sum_slots(d.slices_p, C), slots_q = (int)sum_slots(d.slices_q, C);
  unsigned base[C], mine = 0;  // addresses of the cluster's blocks, and of block `lane`
  // The products of this block's rows of P (m = 0) or Q (m = 1) with `vec`: f(unit, row, product, t)
  // fills the row's terms of the K sums, which go to the entries at `part` of every block.
  auto products = [&](int m, const double* vec, auto& t, unsigned part, auto&& f) {
    constexpr int K = (int)(sizeof(t) / sizeof(double));
    const int n = m == 0 ? np : nq, slices = m == 0 ? d.slices_p : d.slices_q;
    const int rows = m == 0 ? d.rows : d.cols, slots = m == 0 ? slots_p : slots_q;
    const unsigned bar = 8u * m;
    // The next slice's place is loaded while this one's product is formed (128 systems of 5000 x 5000, one
    // block each, operators in L2: 137 -> 124 ms).
    auto place = [&](int i, int64_t& first, int& len) {
      const int s = (int)rank + C * i;
      first       = 0;
      len         = 0;
      if (s >= slices) return;
      if constexpr (CACHED) {
        const int2 t = reinterpret_cast<const int2*>(dyn + S.tab[m])[i];
        first        = t.x;
        len          = t.y;
      } else {
        const int64_t* so = m == 0 ? d.p_slice : d.q_slice;
        first             = __ldg(so + s);
        len               = (int)((__ldg(so + s + 1) - first) >> 5);
      }
    };
    int64_t next;
    int next_len;
    place(warp, next, next_len);
    for (int i = warp; i < n; i += kClWarps) {
      const int s = (int)rank + C * i;
      if (s >= slices) break;
      const int r         = s * kWarp + lane;
      const int64_t first = next;
      const int len       = next_len;
      place(i + kClWarps, next, next_len);
      double acc  = 0.0;
      // Eight elements at a time, so that their loads, then their gathers, are in flight together.
      auto sum = [&](const double* vp, const auto* ip, int len) {
        for (int k = 0; k < len; k += 8) {
          int j[8];
          double a[8], g[8];
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (k + e < len) {
              j[e] = ip[kWarp * (k + e)];
              a[e] = vp[kWarp * (k + e)];
            }
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (k + e < len) g[e] = vec[j[e]];
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (k + e < len) acc = fma(a[e], g[e], acc);
        }
      };
      if constexpr (CACHED)
        sum(at(S.val[m]) + first + lane,
            reinterpret_cast<const unsigned short*>(dyn + S.idx[m]) + first + lane, len);
      else
        sum((m == 0 ? d.p_val : d.q_val) + first + lane, (m == 0 ? d.p_idx : d.q_idx) + first + lane,
            len);
#pragma unroll
      for (int q = 0; q < K; ++q) t[q] = 0.0;
      if (r < rows) f(i, r, acc, t);
      send_sums<K, C>(t, mine, part, bar, s, slots);
    }
    if ((int)rank + C * warp >= slices) {  // a warp without slices
#pragma unroll
      for (int q = 0; q < K; ++q) t[q] = 0.0;
      send_sums<K, C>(t, mine, part, bar, (int)rank + C * warp, slots);
    }
  };

  // u = b, beta = |b| (every block sums its whole copy)
  double t1[1] = {0.0}, r1[1];
  for (int r = threadIdx.x; r < d.rows; r += T) {
    const double bv = d.b[r];
    u[r]            = bv;
    t1[0] = fma(bv, bv, t1[0]);
  }
  block_sums<1, kClWarps>(t1, part_a, r1);
  __syncthreads();  // part_a is read before other blocks write it
  double beta        = sqrt(r1[0]);
  const double bnorm = beta;
  if (!(beta > 0.0) || !isfinite(beta)) {  // in every block of the cluster
    if (rank == 0) {
      for (int j = threadIdx.x; j < d.cols; j += T) d.z[j] = 0.0;
      if (threadIdx.x == 0) outs[system] = lsqr_out{0, 0, beta, 0.0};
    }
    return;
  }
  // Exchanges of u (after P's products) and of v (after Q's): every entry and every sum, to every block.
  const unsigned home = (unsigned)__cvta_generic_to_shared(dyn), bar_u = home, bar_v = home + 8;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(base[c]) : "r"(home), "r"(c));
    if (lane == c) mine = base[c];
  }
  const unsigned bytes_u = 8u * (d.rows + slots_p), bytes_v = 8u * (d.cols + 2 * slots_q);
  if (threadIdx.x == 0) {
    phase_init(bar_u);
    phase_init(bar_v);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    phase_expect(bar_u, bytes_u);
    phase_expect(bar_v, bytes_v - 8u * slots_q);  // the first one has a single sum
  }
  unsigned phase_u = 0, phase_v = 0;
  bool ok          = true;
  auto wait_v = [&]() {
    if (!(ok = phase_wait(bar_v, phase_v))) return false;
    phase_v ^= 1;
    if (threadIdx.x == 0) phase_expect(bar_v, bytes_v);
    return true;
  };
  // Every block of the cluster is running, with its barriers, before any stores into another's
  // shared memory.
  lsqr_barrier();
  double us = 1.0 / beta;  // the normalised u is u * us
  // v = Op^T u / beta, alpha = |v|; x = w = 0 (w becomes v_1 in the first transpose product)
  products(1, u, t1, (unsigned)S.part_b, [&](int i, int j, double acc, double (&t)[1]) {
    const double vj = acc * us;
    send_all<C>(base, (unsigned)S.v + 8u * j, 8, vj);
    x[i * kWarp + lane] = 0.0;
    w[i * kWarp + lane] = 0.0;
    t[0]                = vj * vj;
  });
  wait_v();
  cluster_totals<1>(part_b, d.slices_q, slots_q, r1);
  double alpha  = sqrt(r1[0]);
  double vs     = alpha > 0.0 ? 1.0 / alpha : 0.0;
  double rhobar = alpha, phibar = beta, anorm2 = 0.0, xnorm = 0.0;
  double c1 = 0.0, c2 = 0.0;  // pending update: x += c1 w; w = v - c2 w
  double rnorm = beta, arnorm = alpha * beta;
  int flag = 3, it = 0;
  if (!ok) {
    flag = kLsqrFailed;
  } else if (!(alpha > 0.0)) {
    flag = 2;  // Op^T b = 0: z = 0 is the least-squares solution
  } else {
    for (it = 1; it <= d.max_iter; ++it) {
      // u <- Op v - alpha u  (normalised v = v * vs, normalised u = u * us)
      products(0, v, t1, (unsigned)S.part_a, [&](int, int r, double acc, double (&t)[1]) {
        const double un = fma(acc, vs, -alpha * (u[r] * us));
        send_all<C>(base, 16 + 8u * r, 0, un);
        t[0] = un * un;
      });
      if (!(ok = phase_wait(bar_u, phase_u))) break;
      phase_u ^= 1;
      if (threadIdx.x == 0) phase_expect(bar_u, bytes_u);
      cluster_totals<1>(part_a, d.slices_p, slots_p, r1);
      beta = sqrt(r1[0]);
      us   = beta > 0.0 ? 1.0 / beta : 0.0;
      anorm2 = fma(alpha, alpha, fma(beta, beta, anorm2));
      // pending x / w update, then v <- Op^T u - beta v
      double t2[2], r2[2];
      products(1, u, t2, (unsigned)S.part_b, [&](int i, int j, double acc, double (&t)[2]) {
        const int q     = i * kWarp + lane;
        const double vo = v[j] * vs;
        double wj       = w[q];
        const double xj = fma(c1, wj, x[q]);
        wj              = fma(-c2, wj, vo);
        x[q]            = xj;
        w[q]            = wj;
        const double vn = fma(acc, us, -beta * vo);
        send_all<C>(base, (unsigned)S.v + 8u * j, 8, vn);
        t[0] = vn * vn;
        t[1] = xj * xj;
      });
      if (!wait_v()) break;
      cluster_totals<2>(part_b, d.slices_q, slots_q, r2);
      alpha = sqrt(r2[0]);
      vs    = alpha > 0.0 ? 1.0 / alpha : 0.0;
      xnorm = sqrt(r2[1]);
      // Plane rotation (no damping) and the new pending update.
      const double rho = sqrt(fma(rhobar, rhobar, beta * beta));
      const double cs = rhobar / rho, sn = beta / rho;
      const double theta = sn * alpha;
      rhobar             = -cs * alpha;
      const double phi   = cs * phibar;
      phibar             = sn * phibar;
      c1                 = phi / rho;
      c2                 = theta / rho;
      rnorm              = phibar;
      arnorm             = alpha * fabs(sn * phi);
      const double anorm = sqrt(anorm2);
      if (rnorm <= fma(d.tol * anorm, xnorm, d.tol * bnorm)) {
        flag = 1;
        break;
      }
      if (arnorm <= d.tol * anorm * rnorm) {
        flag = 2;
        break;
      }
      if (!(alpha > 0.0) || !(beta > 0.0)) {  // exact breakdown: the Krylov space is exhausted
        flag = 1;
        break;
      }
    }
    if (!ok) flag = kLsqrFailed;
    if (it > d.max_iter) it = d.max_iter;
  }
  // Every exchange that was sent to this block is in (each is waited for before the next); after a
  // failed one, all blocks end theirs before any leaves.
  __syncthreads();
  lsqr_barrier();
  // The last pending x update, then the result.
  for (int i = warp; i < nq; i += kClWarps) {
    const int j = ((int)rank + C * i) * kWarp + lane, q = i * kWarp + lane;
    if (j < d.cols) d.z[j] = fma(c1, w[q], x[q]);
  }
  if (threadIdx.x == 0 && (rank == 0 || flag == kLsqrFailed))
    outs[system] = lsqr_out{it, flag, rnorm, arnorm};
}

// Host-side packing of one problem: equilibration, transposition, row sorting, sliced ELL.
struct packed {
  int rows = 0, cols = 0;
  std::vector<double> dr, dc;          // equilibration: Op_s = diag(dr) Op diag(dc)
  std::vector<int> perm_p, perm_q;     // sorted position -> original row (P) / column (Q rows)
  std::vector<int64_t> p_slice, q_slice;
  std::vector<int> p_idx, q_idx;
  std::vector<double> p_val, q_val, b;
};

// Sliced ELL of a CSR matrix (rows sorted by length, descending) whose column indices are mapped
// through `colmap`.
void to_sell(int rows, const std::vector<int64_t>& off, const std::vector<int>& idx,
             const std::vector<double>& val, const std::vector<int>& colmap,
             std::vector<int>& perm, std::vector<int64_t>& slice, std::vector<int>& sidx,
             std::vector<double>& sval)
{
  perm.resize(rows);
  std::iota(perm.begin(), perm.end(), 0);
  std::stable_sort(perm.begin(), perm.end(), [&](int a, int b) {
    return off[a + 1] - off[a] > off[b + 1] - off[b];
  });
  const int slices = (rows + kWarp - 1) / kWarp;
  slice.assign(slices + 1, 0);
  for (int s = 0; s < slices; ++s) {
    const int r0      = perm[s * kWarp];  // the longest row of the slice comes first
    const int64_t len = off[r0 + 1] - off[r0];
    slice[s + 1]      = slice[s] + len * kWarp;
  }
  sidx.assign(slice[slices], 0);
  sval.assign(slice[slices], 0.0);
  for (int s = 0; s < slices; ++s)
    for (int t = 0; t < kWarp && s * kWarp + t < rows; ++t) {
      const int r = perm[s * kWarp + t];
      int k       = 0;
      for (int64_t e = off[r]; e < off[r + 1]; ++e, ++k) {
        sidx[slice[s] + (int64_t)k * kWarp + t] = colmap[idx[e]];
        sval[slice[s] + (int64_t)k * kWarp + t] = val[e];
      }
    }
}

void pack(const lsqr_problem& p, packed& out)
{
  const int R = p.rows, Cc = p.cols;
  out.rows = R;
  out.cols = Cc;
  const int64_t nnz = p.off[R];
  // Two-sided equilibration: repeatedly divide rows and columns by the square roots of their
  // 2-norms (computed from the same scaled matrix), which brings both towards unit norm.
  out.dr.assign(R, 1.0);
  out.dc.assign(Cc, 1.0);
  std::vector<double> rn(R), cn(Cc);
  for (int pass = 0; pass < kEquilibrationPasses; ++pass) {
    std::fill(rn.begin(), rn.end(), 0.0);
    std::fill(cn.begin(), cn.end(), 0.0);
    for (int r = 0; r < R; ++r)
      for (int64_t e = p.off[r]; e < p.off[r + 1]; ++e) {
        const double a = p.val[e] * out.dr[r] * out.dc[p.idx[e]];
        rn[r] += a * a;
        cn[p.idx[e]] += a * a;
      }
    for (int r = 0; r < R; ++r)
      if (rn[r] > 0.0) out.dr[r] /= std::sqrt(std::sqrt(rn[r]));
    for (int j = 0; j < Cc; ++j)
      if (cn[j] > 0.0) out.dc[j] /= std::sqrt(std::sqrt(cn[j]));
  }
  // Scaled P in CSR, and its transpose Q.
  std::vector<double> sv(nnz);
  for (int r = 0; r < R; ++r)
    for (int64_t e = p.off[r]; e < p.off[r + 1]; ++e)
      sv[e] = p.val[e] * out.dr[r] * out.dc[p.idx[e]];
  std::vector<int64_t> qoff(Cc + 1, 0);
  for (int64_t e = 0; e < nnz; ++e) ++qoff[p.idx[e] + 1];
  for (int j = 0; j < Cc; ++j) qoff[j + 1] += qoff[j];
  std::vector<int> qidx(nnz);
  std::vector<double> qval(nnz);
  {
    std::vector<int64_t> pos(qoff.begin(), qoff.end() - 1);
    for (int r = 0; r < R; ++r)
      for (int64_t e = p.off[r]; e < p.off[r + 1]; ++e) {
        const int64_t q = pos[p.idx[e]]++;
        qidx[q]         = r;
        qval[q]         = sv[e];
      }
  }
  // Row orders first (P's columns refer to Q's sorted rows and the other way round).
  std::vector<int> idp(R), idq(Cc);
  std::iota(idp.begin(), idp.end(), 0);
  std::iota(idq.begin(), idq.end(), 0);
  std::vector<int64_t> tmp_slice;
  std::vector<int> tmp_idx;
  std::vector<double> tmp_val;
  out.perm_p.resize(R);
  out.perm_q.resize(Cc);
  std::iota(out.perm_p.begin(), out.perm_p.end(), 0);
  std::stable_sort(out.perm_p.begin(), out.perm_p.end(), [&](int a, int b) {
    return p.off[a + 1] - p.off[a] > p.off[b + 1] - p.off[b];
  });
  std::iota(out.perm_q.begin(), out.perm_q.end(), 0);
  std::stable_sort(out.perm_q.begin(), out.perm_q.end(), [&](int a, int b) {
    return qoff[a + 1] - qoff[a] > qoff[b + 1] - qoff[b];
  });
  std::vector<int> inv_p(R), inv_q(Cc);
  for (int i = 0; i < R; ++i) inv_p[out.perm_p[i]] = i;
  for (int j = 0; j < Cc; ++j) inv_q[out.perm_q[j]] = j;
  std::vector<int> check;
  to_sell(R, p.off, p.idx, sv, inv_q, check, out.p_slice, out.p_idx, out.p_val);
  to_sell(Cc, qoff, qidx, qval, inv_p, check, out.q_slice, out.q_idx, out.q_val);
  out.b.resize(R);
  for (int i = 0; i < R; ++i) out.b[i] = p.b[out.perm_p[i]] * out.dr[out.perm_p[i]];
}

template <typename F>
void parallel_for(int count, F&& f)
{
  const int nt = std::max(1, std::min<int>(count, (int)std::thread::hardware_concurrency()));
  if (nt <= 1) {
    for (int i = 0; i < count; ++i) f(i);
    return;
  }
  std::vector<std::thread> pool;
  std::atomic<int> next{0};
  for (int t = 0; t < nt; ++t)
    pool.emplace_back([&]() {
      for (int i; (i = next++) < count;) f(i);
    });
  for (auto& th : pool) th.join();
}

// Most elements that one of C blocks holds of a sliced matrix (slice s in block s % C).
int64_t most_elements(const std::vector<int64_t>& slice, int C)
{
  std::vector<int64_t> share(C, 0);
  for (size_t s = 0; s + 1 < slice.size(); ++s) share[s % C] += slice[s + 1] - slice[s];
  return *std::max_element(share.begin(), share.end());
}
size_t cluster_smem(const packed& q, int C, bool cached)
{
  return lsqr_smem(q.rows, q.cols, (int)q.p_slice.size() - 1, (int)q.q_slice.size() - 1,
                   cached ? most_elements(q.p_slice, C) : 0,
                   cached ? most_elements(q.q_slice, C) : 0, C, cached)
    .bytes;
}

// Blocks per cluster and whether their shares of the operators are cached.
struct cluster_plan {
  int blocks   = 1;
  bool cached  = false;
  size_t smem  = 0;
  void configure(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&attr)[1], int systems,
                 cudaStream_t s) const
  {
    cfg                      = cudaLaunchConfig_t{};
    cfg.gridDim              = dim3(systems * blocks);
    cfg.blockDim             = dim3(kClThreads);
    cfg.dynamicSmemBytes     = smem;
    cfg.stream               = s;
    // Also for one block: st.async is an illegal instruction in a launch without a cluster size.
    attr[0].id               = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs                = attr;
    cfg.numAttrs             = 1;
  }
};

using cluster_kernel_t = void (*)(const lsqr_desc*, lsqr_out*);
cluster_kernel_t cluster_kernel(int blocks, bool cached)
{
  switch (blocks) {
    case 1: return cached ? lsqr_cluster_kernel<1, true> : lsqr_cluster_kernel<1, false>;
    case 2: return cached ? lsqr_cluster_kernel<2, true> : lsqr_cluster_kernel<2, false>;
    case 4: return cached ? lsqr_cluster_kernel<4, true> : lsqr_cluster_kernel<4, false>;
    case 8: return cached ? lsqr_cluster_kernel<8, true> : lsqr_cluster_kernel<8, false>;
    default: return cached ? lsqr_cluster_kernel<16, true> : lsqr_cluster_kernel<16, false>;
  }
}

// The plan with the least estimated time (smem 0: no shape can be launched): waves of clusters, each iteration of one taking a latency,
// a share for every block and, between blocks, for every entry of u and v, and the products, shared by
// the blocks.  Fitted to these us an iteration with 1, 2, 4, 8 and 16 blocks, operators in shared
// memory, then from L2 (stored elements of both operators, rows + columns):
//      704,   66:  2.7  2.7  2.6  2.7  2.8    3.4  3.3  3.3  3.3  3.7
//    4 704,  600:  3.6  2.6  2.5  2.5  2.7    4.8  3.5  3.5  3.5  3.9
//   13 088, 1600:  5.8  3.8  2.8  2.7  2.9    7.9  5.1  3.7  3.6  4.1
//   40 672, 5000:    -    -  4.8  4.0  4.1   18.3 10.2  7.2  5.8  4.9
// (within 18 %, 7 % in the mean).
// `share`: the part of the GPU that the systems have while others run beside them.
cluster_plan plan_clusters(const std::vector<packed>& pk, const std::vector<int>& ids, size_t limit,
                           double share)
{
  cluster_plan best;
  if (ids.empty()) return best;
  double nnz = 0.0, entries = 0.0, best_us = 0.0;
  for (int i : ids) {
    nnz += (double)(pk[i].p_val.size() + pk[i].q_val.size()) / ids.size();
    entries += (double)(pk[i].rows + pk[i].cols) / ids.size();
  }
  for (const bool cached : {true, false})
    for (const int c : {16, 8, 4, 2, 1}) {
      cluster_plan p;
      p.blocks = c;
      p.cached = cached;
      for (int i : ids) p.smem = std::max(p.smem, cluster_smem(pk[i], c, cached));
      const void* fn = (const void*)cluster_kernel(c, cached);
      if (p.smem > limit) continue;
      if (c > 8 && cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
                     cudaSuccess) {
        (void)cudaGetLastError();
        continue;
      }
      allow_max_dynamic_smem(fn);
      cudaLaunchConfig_t cfg{};
      cudaLaunchAttribute attr[1];
      p.configure(cfg, attr, (int)ids.size(), nullptr);
      int active = 0;
      if (cudaOccupancyMaxActiveClusters(&active, fn, &cfg) != cudaSuccess || active < 1) {
        (void)cudaGetLastError();
        continue;
      }
      const double waves = std::ceil((double)ids.size() / std::max(1.0, active * share));
      const double us    = waves * ((cached ? 2.3 : 3.0) + 0.03 * c + (c > 1 ? entries * 5e-5 : 0.0) +
                                 nnz * (cached ? 2.2e-4 : 3.5e-4) / c);
      if (best.smem == 0 || us < best_us) {
        best    = p;
        best_us = us;
      }
    }
  return best;
}

// Streams beside `s` for launches that may run at the same time: each begins after the work that is in
// s when it is taken, and join() makes s wait for all of them.
class side_streams {
 public:
  explicit side_streams(cudaStream_t s) : s_(s) {}
  side_streams(const side_streams&)            = delete;
  side_streams& operator=(const side_streams&) = delete;
  ~side_streams()
  {
    for (auto& l : lanes_) {
      cudaStreamSynchronize(l.stream);  // after an error too: the caller's buffers are freed in s
      cudaStreamDestroy(l.stream);
      cudaEventDestroy(l.event);
    }
  }
  cudaStream_t take()
  {
    lane l{};
    B200_CUDA_CHECK(cudaEventCreateWithFlags(&l.event, cudaEventDisableTiming));
    const cudaError_t e = cudaStreamCreateWithFlags(&l.stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) cudaEventDestroy(l.event);
    B200_CUDA_CHECK(e);
    lanes_.push_back(l);
    B200_CUDA_CHECK(cudaEventRecord(l.event, s_));
    B200_CUDA_CHECK(cudaStreamWaitEvent(l.stream, l.event, 0));
    return l.stream;
  }
  void join()
  {
    for (auto& l : lanes_) {
      B200_CUDA_CHECK(cudaEventRecord(l.event, l.stream));
      B200_CUDA_CHECK(cudaStreamWaitEvent(s_, l.event, 0));
    }
  }

 private:
  struct lane {
    cudaStream_t stream;
    cudaEvent_t event;
  };
  cudaStream_t s_;
  std::vector<lane> lanes_;
};

// Systems of like size, launched together: those whose shares of the operators fit in the shared memory
// of the same number of blocks (the last class: of no number).  A large system so neither takes
// the cache from small ones nor gives them its cluster.
struct size_class {
  std::vector<int> ids;
  cluster_plan plan;
};
constexpr int kClassBlocks[] = {1, 2, 4, 8, 16};
constexpr int kPortableBlocks = 8;  // the largest cluster that every launch may have
int class_of(const packed& q, size_t limit)
{
  int k = 0;
  for (const int c : kClassBlocks) {
    if (cluster_smem(q, c, true) <= limit) break;
    ++k;
  }
  return k;
}

}  // namespace

std::vector<lsqr_result> lsqr_solve_batch(const std::vector<const lsqr_problem*>& ps,
                                          cudaStream_t s, double tol, int max_iter)
{
  const int count = (int)ps.size();
  std::vector<lsqr_result> res(count);
  std::vector<packed> pk(count);
  for (int i = 0; i < count; ++i) {
    const lsqr_problem& p = *ps[i];
    if ((int)p.off.size() != p.rows + 1 || (int)p.b.size() != p.rows || p.rows < 0 || p.cols < 0 ||
        (int64_t)p.idx.size() < p.off[p.rows] || (int64_t)p.val.size() < p.off[p.rows])
      throw std::invalid_argument("lsqr: malformed problem");
    for (int64_t e = 0; e < p.off[p.rows]; ++e)
      if (p.idx[e] < 0 || p.idx[e] >= p.cols) throw std::invalid_argument("lsqr: column out of range");
  }
  parallel_for(count, [&](int i) { pack(*ps[i], pk[i]); });
  trace("lsqr: packing");

  // Systems with work go to the device: those whose vectors fit in a cluster's blocks, and the rest.
  const size_t limit = max_dynamic_smem((const void*)cluster_kernel(16, true));
  std::vector<size_class> classes(std::size(kClassBlocks) + 1);
  std::vector<int> glob_ids;
  for (int i = 0; i < count; ++i) {
    res[i].z.assign(ps[i]->cols, 0.0);
    if (pk[i].rows == 0 || pk[i].cols == 0) continue;
    if (cluster_smem(pk[i], kPortableBlocks, false) <= limit)
      classes[class_of(pk[i], limit)].ids.push_back(i);
    else
      glob_ids.push_back(i);
  }
  std::vector<int> order;              // systems as they are launched
  std::vector<int> blocks(count, 1);   // of the cluster of each
  // A class's share of the GPU is its share of the work: iterations grow with the rows and columns.
  std::vector<double> work(classes.size(), 0.0);
  for (size_t k = 0; k < classes.size(); ++k)
    for (int i : classes[k].ids)
      work[k] += (double)(pk[i].rows + pk[i].cols) *
                 (2.3 + 2.2e-4 * (double)(pk[i].p_val.size() + pk[i].q_val.size()));
  const double all = std::accumulate(work.begin(), work.end(), 0.0);
  for (auto& k : classes) {
    k.plan = plan_clusters(pk, k.ids, limit, work[&k - classes.data()] / std::max(all, 1e-300));
    if (k.plan.smem == 0) {
      glob_ids.insert(glob_ids.end(), k.ids.begin(), k.ids.end());
      k.ids.clear();
    }
    for (int i : k.ids) blocks[i] = k.plan.blocks;
    order.insert(order.end(), k.ids.begin(), k.ids.end());
  }
  size_t scratch_doubles = 0;
  for (int i : glob_ids) scratch_doubles += (size_t)pk[i].rows + 3 * (size_t)pk[i].cols;
  order.insert(order.end(), glob_ids.begin(), glob_ids.end());
  if (order.empty()) return res;

  // One upload of every array: offsets, indices, values, right-hand sides; outputs z.
  size_t n_off = 0, n_idx = 0, n_val = 0, n_b = 0, n_z = 0;
  for (int i : order) {
    n_off += pk[i].p_slice.size() + pk[i].q_slice.size();
    n_idx += pk[i].p_idx.size() + pk[i].q_idx.size();
    n_val += pk[i].p_val.size() + pk[i].q_val.size();
    n_b += pk[i].rows;
    n_z += pk[i].cols;
  }
  std::vector<int64_t> h_off;
  std::vector<int> h_idx;
  std::vector<double> h_val, h_b;
  h_off.reserve(n_off);
  h_idx.reserve(n_idx);
  h_val.reserve(n_val + n_b);
  h_b.reserve(n_b);
  struct where {
    size_t p_off, q_off, p_idx, q_idx, p_val, q_val, b, z, scratch;
  };
  std::vector<where> at(count);
  size_t z_pos = 0, scratch_pos = 0;
  for (int i : order) {
    const packed& q = pk[i];
    where w{};
    w.p_off = h_off.size();
    h_off.insert(h_off.end(), q.p_slice.begin(), q.p_slice.end());
    w.q_off = h_off.size();
    h_off.insert(h_off.end(), q.q_slice.begin(), q.q_slice.end());
    w.p_idx = h_idx.size();
    h_idx.insert(h_idx.end(), q.p_idx.begin(), q.p_idx.end());
    w.q_idx = h_idx.size();
    h_idx.insert(h_idx.end(), q.q_idx.begin(), q.q_idx.end());
    w.p_val = h_val.size();
    h_val.insert(h_val.end(), q.p_val.begin(), q.p_val.end());
    w.q_val = h_val.size();
    h_val.insert(h_val.end(), q.q_val.begin(), q.q_val.end());
    w.b = h_b.size();
    h_b.insert(h_b.end(), q.b.begin(), q.b.end());
    w.z = z_pos;
    z_pos += q.cols;
    w.scratch = scratch_pos;
    if (std::find(glob_ids.begin(), glob_ids.end(), i) != glob_ids.end())
      scratch_pos += (size_t)q.rows + 3 * (size_t)q.cols;
    at[i] = w;
  }
  alloc_scope scope(s);
  dbuf<int64_t> d_off(std::max<size_t>(h_off.size(), 1));
  dbuf<int> d_idx(std::max<size_t>(h_idx.size(), 1));
  dbuf<double> d_val(std::max<size_t>(h_val.size(), 1)), d_b(std::max<size_t>(h_b.size(), 1));
  dbuf<double> d_z(std::max<size_t>(n_z, 1)), d_scratch(std::max<size_t>(scratch_doubles, 1));
  d_off.upload(h_off.data(), h_off.size(), s);
  d_idx.upload(h_idx.data(), h_idx.size(), s);
  d_val.upload(h_val.data(), h_val.size(), s);
  d_b.upload(h_b.data(), h_b.size(), s);
  const int default_iter = max_iter;
  std::vector<lsqr_desc> h_desc;
  for (int i : order) {
    const packed& q = pk[i];
    const where& w  = at[i];
    lsqr_desc d{};
    d.rows     = q.rows;
    d.cols     = q.cols;
    d.slices_p = (int)q.p_slice.size() - 1;
    d.slices_q = (int)q.q_slice.size() - 1;
    d.p_slice  = d_off.data() + w.p_off;
    d.q_slice  = d_off.data() + w.q_off;
    d.p_idx    = d_idx.data() + w.p_idx;
    d.q_idx    = d_idx.data() + w.q_idx;
    d.p_val    = d_val.data() + w.p_val;
    d.q_val    = d_val.data() + w.q_val;
    d.b        = d_b.data() + w.b;
    d.z        = d_z.data() + w.z;
    d.scratch  = d_scratch.data() + w.scratch;
    d.share_p  = most_elements(q.p_slice, blocks[i]);
    d.share_q  = most_elements(q.q_slice, blocks[i]);
    d.tol      = tol;
    d.max_iter = default_iter > 0 ? default_iter
                                  : (int)std::min<long long>(200000, 20LL * (q.rows + q.cols));
    h_desc.push_back(d);
  }
  dbuf<lsqr_desc> d_desc(h_desc.size());
  dbuf<lsqr_out> d_out(h_desc.size());
  d_desc.upload(h_desc.data(), h_desc.size(), s);
  trace_sync(s, "lsqr: upload");
  // Launched from the largest systems down, which take the longest; the last launch is in s itself.
  side_streams side(s);
  size_t first = order.size();
  int launches = !glob_ids.empty();
  for (const auto& k : classes) launches += !k.ids.empty();
  auto next = [&](size_t systems) {
    first -= systems;
    return --launches > 0 ? side.take() : s;
  };
  if (!glob_ids.empty()) {
    const cudaStream_t ls = next(glob_ids.size());
    lsqr_kernel<<<(int)glob_ids.size(), kLsqrThreads, 0, ls>>>(d_desc.data() + first,
                                                               d_out.data() + first);
    B200_LAUNCH_CHECK();
  }
  for (auto k = classes.rbegin(); k != classes.rend(); ++k) {
    if (k->ids.empty()) continue;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    k->plan.configure(cfg, attr, (int)k->ids.size(), next(k->ids.size()));
    B200_CUDA_CHECK(cudaLaunchKernelEx(&cfg, cluster_kernel(k->plan.blocks, k->plan.cached),
                                       (const lsqr_desc*)d_desc.data() + first,
                                       d_out.data() + first));
  }
  side.join();
  trace_sync(s, "lsqr: kernel");
  std::vector<double> h_z(n_z);
  std::vector<lsqr_out> h_out(h_desc.size());
  d_z.download(h_z.data(), n_z, s);
  d_out.download(h_out.data(), h_out.size(), s);
  B200_CUDA_CHECK(cudaStreamSynchronize(s));
  for (size_t k = 0; k < order.size(); ++k) {
    const int i     = order[k];
    const packed& q = pk[i];
    lsqr_result& r  = res[i];
    for (int j = 0; j < q.cols; ++j) {
      const int c = q.perm_q[j];
      r.z[c]      = h_z[at[i].z + j] * q.dc[c];
    }
    r.iterations = h_out[k].iterations;
    r.flag       = h_out[k].flag;
    if (r.flag == kLsqrFailed)
      throw cuda_error("lsqr: an exchange between blocks passed its poll limit");
    r.rnorm      = h_out[k].rnorm;
    r.arnorm     = h_out[k].arnorm;
  }
  return res;
}

}  // namespace cuopt_b200
