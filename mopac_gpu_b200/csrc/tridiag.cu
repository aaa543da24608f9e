// Unblocked Householder tridiagonalisation with the matrix resident in shared
// memory, one message per column.
//
// Both kernels below run the textbook reduction: for each column j the
// reflector v_j, y = A v_j, w_j = tau (y - (tau/2) (y.v) v), and the rank-2
// update A -= v w^T + w v^T.  The columns of A are dealt cyclically to the
// CTAs, whole columns each, so y(c) = A(:, c).v needs no sum across CTAs, and
// the update of step j - 1 is applied in the same pass over the CTA's columns
// that forms y of step j.  That pass also hands on A(j+1, c), so one exchange
// of the pairs (y(c), A(j+1, c)) gives every CTA, by symmetry, both the vector
// it needs for w_j and the next column before its update; every CTA then forms
// w_j, the updated column and the next reflector itself, in the same order of
// operations, and no second exchange (for a norm or a reflector) is needed.
//
//   tridiag_cluster  one thread-block cluster, the matrix in registers, a
//                    record sent to each CTA's shared memory with st.async,
//                    which counts it on that CTA's mbarrier: no barrier across
//                    the cluster inside the loop.  Orders up to 608 (5 columns
//                    a warp, 128 warps).
//   tridiag_grid     one CTA per SM, the matrix in shared memory, the exchange
//                    through L2: a record is valid once it differs from a NaN
//                    sentinel, so it needs no flag.  Orders up to 2048 (14
//                    columns a CTA).
//
// Both are bound by the chain of a column: the exchange, two block sums, a
// square root and a division, then the pass (FP64 multiply-adds).  Measured on
// one B200, us per column: 1.1 at order 38 (1 CTA), 1.3 at 144 (4), 1.6 at 320
// (8), 2.3 at 600 (16); grid 3.8 at 700, 4.6 at 1501, 5.4 at 2048; panels of 32
// columns with two grid barriers a column took 19 at order 600 and 14 to 18 at
// 1501 to 3072.  In one cluster an exchange costs 300 to 700 cycles, over the
// whole chip 2700 (an L2 round trip each way), which is why a cluster takes
// what fits: at order 609 the grid needs 2.4 ms for what the cluster does at
// 608 in 1.4.
#include <cooperative_groups.h>

#include <map>
#include <mutex>

#include "mb_common.cuh"

namespace cg = cooperative_groups;

namespace {

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Reflector of a column with alpha = its first element and sig = the sum of
// squares of the others: beta, tau and the scale of the tail (dlarfg without
// its rescaling loop).
__device__ __forceinline__ void reflector(double alpha, double sig, double& beta, double& tau, double& scal) {
  if (sig == 0.0) {
    beta = alpha;
    tau = 0.0;
    scal = 0.0;
  } else {
    beta = -copysign(sqrt(alpha * alpha + sig), alpha);
    tau = (beta - alpha) / beta;
    scal = 1.0 / (alpha - beta);
  }
}

// ---------------------------------------------------------------- cluster
constexpr int CW = 8;          // warps per CTA
constexpr int CT = 32 * CW;
constexpr unsigned long long kWaitNs = 2000000000ull;

struct ClusterArgs {
  int n, perturb;
  double* pk;    // packed lower triangle; its diagonal receives the perturbation
  double* vall;  // n x n, column j = reflector j (zero down to row j, 1 at j + 1)
  double* d;
  double* e;
  double* tau;
  int* status;
};

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned peer_addr(unsigned local, int rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
// A record to a CTA of the cluster; it counts 16 bytes on that CTA's barrier.
__device__ __forceinline__ void send_record(unsigned dst, unsigned bar, double x, double y) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(dst),
               "d"(x), "d"(y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ bool records_arrived(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Sum of the CW per-warp partials.
__device__ __forceinline__ double sum_partials(const double2* s) {
  const double2 a = s[0], b = s[1], c = s[2], d = s[3];
  return ((a.x + a.y) + (b.x + b.y)) + ((c.x + c.y) + (d.x + d.y));
}

// N sums over a warp at once (N a power of two): each step halves the values
// a lane holds; afterwards lane l holds the whole sum of value
// l / (32 / N).
template <int N>
__device__ __forceinline__ double warp_sums(double (&x)[N], int lane) {
  int o = 16;
#pragma unroll
  for (int h = N / 2; h >= 1; h >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double send = up ? x[i] : x[i + h];
      const double keep = up ? x[i + h] : x[i];
      x[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  for (; o >= 1; o >>= 1) x[0] += __shfl_xor_sync(0xffffffffu, x[0], o);
  return x[0];
}

// The pass over columns I0 .. C - 1 of a warp: pending update, dot with the
// new reflector; element j + 1 of each column, in block kn, goes to an.
template <int K, int C, int I0>
__device__ __forceinline__ void column_pass(double (&A)[C][K], double (&acc)[8], double* an, const double2 (&q)[C],
                                            const double2* vw, const double* vn, int lane, int kn, int jl) {
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (k < kn) continue;
    const double2 r = vw[lane + 32 * k];
    const double u = vn[lane + 32 * k];
#pragma unroll
    for (int i = I0; i < C; ++i) {
      const double x = fma(-r.y, q[i].x, fma(-r.x, q[i].y, A[i][k]));
      A[i][k] = x;
      acc[i] = fma(x, u, acc[i]);
    }
    if (k == kn && lane == jl) {
#pragma unroll
      for (int i = I0; i < C; ++i) an[i] = A[i][k];
    }
  }
}

// K: blocks of 32 rows; C: columns of a warp, which keeps them in registers
// (lane l rows l, l + 32, ...).  Column c belongs to CTA c % cs; warp w of CTA
// r owns columns w cs + r + 8 cs i.  Threads share the rows of v, w and the
// next column.  ONE: a cluster of one CTA, the records stay in its own memory.
template <int K, int C, bool ONE>
__global__ void __launch_bounds__(CT, 1) tridiag_cluster(ClusterArgs p) {
  constexpr int LD = 32 * K, R = (LD + CT - 1) / CT;
  __shared__ double2 xy[2][LD];    // records (y(c), A(j + 1, c)) of two exchanges
  __shared__ double2 vw[LD];       // (v, w) of the pending update
  __shared__ double vn[LD];        // the new reflector
  __shared__ double2 s_red[2][CW / 2];
  __shared__ double s_alpha, s_an[CW][8];
  __shared__ __align__(8) unsigned long long bar[2];
  __shared__ int s_fail;
  const int cs = ONE ? 1 : (int)cg::this_cluster().num_blocks();
  const int rank = ONE ? 0 : (int)cg::this_cluster().block_rank();
  const int n = p.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c0 = warp * cs + rank, cstep = CW * cs;
  // this CTA's last column: it leaves the loop after that
  const int last = rank < n ? n - 1 - (n - 1 - rank) % cs : -1;
  double A[C][K];
#pragma unroll
  for (int i = 0; i < C; ++i)
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int c = c0 + cstep * i, r = lane + 32 * k;
      double x = 0.0;
      if (c < n && r < n) {
        const long long q = r >= c ? mb_tri(r, c) : mb_tri(c, r);
        x = p.pk[q];
        if (r == c && p.perturb) {
          x = DADD(x, DMUL((double)(r + 1), 1.0e-10));
          p.pk[q] = x;
        }
      }
      A[i][k] = x;
    }
  for (int r = tid; r < LD; r += CT) xy[0][r] = xy[1][r] = make_double2(0.0, 0.0);
  auto arm = [&](int t) {  // exchange t brings columns t .. n - 1
    if (t < n)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&bar[t & 1])),
                   "r"(16 * (n - t))
                   : "memory");
  };
  if (tid == 0) {
    s_fail = 0;
    if (!ONE) {
      for (int q = 0; q < 2; ++q)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bar[q])) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      arm(0);
      arm(1);
    }
  }
  __syncthreads();
  // After warp_sums four lanes hold each column's y: lane 4 i + u sends column
  // i's record to CTAs u, u + 4, ...
  const int ci = lane >> 2, cc = c0 + cstep * ci;
  unsigned to[4] = {}, tobar[4] = {};
  if (!ONE) {
    cluster_barrier();  // every CTA runs, with its barriers armed
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int q = (lane & 3) + 4 * u;
      to[u] = peer_addr(smem_addr(xy), q < cs ? q : 0);
      tobar[u] = peer_addr(smem_addr(bar), q < cs ? q : 0);
    }
  }
  auto send = [&](int t, double y, double a) {
    if (ONE) {
      if ((lane & 3) == 0) xy[t & 1][cc] = make_double2(y, a);
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if ((lane & 3) + 4 * u < cs)
          send_record(to[u] + (unsigned)sizeof(double2) * ((t & 1) * LD + cc), tobar[u] + 8u * (t & 1), y, a);
    }
  };
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < C; ++i) s_an[warp][i] = A[i][0];
  }
  __syncwarp();
  if (ci < C && cc < n) send(0, 0.0, s_an[warp][ci]);

  double v[R], tau = 0.0;
#pragma unroll
  for (int q = 0; q < R; ++q) v[q] = 0.0;
  for (int j = 0; j < last || j == n - 1; ++j) {
    if (j == n - 1 && last != n - 1) break;
    if (ONE) {
      __syncthreads();
    } else {
      const unsigned b = smem_addr(&bar[j & 1]), par = (unsigned)(j >> 1) & 1u;
      if (!records_arrived(b, par)) {
        unsigned long long t0 = 0;
        for (unsigned it = 1; !records_arrived(b, par); ++it)
          if ((it & 255u) == 0) {
            unsigned long long now;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (t0 == 0) t0 = now;
            if (now - t0 > kWaitNs) {
              s_fail = 1;
              break;
            }
          }
      }
      if (tid == 0) arm(j + 2);
    }
    const double2* in = xy[j & 1];
    double w[R], a[R], pv = 0.0;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int r = tid + CT * q;
      w[q] = a[q] = 0.0;
      if (r >= j && r < n) {
        const double2 x = in[r];
        w[q] = x.x;
        a[q] = x.y;
      }
      pv = fma(w[q], v[q], pv);
    }
    const double yj = in[j].x;
    pv = warp_sum(pv);
    if (lane == 0) ((double*)s_red[0])[warp] = pv;
    __syncthreads();
    if (!ONE && s_fail) {
      if (tid == 0) atomicCAS(p.status, MB_OK, MB_ERR_TIMEOUT);
      break;
    }
    pv = sum_partials(s_red[0]);
    const double hw = -0.5 * tau * pv;
    const double wj = tau * (yj + hw);  // w(j): v(j) = 1
    // d, e, tau and the reflector leave through the CTA of column j + 1, which
    // is still in the loop
    const bool store = rank == (j + 1 < n ? j + 1 : j) % cs;
    double sig = 0.0;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int r = tid + CT * q;
      w[q] = tau * fma(hw, v[q], w[q]);
      const double x = fma(-v[q], wj, a[q]) - w[q];  // column j with the pending update
      a[q] = x;
      if (r < LD) vw[r] = make_double2(v[q], w[q]);
      if (r == j && store) p.d[j] = x;
      if (r == j + 1) s_alpha = x;
      if (r >= j + 2) sig = fma(x, x, sig);
    }
    if (j == n - 1) break;
    sig = warp_sum(sig);
    if (lane == 0) ((double*)s_red[1])[warp] = sig;
    __syncthreads();
    double beta, taun, scal;
    reflector(s_alpha, sum_partials(s_red[1]), beta, taun, scal);
    if (store && tid == 0) {
      p.e[j] = beta;
      p.tau[j] = taun;
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int r = tid + CT * q;
      const double x = r == j + 1 ? 1.0 : (r > j + 1 ? a[q] * scal : 0.0);
      if (r < LD) vn[r] = x;
      if (store && r < n) p.vall[(long long)j * n + r] = x;
      v[q] = x;
    }
    tau = taun;
    __syncthreads();
    // columns retire in the order i = 0, 1, ...: the first half is passed over
    // once it is done
    const int kn = (j + 1) >> 5, jl = (j + 1) & 31;
    double2 q[C];
    double acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.0;
#pragma unroll
    for (int i = 0; i < C; ++i) {
      const int c = c0 + cstep * i;
      q[i] = vw[c < LD ? c : 0];
    }
    if (c0 + cstep * (C / 2 - 1) > j) column_pass<K, C, 0>(A, acc, s_an[warp], q, vw, vn, lane, kn, jl);
    else if (c0 + cstep * (C - 1) > j) column_pass<K, C, C / 2>(A, acc, s_an[warp], q, vw, vn, lane, kn, jl);
    __syncwarp();
    const double y = warp_sums<8>(acc, lane);
    if (ci < C && cc > j && cc < n) send(j + 1, y, s_an[warp][ci]);
  }
  if (!ONE) cluster_barrier();  // no CTA leaves while a record may be on its way to it
}

// ------------------------------------------------------------------- grid
constexpr int GT = 512;            // threads per CTA
constexpr int GW = GT / 32;
constexpr int GC = 14;             // columns per CTA at most
constexpr unsigned long long kEmpty = 0xFFFFFFFFFFFFFFFFull;  // a NaN no arithmetic produces

struct GridArgs {
  int m;            // order of the trailing matrix
  const double* a;  // its (0, 0), column-major, leading dimension lda
  long long lda;
  double* vall;     // its reflectors, same leading dimension
  double* d;
  double* e;
  double* tau;
  double2* xy;      // four buffers of m records, all bytes 0xFF at launch
  int* abort_flag;  // 0 at launch
  int* status;
};

__device__ __forceinline__ void ld_record(const double2* p, unsigned long long& x, unsigned long long& y) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_record(double2* p, unsigned long long x, unsigned long long y) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(x), "l"(y) : "memory");
}
__device__ __forceinline__ unsigned long long record_bits(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return b == kEmpty ? 0x7FF8000000000000ull : b;
}

// Buffers: exchange t uses buffer t % 4.  A CTA leaves once its last column
// is done, so every CTA that reads exchange t - 2 publishes in exchange t - 1,
// after that read.  A CTA that holds all of exchange t - 1 may therefore, after
// publishing exchange t, empty its own records of exchange t - 2 for exchange
// t + 2; the fence orders that before its records of exchange t + 1, which
// every reader of exchange t + 2 has seen.
// Pending update and dot with the new reflector u of the thread's rows, blocks
// Q0 and up, of the CTA's columns first .. nloc - 1; the next column's rows
// are on their way while one is updated.
template <int GR, int NC, int Q0>
__device__ __forceinline__ void grid_pass(double* A, const double2* s_vw, int first, int nloc, const double (&v)[GR],
                                          const double (&w)[GR], const double (&u)[GR], double (&acc)[NC]) {
  constexpr int LD = GR * GT;
  double x[GR];
#pragma unroll
  for (int q = Q0; q < GR; ++q) x[q] = A[first * LD + GT * q];
#pragma unroll
  for (int lc = 0; lc < NC; ++lc) {
    if (lc < first || lc >= nloc) continue;
    double* cur = A + lc * LD;
    const double* nxt = lc + 1 < nloc ? cur + LD : cur;
    const double2 s = s_vw[lc];
    double y[GR];
#pragma unroll
    for (int q = Q0; q < GR; ++q) y[q] = nxt[GT * q];
#pragma unroll
    for (int q = Q0; q < GR; ++q) {
      const double t = fma(-w[q], s.x, fma(-v[q], s.y, x[q]));
      acc[lc] = fma(t, u[q], acc[lc]);
      cur[GT * q] = t;
      x[q] = y[q];
    }
  }
}

// GR: rows per thread, GR * GT >= m; NC >= the CTA's columns, 8 or 16; the columns in shared memory are padded to
// that many rows with zeros, which the reduction leaves zero.
template <int GR, int NC>
__global__ void __launch_bounds__(GT, 1) tridiag_grid(GridArgs p) {
  extern __shared__ double gAs[];
  __shared__ double2 s_vw[GC];
  __shared__ double s_red[2][GW], s_part[GW][17];
  __shared__ double s_yj, s_alpha;
  __shared__ int s_fail;
  constexpr int LD = GR * GT;
  const int m = p.m, G = gridDim.x, b = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nloc = (m - b + G - 1) / G;  // G <= m
  const int last = b + G * (nloc - 1);
  if (tid == 0) s_fail = 0;
  for (int lc = 0; lc < nloc; ++lc)
    for (int r = tid; r < LD; r += GT) gAs[lc * LD + r] = r < m ? p.a[(long long)(b + G * lc) * p.lda + r] : 0.0;
  __syncthreads();
  if (tid < nloc) st_record(p.xy + b + G * tid, record_bits(0.0), record_bits(gAs[tid * LD]));

  double v[GR], tau = 0.0;
  int slot[GR];  // the CTA's column of the thread's row, if it is one
#pragma unroll
  for (int q = 0; q < GR; ++q) {
    v[q] = 0.0;
    const int r = tid + GT * q;
    slot[q] = r >= b && r < m && (r - b) % G == 0 ? (r - b) / G : -1;
  }
  for (int j = 0; j < last || j == m - 1; ++j) {
    // exchange j: (y(r), A(j, r)) of the thread's rows r >= j
    const double2* in = p.xy + (long long)(j & 3) * m;
    double w[GR], a[GR], pv = 0.0;
    {
      unsigned pend = 0;
#pragma unroll
      for (int q = 0; q < GR; ++q) {
        const int r = tid + GT * q;
        w[q] = a[q] = 0.0;
        if (r >= j && r < m) pend |= 1u << q;
      }
      unsigned spins = 0;
      unsigned long long t0 = 0;
      while (pend) {
        unsigned long long x[GR], y[GR];
#pragma unroll
        for (int q = 0; q < GR; ++q) {
          x[q] = y[q] = kEmpty;
          if (pend & (1u << q)) ld_record(in + tid + GT * q, x[q], y[q]);
        }
#pragma unroll
        for (int q = 0; q < GR; ++q)
          if (x[q] != kEmpty && y[q] != kEmpty) {
            w[q] = __longlong_as_double((long long)x[q]);
            a[q] = __longlong_as_double((long long)y[q]);
            pend &= ~(1u << q);
          }
        if (pend && (++spins & 1023u) == 0) {
          unsigned long long now;
          asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
          if (t0 == 0) t0 = now;
          int stop;
          asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(stop) : "l"(p.abort_flag) : "memory");
          if (stop != 0 || now - t0 > kWaitNs) {
            atomicExch(p.abort_flag, 1);
            s_fail = 1;
            break;
          }
        }
      }
    }
#pragma unroll
    for (int q = 0; q < GR; ++q) {
      pv = fma(w[q], v[q], pv);
      if (tid + GT * q == j) s_yj = w[q];
    }
    pv = warp_sum(pv);
    if (lane == 0) s_red[0][warp] = pv;
    __syncthreads();
    if (s_fail) {
      if (tid == 0) atomicCAS(p.status, MB_OK, MB_ERR_TIMEOUT);
      return;
    }
    pv = s_red[0][lane & (GW - 1)];
#pragma unroll
    for (int o = GW / 2; o > 0; o >>= 1) pv += __shfl_xor_sync(0xffffffffu, pv, o);
    const double hw = -0.5 * tau * pv;
    const double wj = tau * (s_yj + hw);
    const bool store = b == (j + 1 < m ? j + 1 : j) % G;  // a CTA that is still in the loop
    double sig = 0.0;
#pragma unroll
    for (int q = 0; q < GR; ++q) {
      const int r = tid + GT * q;
      w[q] = tau * fma(hw, v[q], w[q]);
      const double x = fma(-v[q], wj, a[q]) - w[q];
      a[q] = x;
      if (r == j && store) p.d[j] = x;
      if (r == j + 1) s_alpha = x;
      if (r >= j + 2) sig = fma(x, x, sig);
      if (slot[q] >= 0) s_vw[slot[q]] = make_double2(v[q], w[q]);
    }
    if (j == m - 1) break;
    sig = warp_sum(sig);
    if (lane == 0) s_red[1][warp] = sig;
    __syncthreads();
    sig = s_red[1][lane & (GW - 1)];
#pragma unroll
    for (int o = GW / 2; o > 0; o >>= 1) sig += __shfl_xor_sync(0xffffffffu, sig, o);
    double beta, taun, scal;
    reflector(s_alpha, sig, beta, taun, scal);
    if (store && tid == 0) {
      p.e[j] = beta;
      p.tau[j] = taun;
    }
#pragma unroll
    for (int q = 0; q < GR; ++q) {
      const int r = tid + GT * q;
      a[q] = r == j + 1 ? 1.0 : (r > j + 1 ? a[q] * scal : 0.0);
      if (store && r < m) p.vall[(long long)j * p.lda + r] = a[q];
    }
    // the pass over the CTA's columns c > j; blocks below row j + 1 hold
    // finished rows only
    double acc[NC];
#pragma unroll
    for (int lc = 0; lc < NC; ++lc) acc[lc] = 0.0;
    const int first = j + 1 <= b ? 0 : (j + 1 - b + G - 1) / G;
    const int q0 = (j + 1) / GT;
    if (q0 == 0) grid_pass<GR, NC, 0>(gAs + tid, s_vw, first, nloc, v, w, a, acc);
    else if (GR > 1 && q0 == 1) grid_pass<GR, NC, 1>(gAs + tid, s_vw, first, nloc, v, w, a, acc);
    else if (GR > 2 && q0 == 2) grid_pass<GR, NC, 2>(gAs + tid, s_vw, first, nloc, v, w, a, acc);
    else if (GR > 3 && q0 == 3) grid_pass<GR, NC, 3>(gAs + tid, s_vw, first, nloc, v, w, a, acc);
    {
      const double y = warp_sums<NC>(acc, lane);
      if (lane % (32 / NC) == 0) s_part[warp][lane / (32 / NC)] = y;
    }
    __syncthreads();
    if (warp >= first && warp < nloc) {
      double y = s_part[lane & (GW - 1)][warp];
#pragma unroll
      for (int o = GW / 2; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
      if (lane == 0) {
        const int c = b + G * warp, t = j + 1;
        st_record(p.xy + (long long)(t & 3) * m + c, record_bits(y), record_bits(gAs[warp * LD + j + 1]));
        st_record(p.xy + (long long)((t + 2) & 3) * m + c, kEmpty, kEmpty);
      }
    }
    __threadfence();  // also between the reads of exchange t - 1 and of t
#pragma unroll
    for (int q = 0; q < GR; ++q) v[q] = a[q];
    tau = taun;
  }
}

}  // namespace

// Shared memory of a CTA of the grid kernel; its static part is below 4 KB.
static const size_t kMaxSmem = 232448;

// Orders the cluster kernel takes on a device that can (or cannot) hold a cluster of
// 16 CTAs, which is beyond the portable size of 8.
extern "C" int mb_tridiag_cluster_orders(int clusters16) { return clusters16 > 0 ? 608 : 320; }

// The same on the current device; asked once per device.
extern "C" int mb_tridiag_cluster_max(void) {
  static std::mutex mu;
  static std::map<int, int> known;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return mb_tridiag_cluster_orders(0);
  std::lock_guard<std::mutex> lock(mu);
  const auto it = known.find(dev);
  if (it != known.end()) return it->second;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(16);
  cfg.blockDim = dim3(CT);
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 16;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const void* fn = (const void*)tridiag_cluster<19, 5, false>;
  int count = 0;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&count, fn, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    count = 0;
  }
  return known[dev] = mb_tridiag_cluster_orders(count);
}

extern "C" int mb_tridiag_cluster(int n, double* pk, int perturb, double* vall, double* d, double* e, double* tau,
                                  int* status, cudaStream_t stream) {
  if (n < 2 || n > mb_tridiag_cluster_max()) return mb_set_error(MB_ERR_ARG, "mb_tridiag_cluster: order out of range");
  // 8 warps a CTA, each with C columns: 64 = 8 x 8, 160 = 4 x 8 x 5, 320 = 8 x 8 x 5, 608 <= 16 x 8 x 5
  const int cs = n <= 64 ? 1 : n <= 160 ? 4 : n <= 320 ? 8 : 16;
  void* fn = n <= 64 ? (void*)tridiag_cluster<2, 8, true>
             : n <= 160 ? (void*)tridiag_cluster<5, 5, false>
             : n <= 320 ? (void*)tridiag_cluster<10, 5, false>
                        : (void*)tridiag_cluster<19, 5, false>;
  ClusterArgs a{n, perturb, pk, vall, d, e, tau, status};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs);
  cfg.blockDim = dim3(CT);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cs;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  void* args[] = {&a};
  MB_CUDA(cudaLaunchKernelExC(&cfg, fn, args));
  mb_count_launch();
  return MB_OK;
}

// Rows per thread and shared memory of the grid kernel at order m on ctas CTAs;
// 0 rows when it does not take that order.
static int grid_shape(int m, int ctas, size_t* smem) {
  const int gr = (m + GT - 1) / GT, nloc = (m + ctas - 1) / ctas;
  *smem = sizeof(double) * (size_t)nloc * gr * GT;
  return m >= 2 && gr <= 4 && nloc <= GC && *smem + 3072 <= kMaxSmem ? gr : 0;
}

// The largest order the grid kernel takes.
extern "C" int mb_tridiag_grid_max(int ctas) {
  size_t smem;
  int m = 4 * GT;
  while (m > 1 && !grid_shape(m, ctas, &smem)) --m;
  return m;
}

// Reduces the matrix a (order m, leading dimension lda, read only).  scratch:
// 64 m + 16 bytes, 16-byte aligned.
extern "C" int mb_tridiag_grid(int m, int ctas, const double* a, long long lda, double* vall, double* d, double* e,
                               double* tau, void* scratch, int* status, cudaStream_t stream) {
  if (m < 2 || ctas < 1) return mb_set_error(MB_ERR_ARG, "mb_tridiag_grid: order out of range");
  if (ctas > m) ctas = m;
  size_t smem;
  const int gr = grid_shape(m, ctas, &smem);
  if (gr == 0) return mb_set_error(MB_ERR_ARG, "mb_tridiag_grid: order out of range");
  void* const fns[2][4] = {{(void*)tridiag_grid<1, 8>, (void*)tridiag_grid<2, 8>, (void*)tridiag_grid<3, 8>,
                            (void*)tridiag_grid<4, 8>},
                           {(void*)tridiag_grid<1, 16>, (void*)tridiag_grid<2, 16>, (void*)tridiag_grid<3, 16>,
                            (void*)tridiag_grid<4, 16>}};
  void* fn = fns[(m + ctas - 1) / ctas > 8][gr - 1];
  MB_TRY(mb_smem_optin(fn, smem));
  GridArgs g;
  g.m = m;
  g.a = a;
  g.lda = lda;
  g.vall = vall;
  g.d = d;
  g.e = e;
  g.tau = tau;
  g.xy = (double2*)scratch;
  g.abort_flag = (int*)((char*)scratch + sizeof(double2) * 4 * (size_t)m);
  g.status = status;
  MB_CUDA(cudaMemsetAsync(g.xy, 0xFF, sizeof(double2) * 4 * (size_t)m, stream));
  MB_CUDA(cudaMemsetAsync(g.abort_flag, 0, sizeof(int), stream));
  void* args[] = {&g};
  MB_CUDA(cudaLaunchCooperativeKernel(fn, ctas, GT, args, smem, stream));
  mb_count_launch();
  return MB_OK;
}
