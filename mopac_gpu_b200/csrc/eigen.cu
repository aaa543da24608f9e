// Full symmetric eigensolver in FP64 on the device, replacing the LAPACK /
// cuSOLVER dsyevd call of eigenvectors_LAPACK (matrix/eigenvectors_LAPACK.F90
// :53-121, cuda_wrappers.cu:469-505).
//
//   1. i*1e-10 added to diagonal element i of the packed input (the
//      reference's parity-critical perturbation, eigenvectors_LAPACK.F90:53-55).
//   2. Householder tridiagonalisation.  Up to order 608 (320 on a device without
//      clusters of 16 CTAs) and up to 2048 the matrix stays in the registers of one
//      cluster or in the SMs' shared memory (tridiag.cu).  A larger one is first taken down to that size
//      in panels (eigen_panel.cu): a cooperative kernel forms 32 reflectors (two
//      grid barriers per column), and the trailing matrix gets the rank-64
//      update A -= V W^T + W V^T as FP64 GEMM.
//   3. Eigenvalues of the tridiagonal matrix by multisection on Sturm counts,
//      one warp per eigenvalue.
//   4. Eigenvectors of the tridiagonal matrix by inverse iteration with partial
//      pivoting; eigenvalues closer than 1e-8 * ||T|| form clusters whose
//      vectors are re-orthogonalised inside the iteration (one thread per
//      cluster, members in order).
//   5. Back-transformation C = Q Z: up to order 608 reflector by reflector with
//      the vectors in registers, above with the compact WY form of 64
//      reflectors, Z -= V (T (V^T Z)), as FP64 GEMMs (eigen_panel.cu).
// Eigenvalues ascend; eigenvectors are the columns of C.
//
// Whole eigensolve on the Fock matrix of a water lattice (ms, one B200, medians of
// nine in a caller's workspace), in brackets the blocked form of eigen_panel.cu on
// the same box: order 38 0.10 (0.57), 144 0.36 (2.1), 320 0.84 (4.6), 600 2.1 (9.0),
// 1026 6.4 (16.4), 1501 10.7 (25.7), 2048 17.1 (37.7), 3072 46.5 (69.5).
#include "eigen_ws.cuh"
#include "mb_common.cuh"

namespace {

// ---------------------------------------------------------------- bisection
// 1/q from the hardware's approximate reciprocal refined by two Newton steps,
// r <- r + r (1 - q r): about 1e-16 relative, cheaper than the IEEE division.
// |q| >= pivmin (a normal number) here, so flushing subnormals loses nothing.
// A Sturm count is exact for a matrix within a few ulps of T, so the
// eigenvalue bounds keep the bisection's accuracy.
__device__ __forceinline__ double recip_nr2(double q) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(q));
  double e = fma(-q, r, 1.0);
  r = fma(r, e, r);
  e = fma(-q, r, 1.0);
  return fma(r, e, r);
}

// Sturm count (eigenvalues below x) from the leading principal minors'
// three-term recurrence p_i = (d_i - x) p_(i-1) - e_(i-1)^2 p_(i-2): its
// dependent chain is one multiply-add per row, against a reciprocal and four
// for the quotients q_i = p_i / p_(i-1), and a change of sign from p_(i-1) to
// p_i is a negative q_i.  Eight rows at a time, from a pair scaled by a power
// of two to [1, 2); T has norm <= 1 here, so a row grows p at most threefold.
// A block in which some |p_i| falls below kSturmTiny (a chain of tiny
// couplings at one of its eigenvalues) is taken again by quotients, whose
// pivots are bounded below by pivmin.  de[i] = (d_i, e_(i-1)^2), followed by
// 2 SB records (2, 0): rows that keep the sign of p.
constexpr int SB = 8;
constexpr int kSturmTiny = 0x27100000;  // high word of 2^-398, about 1e-120
constexpr double kPivmin = 1.0e-290;

__device__ __forceinline__ int sturm_count(int n, const double2* __restrict__ de, double x) {
  double p1 = de[0].x - x, p0 = 1.0;
  if (fabs(p1) < kPivmin) p1 = -kPivmin;
  int cnt = p1 < 0.0;
  double2 nx[SB];  // the next block's rows
#pragma unroll
  for (int u = 0; u < SB; ++u) nx[u] = de[1 + u];
  for (int i0 = 1; i0 < n; i0 += SB) {
    double db[SB], eb[SB];
#pragma unroll
    for (int u = 0; u < SB; ++u) {
      db[u] = nx[u].x - x;
      eb[u] = nx[u].y;
      nx[u] = de[i0 + SB + u];
    }
    const int ex = max((__double2hiint(p0) >> 20) & 0x7ff, (__double2hiint(p1) >> 20) & 0x7ff);
    const double sc = __hiloint2double((2046 - ex) << 20, 0);
    p0 *= sc;
    p1 *= sc;
    const double s0 = p0, s1 = p1;
    int c = 0, least = 0x7fffffff;  // high words of |p| order as |p| does
#pragma unroll
    for (int u = 0; u < SB; ++u) {
      const double p2 = fma(db[u], p1, -(eb[u] * p0));
      c += (unsigned)(__double2hiint(p2) ^ __double2hiint(p1)) >> 31;
      least = min(least, __double2hiint(p2) & 0x7fffffff);
      p0 = p1;
      p1 = p2;
    }
    if (least < kSturmTiny) {
      double q = s1 / s0;
      if (fabs(q) < kPivmin) q = -kPivmin;
      c = 0;
      for (int u = 0; u < SB && i0 + u < n; ++u) {
        q = db[u] - eb[u] * recip_nr2(q);
        if (fabs(q) < kPivmin) q = -kPivmin;
        c += q < 0.0;
      }
      p0 = 1.0;
      p1 = q;  // the pair matters up to a factor only
    }
    cnt += c;
  }
  return cnt;
}

// T scaled by the power of two that brings its Gershgorin bound to (1/2, 1]
// (exact unless an element underflows next to the norm), as the records de
// and dv, and bnd = { lower bound, upper bound, unused, norm, 1 / scale }.
__global__ void tri_bounds(int n, const double* __restrict__ d, const double* __restrict__ e,
                           double2* __restrict__ de, double2* __restrict__ dv, double* __restrict__ bnd) {
  __shared__ double slo[1024], shi[1024];
  double lo = 1e300, hi = -1e300;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0);
    lo = fmin(lo, d[i] - r);
    hi = fmax(hi, d[i] + r);
  }
  slo[threadIdx.x] = lo; shi[threadIdx.x] = hi;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      slo[threadIdx.x] = fmin(slo[threadIdx.x], slo[threadIdx.x + s]);
      shi[threadIdx.x] = fmax(shi[threadIdx.x], shi[threadIdx.x + s]);
    }
    __syncthreads();
  }
  const double norm = fmax(fabs(slo[0]), fabs(shi[0]));
  // 2^-k with norm 2^-k in (1/2, 1]; k clamped so that 2^k and 2^-k are normal
  int k = 0;
  if (norm > 0.0 && norm < 1e300) frexp(norm, &k);
  k = max(-1000, min(1000, k));
  const double sc = ldexp(1.0, -k);
  if (threadIdx.x == 0) {
    const double tnorm = norm * sc;
    const double pad = 2.0 * 2.220446049250313e-16 * tnorm * n + 1e-300;
    bnd[0] = slo[0] * sc - pad;
    bnd[1] = shi[0] * sc + pad;
    bnd[2] = 0.0;
    bnd[3] = tnorm;
    bnd[4] = ldexp(1.0, k);
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double f = i > 0 ? e[i - 1] * sc : 0.0;
    de[i] = make_double2(d[i] * sc, f * f);
    dv[i] = make_double2(d[i] * sc, i < n - 1 ? e[i] * sc : 0.0);
  }
  if (threadIdx.x < 2 * SB) de[n + threadIdx.x] = make_double2(2.0, 0.0);
}

// One warp per eigenvalue: each pass the 32 lanes evaluate Sturm counts at 32
// interior points of the bracket, shrinking it 33-fold (about a dozen passes
// instead of ~60 bisection steps, with 32x the parallelism).  ws receives the
// eigenvalues of the scaled T, w those of T.
__global__ void bisect_kernel(int n, const double2* __restrict__ de, const double* __restrict__ bnd,
                              double* __restrict__ ws, double* __restrict__ w) {
  const int m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (m >= n) return;
  double lo = bnd[0], hi = bnd[1];
  const double eps = 2.220446049250313e-16;
  for (int it = 0; it < 64; ++it) {
    if (hi - lo <= 2.0 * eps * fmax(fabs(lo), fabs(hi)) + kPivmin) break;
    const double x = lo + (hi - lo) * ((double)(lane + 1) / 33.0);
    const int cnt = sturm_count(n, de, x);
    const unsigned above = __ballot_sync(0xffffffffu, cnt > m);  // lanes whose point lies above eigenvalue m
    double nlo = lo, nhi = hi;
    if (above == 0u) {
      nlo = __shfl_sync(0xffffffffu, x, 31);
    } else {
      const int first = __ffs(above) - 1;
      nhi = __shfl_sync(0xffffffffu, x, first);
      if (first > 0) nlo = __shfl_sync(0xffffffffu, x, first - 1);
    }
    if (!(nlo > lo) && !(nhi < hi)) break;  // no representable progress
    lo = nlo;
    hi = nhi;
  }
  if (lane == 0) {
    const double x = 0.5 * (lo + hi);
    ws[m] = x;
    w[m] = x * bnd[4];
  }
}

// --------------------------------------------------------- inverse iteration
// LU with partial pivoting of T - lam I for one vector per thread, every array
// with stride ld.  Row i of the factor: the reciprocal of the pivot, the two
// elements above it, the multiplier and whether rows i and i + 1 changed
// places; later solves of the same vector reuse it.
struct TriLu {
  double *rp, *u1, *u2, *l;
  unsigned char* sw;
  long long ld;
};

// Forward substitution of x (in place) with the stored factor, or (FACTOR)
// while forming it; x(i) * scale is what the sweep reads.  FACTOR reads the
// start vector from the generator state instead.  Every sweep fetches the
// operands of the next eight rows while eight pass through the dependent
// chain.  dv[i] = (d_i, e_i).
constexpr int TB = 8;

template <bool FACTOR>
__device__ __forceinline__ void tri_forward(int n, const double2* __restrict__ dv, double lam, double tiny,
                                            const TriLu& f, double* x, double scale, unsigned long long seed) {
  const long long ld = f.ld;
  unsigned long long s = seed;
  auto rnd = [&]() {
    s ^= s >> 31; s *= 0x94D049BB133111EBull; s ^= s >> 29;
    return ((double)(s >> 11) * (1.0 / 9007199254740992.0)) - 0.5;
  };
  double dd = 0.0, du = 0.0, sub = 0.0, xr;
  double2 tn[TB];
  double xn[TB], ln[TB];
  unsigned char wn[TB];
  auto fetch = [&](int i0) {
#pragma unroll
    for (int u = 0; u < TB; ++u) {
      const int i = min(i0 + u, n - 2);
      if (FACTOR) {
        tn[u] = dv[i + 1];
      } else {
        xn[u] = x[(long long)(i + 1) * ld];
        ln[u] = f.l[(long long)i * ld];
        wn[u] = f.sw[(long long)i * ld];
      }
    }
  };
  if (FACTOR) {
    const double2 t = dv[0];
    dd = t.x - lam;
    du = sub = n > 1 ? t.y : 0.0;
    xr = rnd();
  } else {
    xr = x[0] * scale;
  }
  if (n > 1) fetch(0);
  for (int i0 = 0; i0 < n - 1; i0 += TB) {
    double2 tb[TB];
    double xb[TB], lb[TB];
    unsigned char wb[TB];
#pragma unroll
    for (int u = 0; u < TB; ++u) {
      tb[u] = tn[u];
      xb[u] = xn[u] * scale;
      lb[u] = ln[u];
      wb[u] = wn[u];
    }
    if (i0 + TB < n - 1) fetch(i0 + TB);
#pragma unroll
    for (int u = 0; u < TB; ++u) {
      const int i = i0 + u;
      if (i < n - 1) {
        const long long o = (long long)i * ld;
        if (FACTOR) {
          const double dn = tb[u].x - lam, en = i + 1 < n - 1 ? tb[u].y : 0.0, xv = rnd();
          // a coupling below tiny is rounding of T: a row exchange would divide by it
          const bool swap = fabs(dd) < fabs(sub) && fabs(sub) >= tiny;
          const double piv = fabs(dd) < tiny ? copysign(tiny, dd) : dd;
          const double rd = recip_nr2(piv), rs = recip_nr2(swap ? sub : 1.0);
          const double l = swap ? dd * rs : sub * rd;
          f.rp[o] = swap ? rs : rd;
          f.u1[o] = swap ? dn : du;
          f.u2[o] = swap ? en : 0.0;
          f.l[o] = l;
          f.sw[o] = swap;
          x[o] = swap ? xv : xr;
          dd = swap ? fma(-l, dn, du) : fma(-l, du, dn);
          du = swap ? -l * en : en;
          xr = swap ? fma(-l, xv, xr) : fma(-l, xr, xv);
          sub = en;
        } else {
          x[o] = wb[u] ? xb[u] : xr;
          xr = wb[u] ? fma(-lb[u], xb[u], xr) : fma(-lb[u], xr, xb[u]);
        }
      }
    }
  }
  x[(long long)(n - 1) * ld] = xr;
  if (FACTOR) {
    const double piv = fabs(dd) < tiny ? copysign(tiny, dd) : dd;
    f.rp[(long long)(n - 1) * ld] = recip_nr2(piv);
    f.u1[(long long)(n - 1) * ld] = 0.0;
    f.u2[(long long)(n - 1) * ld] = 0.0;
  }
}

// Back substitution in place; max |x| and the sum of squares.  |x| stays below
// n / eps for a right-hand side of magnitude 1, so the squares cannot overflow.
__device__ __forceinline__ double tri_back(int n, const TriLu& f, double* x, double* sumsq) {
  const long long ld = f.ld;
  double x1 = 0.0, x2 = 0.0, mx = 0.0, s0 = 0.0, s1 = 0.0;
  double xb[TB], rb[TB], a1[TB], a2[TB];
  auto fetch = [&](int i0) {
#pragma unroll
    for (int u = 0; u < TB; ++u) {
      const long long o = (long long)max(i0 - u, 0) * ld;
      xb[u] = x[o];
      rb[u] = f.rp[o];
      a1[u] = f.u1[o];
      a2[u] = f.u2[o];
    }
  };
  fetch(n - 1);
  for (int i0 = n - 1; i0 >= 0; i0 -= TB) {
    double cx[TB], cr[TB], c1[TB], c2[TB];
#pragma unroll
    for (int u = 0; u < TB; ++u) {
      cx[u] = xb[u];
      cr[u] = rb[u];
      c1[u] = a1[u];
      c2[u] = a2[u];
    }
    if (i0 - TB >= 0) fetch(i0 - TB);
#pragma unroll
    for (int u = 0; u < TB; ++u) {
      const int i = i0 - u;
      if (i >= 0) {
        const double v = fma(-c1[u], x1, fma(-c2[u], x2, cx[u])) * cr[u];
        x[(long long)i * ld] = v;
        mx = fmax(mx, fabs(v));
        if (u & 1) s1 = fma(v, v, s1);
        else s0 = fma(v, v, s0);
        x2 = x1;
        x1 = v;
      }
    }
  }
  *sumsq = s0 + s1;
  return mx;
}

// x (stride ld) normalised to unit 2-norm; returns the norm before scaling.
// Eight independent loads per step keep the three sweeps bandwidth-bound.
__device__ double normalise(int n, double* x, long long ld) {
  constexpr int B = 8;
  double mx = 0.0;
  for (int i0 = 0; i0 < n; i0 += B) {
    double t[B];
#pragma unroll
    for (int u = 0; u < B; ++u) t[u] = (i0 + u < n) ? x[(long long)(i0 + u) * ld] : 0.0;
#pragma unroll
    for (int u = 0; u < B; ++u) mx = fmax(mx, fabs(t[u]));
  }
  if (mx == 0.0) return 0.0;
  const double inv = 1.0 / mx;
  double s = 0.0;
  for (int i0 = 0; i0 < n; i0 += B) {
    double t[B];
#pragma unroll
    for (int u = 0; u < B; ++u) t[u] = (i0 + u < n) ? x[(long long)(i0 + u) * ld] : 0.0;
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const double v = t[u] * inv;
      s += v * v;
    }
  }
  const double sc = inv / sqrt(s);
  for (int i0 = 0; i0 < n; i0 += B) {
    double t[B];
#pragma unroll
    for (int u = 0; u < B; ++u) t[u] = (i0 + u < n) ? x[(long long)(i0 + u) * ld] : 0.0;
#pragma unroll
    for (int u = 0; u < B; ++u)
      if (i0 + u < n) x[(long long)(i0 + u) * ld] = t[u] * sc;
  }
  return mx * sqrt(s);
}

// One thread per cluster start; X is n x n with X[i*n + m] = component i of
// vector m (so consecutive threads touch consecutive addresses), still to be
// multiplied by inv[m].  T and w are scaled to norm <= 1.
__global__ void inverse_iteration(int n, const double2* __restrict__ dv, const double* __restrict__ w,
                                  const double* __restrict__ bnd, double* __restrict__ X, double* __restrict__ inv,
                                  TriLu lu, int* status) {
  const int m0 = blockIdx.x * blockDim.x + threadIdx.x;
  if (m0 >= n) return;
  if (*status == MB_ERR_TIMEOUT) return;  // the reduction gave up: T is not whole
  const double tnorm = bnd[3];
  const double ortol = 1.0e-8 * tnorm;
  if (m0 > 0 && !(w[m0] - w[m0 - 1] > ortol)) return;  // not a cluster start
  int m1 = m0 + 1;
  while (m1 < n && !(w[m1] - w[m1 - 1] > ortol)) ++m1;
  const double eps = 2.220446049250313e-16;
  const double tiny = eps * fmax(tnorm, 1e-290);
  const long long ld = n;
  const TriLu f{lu.rp + m0, lu.u1 + m0, lu.u2 + m0, lu.l + m0, lu.sw + m0, ld};
  double lam_prev = 0.0;
  for (int m = m0; m < m1; ++m) {
    double lam = w[m];
    if (m > m0) {  // separate exactly coincident shifts (dstein's perturbation)
      const double pertol = 10.0 * fabs(eps * lam) + tiny;
      if (lam - lam_prev < pertol) lam = lam_prev + pertol;
    }
    lam_prev = lam;
    double* x = X + m;
    // deterministic start vector, generated inside the first forward sweep
    const unsigned long long seed = 0x9E3779B97F4A7C15ull ^ (unsigned long long)(m + 1) * 0xBF58476D1CE4E5B9ull;
    const int nits = (m1 - m0 > 1) ? 4 : 2;
    double scale = 1.0;
    for (int it = 0; it < nits; ++it) {
      if (it == 0) tri_forward<true>(n, dv, lam, tiny, f, x, 1.0, seed);
      else tri_forward<false>(n, dv, lam, tiny, f, x, scale, 0);
      double sq;
      const double mx = tri_back(n, f, x, &sq);
      if (!(mx > 0.0) || !isfinite(sq)) { atomicCAS(status, MB_OK, MB_ERR_NUMERIC); return; }
      if (m1 - m0 == 1) {
        scale = 1.0 / mx;
        inv[m] = 1.0 / sqrt(sq);
        continue;
      }
      // re-orthogonalise against earlier members of the cluster (MGS)
      for (int q = m0; q < m; ++q) {
        const double* y = X + q;
        double dt = 0.0;
        for (int i = 0; i < n; ++i) dt += y[(long long)i * ld] * x[(long long)i * ld];
        for (int i = 0; i < n; ++i) x[(long long)i * ld] -= dt * y[(long long)i * ld];
      }
      const double nr = normalise(n, x, ld);
      if (!(nr > 0.0) || !isfinite(nr)) { atomicCAS(status, MB_OK, MB_ERR_NUMERIC); return; }
      inv[m] = 1.0;
    }
  }
}

// Back-transformation of a small matrix, one reflector at a time: a warp keeps
// two vectors in registers (lane l rows l, l + 32, ...) and applies
// H_j = I - tau_j v_j v_j^T for j = n - 2 .. 0.  The reflectors pass through a
// ring of shared-memory stages of BS_REF columns, which the CTA's warps share;
// vectors are independent, so nothing else is exchanged.  X[i*n + m] =
// component i of vector m before its normalisation inv[m]; c column-major.
constexpr int BS_T = 128, BS_REF = 4, BS_STAGES = 4;

template <int K>
__global__ void __launch_bounds__(BS_T) back_small(int n, const double* __restrict__ V, const double* __restrict__ tau,
                                                   const double* __restrict__ X, const double* __restrict__ inv,
                                                   double* __restrict__ c) {
  extern __shared__ double ring[];  // BS_STAGES x BS_REF x (32 K)
  __shared__ double s_tau[32 * K];
  constexpr int LD = 32 * K;
  const int lane = threadIdx.x & 31;
  const int m0 = 2 * (blockIdx.x * (BS_T / 32) + (threadIdx.x >> 5));
  const bool act = m0 < n;
  const int m1 = m0 + 1 < n ? m0 + 1 : m0;
  double za[K], zb[K];
  const double ia = act ? inv[m0] : 0.0, ib = act ? inv[m1] : 0.0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int r = lane + 32 * k;
    za[k] = act && r < n ? X[(long long)r * n + m0] * ia : 0.0;
    zb[k] = act && r < n ? X[(long long)r * n + m1] * ib : 0.0;
  }
  for (int i = threadIdx.x; i < n - 1; i += BS_T) s_tau[i] = tau[i];
  for (int i = threadIdx.x; i < BS_STAGES * BS_REF * LD; i += BS_T) ring[i] = 0.0;
  __syncthreads();
  const int nref = n - 1, nst = (nref + BS_REF - 1) / BS_REF;
  auto fetch = [&](int t) {  // stage t: reflectors nref - 1 - BS_REF t, descending
    if (t < nst)
      for (int u = 0; u < BS_REF; ++u) {
        const int j = nref - 1 - BS_REF * t - u;
        if (j < 0) break;
        double* dst = ring + ((size_t)(t % BS_STAGES) * BS_REF + u) * LD;
        for (int r = threadIdx.x; r < n; r += BS_T) {
          const unsigned sa = (unsigned)__cvta_generic_to_shared(dst + r);
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(V + (long long)j * n + r) : "memory");
        }
      }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  for (int t = 0; t < BS_STAGES - 1; ++t) fetch(t);
  for (int t = 0; t < nst; ++t) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(BS_STAGES - 2) : "memory");
    __syncthreads();           // stage t has landed; every warp has left stage t - 1
    fetch(t + BS_STAGES - 1);
#pragma unroll 1
    for (int u = 0; u < BS_REF; ++u) {
      const int j = nref - 1 - BS_REF * t - u;
      if (j < 0) break;
      const double* v = ring + ((size_t)(t % BS_STAGES) * BS_REF + u) * LD + lane;
      const int k0 = (j + 1) >> 5;
      double vr[K], sa = 0.0, sb = 0.0, sa1 = 0.0, sb1 = 0.0;
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (k >= k0) {
          vr[k] = v[32 * k];
          if (k & 1) {
            sa1 = fma(vr[k], za[k], sa1);
            sb1 = fma(vr[k], zb[k], sb1);
          } else {
            sa = fma(vr[k], za[k], sa);
            sb = fma(vr[k], zb[k], sb);
          }
        }
      sa += sa1;
      sb += sb1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        sa += __shfl_xor_sync(0xffffffffu, sa, o);
        sb += __shfl_xor_sync(0xffffffffu, sb, o);
      }
      const double t0 = -s_tau[j];
      sa *= t0;
      sb *= t0;
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (k >= k0) {
          za[k] = fma(sa, vr[k], za[k]);
          zb[k] = fma(sb, vr[k], zb[k]);
        }
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  if (!act) return;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int r = lane + 32 * k;
    if (r < n) {
      c[(long long)m0 * n + r] = za[k];
      if (m1 != m0) c[(long long)m1 * n + r] = zb[k];
    }
  }
}

template <int K>
int launch_back_small(int n, const double* V, const double* tau, const double* X, const double* inv, double* c,
                      cudaStream_t stream) {
  const size_t smem = sizeof(double) * BS_STAGES * BS_REF * 32 * K;
  MB_TRY(mb_smem_optin((const void*)back_small<K>, smem));
  const int per = 2 * (BS_T / 32);
  back_small<K><<<(n + per - 1) / per, BS_T, smem, stream>>>(n, V, tau, X, inv, c);
  MB_LAUNCH_CHECK();
  return MB_OK;
}

// Z (column-major n x n): Z(i, m) = X[i*n + m] * inv[m].
__global__ void transpose_kernel(int n, const double* __restrict__ X, const double* __restrict__ inv,
                                 double* __restrict__ Z) {
  __shared__ double t[32][33];
  const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
  // X viewed as row-major [i][m]: tile rows i = by.., cols m = bx..
  for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
    int i = by + yy, m = bx + threadIdx.x;
    if (i < n && m < n) t[yy][threadIdx.x] = X[(long long)i * n + m];
  }
  __syncthreads();
  // Z column-major: Z(i, m) at m*n + i; write with i fastest
  for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
    int m = bx + yy, i = by + threadIdx.x;
    if (i < n && m < n) Z[(long long)m * n + i] = t[threadIdx.x][yy] * inv[m];
  }
}

}  // namespace

extern "C" int mb_eigh_status(int status) {
  if (status == MB_OK) return MB_OK;
  if (status == MB_ERR_TIMEOUT) return mb_set_error(MB_ERR_TIMEOUT, "eigensolver: a wait between CTAs gave up");
  return mb_set_error(MB_ERR_NUMERIC, "eigensolver: inverse iteration failed");
}

extern "C" size_t mb_eigh_ws_bytes(int n) { return sizeof(double) * eigh::ws_doubles(n) + 256; }

// cluster_max: the largest order that the cluster kernel reduces.
extern "C" int mb_eigh_cluster_ws(int n, double* fpacked, int perturb, double* c, double* eigs, void* ws,
                                  int* status_dev, int cluster_max, cudaStream_t stream) {
  const size_t nn = (size_t)n * n;
  const eigh::Ws w = eigh::carve(n, ws);
  MB_CUDA(cudaMemsetAsync(status_dev, 0, sizeof(int), stream));
  if (n == 1) {
    MB_TRY(mb_unpack_dev(1, fpacked, w.A, 1, perturb, fpacked, stream));
    MB_CUDA(cudaMemcpyAsync(eigs, w.A, sizeof(double), cudaMemcpyDeviceToDevice, stream));
    const double one = 1.0;
    MB_CUDA(cudaMemcpyAsync(c, &one, sizeof(double), cudaMemcpyHostToDevice, stream));
    return MB_OK;
  }
  // T's records of the Sturm counts and of the inverse iteration, before Y is used
  double2* de = (double2*)(((uintptr_t)w.Y + 15) & ~(uintptr_t)15);
  double2* dv = de + n + 2 * SB;
  double* inv = w.wvec;  // the eigenvectors' norms, after the panels have used it
  double* weig = w.e2;   // eigenvalues of the scaled T
  // one launch up to the order whose columns fit in the registers of 16 CTAs
  const bool small = n <= cluster_max;
  if (small) {
    mb_kstat_mark(MB_KSTAT_ONCHIP, stream, true);
    MB_TRY(mb_tridiag_cluster(n, fpacked, perturb, w.V, w.d, w.e, w.tau, status_dev, stream));
    mb_kstat_mark(MB_KSTAT_ONCHIP, stream, false);
  } else {
    MB_TRY(mb_unpack_dev(n, fpacked, w.A, n, perturb, fpacked, stream));
    MB_CUDA(cudaMemsetAsync(w.V, 0, sizeof(double) * nn, stream));
    int dev = 0, sms = 0;
    MB_CUDA(cudaGetDevice(&dev));
    MB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    int k = 0;
    MB_TRY(mb_eigh_panels(n, n - mb_tridiag_grid_max(sms), &w, stream, &k));
    const size_t o = (size_t)k * n + k;
    mb_kstat_mark(MB_KSTAT_ONCHIP, stream, true);
    MB_TRY(mb_tridiag_grid(n - k, sms, w.A + o, n, w.V + o, w.d + k, w.e + k, w.tau + k, w.U0, status_dev, stream));
    mb_kstat_mark(MB_KSTAT_ONCHIP, stream, false);
  }
  tri_bounds<<<1, 1024, 0, stream>>>(n, w.d, w.e, de, dv, w.bnd);
  MB_LAUNCH_CHECK();
  bisect_kernel<<<(n * 32 + 127) / 128, 128, 0, stream>>>(n, de, w.bnd, weig, eigs);
  MB_LAUNCH_CHECK();
  // eigenvectors of T; the reduction has no more use for A
  const TriLu lu{w.U0, w.U1, w.U2, w.A, (unsigned char*)w.Z, 0};
  inverse_iteration<<<(n + 31) / 32, 32, 0, stream>>>(n, dv, weig, w.bnd, w.X, inv, lu, status_dev);
  MB_LAUNCH_CHECK();
  if (small) {
    if (n <= 64) return launch_back_small<2>(n, w.V, w.tau, w.X, inv, c, stream);
    if (n <= 160) return launch_back_small<5>(n, w.V, w.tau, w.X, inv, c, stream);
    if (n <= 320) return launch_back_small<10>(n, w.V, w.tau, w.X, inv, c, stream);
    return launch_back_small<20>(n, w.V, w.tau, w.X, inv, c, stream);
  }
  dim3 g((n + 31) / 32, (n + 31) / 32), blk(32, 8);
  transpose_kernel<<<g, blk, 0, stream>>>(n, w.X, inv, w.Z);
  MB_LAUNCH_CHECK();
  return mb_eigh_back(n, &w, c, stream);
}

extern "C" int mb_eigh_ws(int n, double* fpacked, int perturb, double* c, double* eigs, void* ws, int* status_dev,
                          cudaStream_t stream) {
  return mb_eigh_cluster_ws(n, fpacked, perturb, c, eigs, ws, status_dev, mb_tridiag_cluster_max(), stream);
}

extern "C" int mb_eigh_packed_dev(int n, double* fpacked, double* c, double* eigs, cudaStream_t stream) {
  if (n <= 0) return mb_set_error(MB_ERR_ARG, "mb_eigh_packed_dev: n <= 0");
  void* ws = nullptr;
  int* st = nullptr;
  MB_CUDA(cudaMalloc(&ws, mb_eigh_ws_bytes(n)));
  cudaError_t ce = cudaMalloc((void**)&st, sizeof(int));
  if (ce != cudaSuccess) { cudaFree(ws); return mb_set_cuda_error(ce, "cudaMalloc", __FILE__, __LINE__); }
  int rc = mb_eigh_ws(n, fpacked, 1, c, eigs, ws, st, stream);
  int hst = 0;
  if (rc == MB_OK) {
    ce = cudaMemcpyAsync(&hst, st, sizeof(int), cudaMemcpyDeviceToHost, stream);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(stream);
    if (ce != cudaSuccess) rc = mb_set_cuda_error(ce, "eigh status", __FILE__, __LINE__);
    else rc = mb_eigh_status(hst);
  }
  cudaFree(ws);
  cudaFree(st);
  return rc;
}
