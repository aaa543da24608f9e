// Batched SCF: many small molecules (n <= 128 basis functions), each SCF run
// start to finish by one CTA of a persistent kernel.
//
// A CTA takes the next molecule from a shared counter (uneven sizes balance
// themselves) and restates iter (SCF/iter.F90:16-1107) for it in the same
// form as mb_scf_run with full diagonalisation every iteration: level shift,
// Fock build, energy, convergence test, eigensolve, density, cnvg, and the
// exit diagonalisation.  Every thread computes the control scalars from the
// same CTA-wide values (so they agree bit for bit); the CTA runs the phases
// between barriers:
//   * Fock: P staged in shared memory; a thread per diagonal-block element
//     folds that element's contributions in the reference order (pairs with
//     lower atoms, the one-centre terms, pairs with higher atoms) and a thread
//     per off-diagonal element forms its exchange sum -- the operation order
//     of fock2/fock1, so F is bit-identical to the oracle;
//   * eigensolve in shared memory: Householder reduction to tridiagonal form
//     (16 x 16 thread tiles, two barriers per column), eigenvalues through the LUMO
//     by 5-section Sturm counts (four lanes per eigenvalue), the occupied
//     eigenvectors of T by inverse iteration (thread per vector, clusters
//     re-orthogonalised), back-transformation (a lane group per vector);
//   * density P = 2 Z Z^T over the occupied vectors; cnvg with its diagonal
//     statistics in the reference's order (bit-identical).
// Shared memory holds the packed matrix (P, then F, then the n x nocc
// eigenvectors when they fit) and the tridiagonal; 77 KB, two CTAs per SM.
// Each molecule's F, P, P_old live in global memory; each CTA has a global
// scratch for the LU factors, the reflectors and oversized eigenvectors.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "mb_common.cuh"
#include "pm7_params.h"

extern "C" int mb_hcore_batch_dev(const MbHcoreBatch* b, cudaStream_t stream);

namespace {

constexpr int BT_T = 256;                                 // threads per CTA
constexpr int BT_W = BT_T / 32;                           // warps per CTA
constexpr int BT_NMAX = 128;                              // basis functions per molecule
constexpr int BT_AMAX = BT_NMAX * (BT_NMAX + 1) / 2;      // packed lower triangle
constexpr int BT_ZMAX = 11008;                            // n * nocc
constexpr int BT_IMAX = 320;                              // diagonal-block elements, <= 2.5 n
constexpr long long BT_LU = 5LL * BT_ZMAX;                // LU factors of T - lambda I, 5 n per vector
constexpr long long BT_SCR = BT_LU + BT_AMAX + BT_ZMAX;   // + reflectors + oversized Z: doubles per CTA
// reflectors per back-transformation block: a template parameter of the
// kernel (4, 8 or 16), chosen per batch by mb_batch_autotune (default 8)
__host__ __device__ constexpr int bt_tw(int nb) { return ((BT_NMAX - 2 + nb - 1) / nb) * nb * nb; }  // T of every block
constexpr int BT_PHASES = 8;
static_assert(BT_T == 256, "the reduction tile is 16 x 16 threads");  // fock, energy, householder, bisection, inverse iteration, back-transform, density, cnvg

struct Mol {
  int n, nclose, numat, aoff;  // aoff: first atom in the concatenated atom tables
  long long hoff, woff;        // offsets into packed arrays / W
  int doff, pad;               // offset into per-orbital arrays
  double enuclr, atheat;
};

struct BatchArgs {
  const Mol* mol;
  const int* order;          // molecules in the order the CTAs take them
  int nmol;
  const int* first;          // molecule-local first orbital of each atom
  const int* nor;
  const double* h;
  const double* w;
  const long long* wrow;     // molecule-local W offsets of each atom's first pair block
  const int* cum;
  const double* pdiag;
  double* f;
  double* p;
  double* pold;
  double* pold2;
  double* scratch;           // per CTA: BT_SCR doubles (LU factors, reflectors, Z when it is too big)
  double* escf;
  double* ee;
  int* niter;
  int* conv;
  double* homo;
  double* lumo;
  int* next;
  unsigned long long* phase;  // optional: SM cycles per phase, summed over CTAs
  int itrmax;
  double scfcrt;
};

__device__ __forceinline__ long long tri(long long r, long long c) { return r * (r + 1) / 2 + c; }
__device__ __forceinline__ int indx1(int i, int j) { if (i < j) { int t = i; i = j; j = t; } return (i * (i - 1)) / 2 + j; }
// (row, column) of packed lower-triangle index q < 2^24
__device__ __forceinline__ void tri_rc(int q, int& r, int& c) {
  r = (int)((sqrtf(8.0f * (float)q + 1.0f) - 1.0f) * 0.5f);
  while (r * (r + 1) / 2 > q) --r;
  while ((r + 1) * (r + 2) / 2 <= q) ++r;
  c = q - r * (r + 1) / 2;
}

__constant__ int c_bpidx[16] = {1, 2, 4, 7, 2, 3, 5, 8, 4, 5, 6, 9, 7, 8, 9, 10};

// 1/q: hardware estimate and two Newton steps (relative error a few ulps);
// used where an eigenvalue search or inverse iteration divides, both of which
// tolerate that.
__device__ __forceinline__ double recip_nr2(double q) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(q));
  double e = fma(-q, r, 1.0);
  r = fma(r, e, r);
  e = fma(-q, r, 1.0);
  return fma(r, e, r);
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Phase clock (thread 0): charges the cycles since the last mark to phase i.
// ph[BT_PHASES] holds the last mark; ph == nullptr when phase timing is off.
__device__ __forceinline__ void ph_mark(long long* ph, int i) {
  if (ph && threadIdx.x == 0) {
    const long long now = clock64();
    ph[i] += now - ph[BT_PHASES];
    ph[BT_PHASES] = now;
  }
}

struct Smem {
  double* A;      // packed lower (BT_AMAX): P during the Fock build, the matrix during the reduction, Z after it
  double* Z;      // n x nz eigenvectors, Z[i * nz + m]: the A region when n * nz fits, else global scratch
  double* d;
  double* e;
  double* e2;
  double* tau;
  double* pv;
  double* v;
  double* eig;    // eigenvalues 0 .. LUMO
  double* red;    // two sets of BT_W warp partials
  double* scal;
  double* tw;     // the back-transformation blocks' T
  int* afirst;    // the molecule's atom tables
  int* anor;
  int* acum;
  int* orb_atom;  // atom of each orbital
  int* item;      // diagonal-block elements: atom << 4 | element
  long long* awrow;
};

// Sum over the CTA, the same value in every thread: butterfly within each
// warp (commutative pairs, so every lane holds the same bits), then the warp
// sums in a fixed order.
__device__ double block_sum_all(double x, double* red) {
  x = warp_sum(x);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  double r = red[0];
#pragma unroll
  for (int q = 1; q < BT_W; ++q) r += red[q];
  __syncthreads();
  return r;
}

// ------------------------------------------------------------------- Fock
// F = H (+ the level-shift start) + G(P), P staged in S.A, PA = cpa * P
// exactly (the reference's PA is P/2 after every density and w1 * P for the
// diagonal guess).  Every element is written once, in the operation order of
// fock2 (SCF/fock2.F90:149-298) and fock1 (SCF/fock1.F90):
//   * a diagonal-block element of atom a folds the Coulomb terms of the
//     pairs (a, b < a) in b order, a's one-centre terms, then the pairs
//     (b > a, a) in b order;
//   * an element of the block of atoms a > b is its start value minus the
//     exchange sum over a's and b's orbitals.

__device__ __forceinline__ double f_start(const double* __restrict__ h, long long idx, bool diag, double ptot,
                                          double cpa, double shift, bool use_shift) {
  if (!use_shift) return h[idx];
  double v = DADD(DADD(h[idx], DMUL(shift, DMUL(ptot, cpa))), DMUL((double)(idx + 1), 1.0e-16));
  if (diag) v = DSUB(v, shift);
  return v;
}

__device__ __forceinline__ double pk(const double* P, int r, int c) {  // 0-based orbitals
  return r >= c ? P[tri(r, c)] : P[tri(c, r)];
}

// Coulomb contribution of pair (hi > lo) to element q of atom a's block.
__device__ __forceinline__ double pair_q(const Smem& S, const double* __restrict__ w, int hi, int lo, int a, int q,
                                         double acc) {
  const double* P = S.A;
  const int nh = S.anor[hi], nl = S.anor[lo];
  const double* wk = w + S.awrow[hi] + (long long)(nh == 1 ? 1 : 10) * S.acum[lo];
  const int fh = S.afirst[hi], fl = S.afirst[lo];
  if (nh == 4 && nl == 4) {
    const int o = (a == hi) ? fl : fh;
    double s;
    if (a == hi) {
      s = DMUL(pk(P, o, o), wk[q * 10 + c_bpidx[0] - 1]);
#pragma unroll
      for (int m = 1; m < 16; ++m) s = DADD(s, DMUL(pk(P, o + m / 4, o + m % 4), wk[q * 10 + c_bpidx[m] - 1]));
    } else {
      s = DMUL(pk(P, o, o), wk[(c_bpidx[0] - 1) * 10 + q]);
#pragma unroll
      for (int m = 1; m < 16; ++m) s = DADD(s, DMUL(pk(P, o + m / 4, o + m % 4), wk[(c_bpidx[m] - 1) * 10 + q]));
    }
    return DADD(acc, s);
  }
  if (nh != nl) {  // one heavy atom (four orbitals), one hydrogen
    const int fheavy = nh == 4 ? fh : fl, flight = nh == 4 ? fl : fh;
    const bool a_heavy = (a == hi) == (nh == 4);
    if (a_heavy) return DADD(acc, DMUL(P[tri(flight, flight)], wk[q]));
    double sumdia = 0.0, sumoff = 0.0;
#pragma unroll
    for (int i = 0; i <= 3; ++i) {
#pragma unroll
      for (int j = 0; j < i; ++j) sumoff = DADD(sumoff, DMUL(P[tri(fheavy + i, fheavy + j)], wk[i * (i + 1) / 2 + j]));
      sumdia = DADD(sumdia, DMUL(P[tri(fheavy + i, fheavy + i)], wk[i * (i + 1) / 2 + i]));
    }
    return DADD(DADD(acc, DMUL(sumoff, 2.0)), sumdia);
  }
  const int o = (a == hi) ? fl : fh;  // two hydrogens
  return DADD(acc, DMUL(P[tri(o, o)], wk[0]));
}

// Final value of element q of atom a's diagonal block.
__device__ double fock_item(const Smem& S, const Mol& M, const double* __restrict__ w, const double* __restrict__ h,
                            int a, int q, double cpa, double shift, bool use_shift) {
  const double* P = S.A;
  const int fa = S.afirst[a], na = S.anor[a];
  int r, c;
  tri_rc(q, r, c);
  const long long idx = tri(fa + r, fa + c);
  double acc = f_start(h, idx, r == c, P[idx], cpa, shift, use_shift);
  for (int b = 0; b < a; ++b) acc = pair_q(S, w, a, b, a, q, acc);
  {  // fock1: one-centre terms
    const int il = na == 1 ? 1 : 10;
    const double* wo = w + S.awrow[a] + (long long)il * S.acum[a];
    const int iw = r + 1, jw = c + 1, ijw = q + 1;
    double sum = 0.0;
    for (int k = 1; k <= na; ++k)
      for (int l = 1; l <= na; ++l) {
        const int klw = indx1(k, l), ikw = indx1(k, jw), jlw = indx1(l, iw);
        const double pt = pk(P, fa + k - 1, fa + l - 1);
        sum = DSUB(DADD(sum, DMUL(pt, wo[(ijw - 1) + il * (klw - 1)])), DMUL(DMUL(pt, cpa), wo[(ikw - 1) + il * (jlw - 1)]));
      }
    acc = DADD(acc, sum);
  }
  for (int b = a + 1; b < M.numat; ++b) acc = pair_q(S, w, b, a, a, q, acc);
  return acc;
}

// Final value of element (r, c) of the block of atoms a > b.
__device__ double fock_exchange(const Smem& S, const double* __restrict__ w, const double* __restrict__ h, int r,
                                int c, int a, int b, double cpa, double shift, bool use_shift) {
  const double* P = S.A;
  const long long idx = tri(r, c);
  const int na = S.anor[a], nb = S.anor[b], fa = S.afirst[a], fb = S.afirst[b];
  const double* wk = w + S.awrow[a] + (long long)(na == 1 ? 1 : 10) * S.acum[b];
  const int mu = r - fa, nu = c - fb;
  double s;
  if (na == 4 && nb == 4) {
    s = 0.0;
#pragma unroll
    for (int lam = 0; lam < 4; ++lam)
#pragma unroll
      for (int sig = 0; sig < 4; ++sig) {
        const double t = DMUL(DMUL(P[tri(fa + lam, fb + sig)], cpa),
                              wk[(indx1(mu + 1, lam + 1) - 1) * 10 + indx1(nu + 1, sig + 1) - 1]);
        s = (lam == 0 && sig == 0) ? t : DADD(s, t);
      }
  } else if (na == 4) {
    s = 0.0;
#pragma unroll
    for (int j = 1; j <= 4; ++j) s = DADD(s, DMUL(DMUL(P[tri(fa + j - 1, fb)], cpa), wk[indx1(mu + 1, j) - 1]));
  } else if (nb == 4) {
    s = 0.0;
#pragma unroll
    for (int l = 1; l <= 4; ++l) s = DADD(s, DMUL(DMUL(P[tri(fa, fb) + l - 1], cpa), wk[indx1(nu + 1, l) - 1]));
  } else {
    s = DMUL(DMUL(P[idx], cpa), wk[0]);
  }
  return DSUB(f_start(h, idx, false, P[idx], cpa, shift, use_shift), s);
}

__device__ void cta_fock(const BatchArgs& B, const Mol& M, const Smem& S, int nitems, double cpa, double shift,
                         bool use_shift, double* __restrict__ f, const double* __restrict__ p,
                         const double* __restrict__ h) {
  const int mp = M.n * (M.n + 1) / 2;
  for (int q = threadIdx.x; q < mp; q += BT_T) S.A[q] = p[q];
  __syncthreads();
  const double* w = B.w + M.woff;
  // the diagonal-block elements (the long folds) first, then the exchange elements
  for (int u = threadIdx.x; u < nitems + mp; u += BT_T) {
    if (u < nitems) {
      const int it = S.item[u], a = it >> 4, q = it & 15;
      const double v = fock_item(S, M, w, h, a, q, cpa, shift, use_shift);
      int r, c;
      tri_rc(q, r, c);
      f[tri(S.afirst[a] + r, S.afirst[a] + c)] = v;
    } else {
      int r, c;
      tri_rc(u - nitems, r, c);
      const int a = S.orb_atom[r], b = S.orb_atom[c];
      if (a != b) f[tri(r, c)] = fock_exchange(S, w, h, r, c, a, b, cpa, shift, use_shift);
    }
  }
  __syncthreads();
}

// helect: sum_{i>j} pa (h + f) + 0.5 sum_i pa_ii (h_ii + f_ii), pa = cpa * p.
__device__ double cta_helect(int n, const double* p, double cpa, const double* h, const double* f, double* red) {
  double s = 0.0, dsum = 0.0;
  for (int r = threadIdx.x; r < n; r += BT_T) {
    const long long base = (long long)r * (r + 1) / 2;
    double a = 0.0;
    for (int c = 0; c < r; ++c) a += DMUL(p[base + c], cpa) * (h[base + c] + f[base + c]);
    s += a;
    dsum += DMUL(p[base + r], cpa) * (h[base + r] + f[base + r]);
  }
  const double a = block_sum_all(s, red);
  const double b = block_sum_all(dsum, red);
  return a + 0.5 * b;
}

// ------------------------------------------------------------ eigensolver
// Eigenvalues 0 .. max(nz, 1) of the packed symmetric matrix in S.A (lost)
// and, when vectors, the eigenvectors of the lowest nz in S.Z.  scr: the
// CTA's global scratch (LU factors, then the reflectors when Z overlays A).

// (Built without contraction for the Fock build's sake: the multiply-adds of the
// eigensolver and the density are written out.)

// Columns k0 .. kend-1 of the Householder reduction, whose active rows lie in the
// last NA tiles of 16: two barriers a column, the reflector's norm from the
// previous column's update.  Thread (tr, tc) of the 16 x 16 works on element
// (tr, tc) of every tile, so with the tiles' count constant each address is a base
// and an offset known to the compiler, where addresses formed per element took
// most of the issue slots: 1500 alkanes C3..C20 27.7 -> 22.0 ms with the Sturm
// counts below (one B200; 26.5 when inlined, for the registers it takes from the
// other phases).
// Rows and columns below k + 1 take part with zeros; the rows from n up to the
// tile's edge are zero.
template <int NA>
__device__ __noinline__ void reduce_columns(int k0, int kend, int n, double* A, double* redA, double* Sd, double* Se,
                                            double* Stau, double* Spv, double* Sv) {
  constexpr int P = NA > 4 ? 8 : NA > 2 ? 4 : NA;  // rows a lane group reduces, a power of two
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5, tr = tid >> 4, tc = tid & 15;
  double* redB = redA + BT_W;
  const int base = (((n + 15) >> 4) - NA) * 16;
  int rb[NA], cb[NA], db[NA];  // tile (a, b): row element at rb[a] + 16 b, its mirror image at cb[b] + 16 a
#pragma unroll
  for (int a = 0; a < NA; ++a) {
    const int i = base + tr + 16 * a, j = base + tc + 16 * a;
    rb[a] = i * (i + 1) / 2 + base + tc;
    cb[a] = j * (j + 1) / 2 + base + tr;
    db[a] = (tc <= tr ? rb[a] : cb[a]) + 16 * a;
  }
  for (int k = k0; k < kend; ++k) {
    const int k1 = k + 1;
    double sigma = redA[0];
#pragma unroll
    for (int q = 1; q < BT_W; ++q) sigma += redA[q];
    const double alpha = A[tri(k1, k)];
    double beta, tau, scal;
    if (sigma == 0.0) { beta = alpha; tau = 0.0; scal = 0.0; }
    else {
      beta = -copysign(sqrt(fma(alpha, alpha, sigma)), alpha);
      tau = (beta - alpha) / beta;
      scal = 1.0 / (alpha - beta);
    }
    if (tid == 0) {
      Se[k] = beta;
      Stau[k] = tau;
      Sd[k] = A[tri(k, k)];
    }
    // p = tau A22 v: row sums over this thread's columns, then over the 16
    // lanes, which share the rows among them
    double vr[NA], acc[P];
#pragma unroll
    for (int b = 0; b < NA; ++b) {
      const int j = base + tc + 16 * b;
      vr[b] = j < k1 ? 0.0 : j == k1 ? 1.0 : A[cb[b] - base - tr + k] * scal;
    }
#pragma unroll
    for (int a = 0; a < P; ++a) {
      acc[a] = 0.0;
      if (a < NA) {
#pragma unroll
        for (int b = 0; b < NA; ++b)
          acc[a] = fma(A[a > b ? rb[a] + 16 * b : a < b ? cb[b] + 16 * a : db[a]], vr[b], acc[a]);
      }
    }
    int a_own = 0;
#pragma unroll
    for (int h = P / 2, o = 8; o > 0; h /= 2, o /= 2) {
      if (h > 0) {
        const bool up = (tc & o) != 0;
#pragma unroll
        for (int q = 0; q < h; ++q) {
          const double send = up ? acc[q] : acc[q + h];
          acc[q] = (up ? acc[q + h] : acc[q]) + __shfl_xor_sync(0xffffffffu, send, o);
        }
        if (up) a_own += h;
      } else {
        acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
      }
    }
    double dot = 0.0;
    if ((tc & (16 / P - 1)) == 0 && a_own < NA) {
      const int i = base + tr + 16 * a_own;
      const double vi = i < k1 ? 0.0 : i == k1 ? 1.0 : A[i * (i + 1) / 2 + k] * scal;
      const double s = i < k1 ? 0.0 : acc[0] * tau;
      Spv[i] = s;
      Sv[i] = vi;
      dot = s * vi;
    }
    dot = warp_sum(dot);
    if (lane == 0) redB[wp] = dot;
    __syncthreads();
    double dt = redB[0];
#pragma unroll
    for (int q = 1; q < BT_W; ++q) dt += redB[q];
    const double kk = 0.5 * tau * dt;
    // A22 -= v w^T + w v^T, w = p - kk v; the reflector replaces column k;
    // squares of the new column k + 1 below its subdiagonal give the next norm
    double wr[NA];
#pragma unroll
    for (int b = 0; b < NA; ++b) {
      const int j = base + tc + 16 * b;
      vr[b] = Sv[j];
      wr[b] = fma(-kk, vr[b], Spv[j]);
    }
    double nxt = 0.0;
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      const int i = base + tr + 16 * a;
      const double vi = Sv[i], wi = fma(-kk, vi, Spv[i]);
#pragma unroll
      for (int b = 0; b <= a; ++b) {
        if (b == a && tc > tr) continue;
        double* x = A + rb[a] + 16 * b;
        const double u = fma(-vi, wr[b], fma(-wi, vr[b], *x));
        *x = u;
        if (b == 0 && tc == (k1 & 15) && i >= k + 3) nxt = fma(u, u, nxt);
      }
      if (tc == (k & 15) && i >= k + 2) A[rb[a] - base - tc + k] = vi;
    }
    nxt = warp_sum(nxt);
    if (lane == 0) redA[wp] = nxt;
    __syncthreads();
  }
}

// Sturm count from the leading principal minors' three-term recurrence,
// p_i = (d_i - x) p_(i-1) - e_(i-1)^2 p_(i-2): a dependent chain of one multiply-add
// a row, where the quotients p_i / p_(i-1) take a reciprocal.  Eight rows at a time
// from a pair scaled by a power of two; T has norm <= 1, so a row grows p at most
// threefold.  A block in which some |p_i| falls below 1e-120 (2^-398) is taken again by
// quotients.  de[i] = (d_i, e_(i-1)^2), followed by 2 SB records (2, 0): rows that
// keep the sign of p.
constexpr int SB = 8;
constexpr int kSturmTiny = 0x27100000;  // high word of 2^-398
constexpr double kPivmin = 1.0e-290;

__device__ __forceinline__ int sturm(int n, const double2* de, double x) {
  double p1 = de[0].x - x, p0 = 1.0;
  if (fabs(p1) < kPivmin) p1 = -kPivmin;
  int cnt = p1 < 0.0;
  for (int i0 = 1; i0 < n; i0 += SB) {
    double db[SB], eb[SB];
#pragma unroll
    for (int u = 0; u < SB; ++u) {
      const double2 t = de[i0 + u];
      db[u] = t.x - x;
      eb[u] = t.y;
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
        q = fma(-eb[u], recip_nr2(q), db[u]);
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

// reltol: relative width at which an eigenvalue's bracket stops shrinking.
template <int BT_NB>
__device__ void cta_eigh(int n, int nz, bool vectors, double reltol, Smem& S, double* scr, long long* ph) {
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  double* A = S.A;
  // ---- Householder reduction to tridiagonal form, lower
  const int ntile = (n + 15) >> 4;
  {
    double part = 0.0;
    for (int i = 2 + tid; i < n; i += BT_T) part = fma(A[tri(i, 0)], A[tri(i, 0)], part);
    for (int q = n * (n + 1) / 2 + tid; q < 8 * ntile * (16 * ntile + 1); q += BT_T) A[q] = 0.0;
    part = warp_sum(part);
    if (lane == 0) S.red[wp] = part;
    __syncthreads();
  }
  for (int na = ntile; na >= 1; --na) {
    // columns k whose row k + 1 is the first active row's tile
    const int base = (ntile - na) * 16, k0 = base > 0 ? base - 1 : 0, kend = min(base + 15, n - 2);
    switch (na) {
      case 8: reduce_columns<8>(k0, kend, n, A, S.red, S.d, S.e, S.tau, S.pv, S.v); break;
      case 7: reduce_columns<7>(k0, kend, n, A, S.red, S.d, S.e, S.tau, S.pv, S.v); break;
      case 6: reduce_columns<6>(k0, kend, n, A, S.red, S.d, S.e, S.tau, S.pv, S.v); break;
      case 5: reduce_columns<5>(k0, kend, n, A, S.red, S.d, S.e, S.tau, S.pv, S.v); break;
      case 4: reduce_columns<4>(k0, kend, n, A, S.red, S.d, S.e, S.tau, S.pv, S.v); break;
      case 3: reduce_columns<3>(k0, kend, n, A, S.red, S.d, S.e, S.tau, S.pv, S.v); break;
      case 2: reduce_columns<2>(k0, kend, n, A, S.red, S.d, S.e, S.tau, S.pv, S.v); break;
      default: reduce_columns<1>(k0, kend, n, A, S.red, S.d, S.e, S.tau, S.pv, S.v); break;
    }
  }
  if (tid == 0) {
    if (n >= 2) {
      S.d[n - 2] = A[tri(n - 2, n - 2)];
      S.e[n - 2] = A[tri(n - 1, n - 2)];
      S.tau[n - 2] = 0.0;
    }
    S.d[n - 1] = A[tri(n - 1, n - 1)];
  }
  // reflectors to global scratch when Z is to overlay A
  const bool zshared = S.Z == S.A;
  double* refl = zshared ? scr + BT_LU : A;
  if (vectors && zshared)
    for (int q = tid; q < n * (n + 1) / 2; q += BT_T) refl[q] = A[q];
  __syncthreads();
  ph_mark(ph, 2);
  // ---- bounds; T scaled by a power of two to norm <= 1 as the records of the
  // Sturm counts (in the room of the back-transformation's T)
  double2* de = reinterpret_cast<double2*>(S.tw);
  if (tid < 32) {
    double lo = 1e300, hi = -1e300;
    for (int i = lane; i < n; i += 32) {
      const double r = (i > 0 ? fabs(S.e[i - 1]) : 0.0) + (i < n - 1 ? fabs(S.e[i]) : 0.0);
      lo = fmin(lo, S.d[i] - r);
      hi = fmax(hi, S.d[i] + r);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    const double tnorm = fmax(fabs(lo), fabs(hi));
    const double pad = 2.0 * 2.220446049250313e-16 * tnorm * n + 1e-300;
    // 2^-e with tnorm < 2^e; 1 when the norm is zero or not finite, or tiny
    const int ex = (__double2hiint(tnorm) >> 20) & 0x7ff;
    const double sc = (ex > 64 && ex < 1982) ? __hiloint2double((2045 - ex) << 20, 0) : 1.0;
    if (lane == 0) {
      S.scal[4] = lo - pad;
      S.scal[5] = hi + pad;
      S.scal[6] = sc;
      S.scal[7] = tnorm;
    }
    for (int i = lane; i < n + 2 * SB; i += 32) {
      const double ep = i > 0 && i < n ? S.e[i - 1] * sc : 0.0;
      de[i] = i < n ? make_double2(S.d[i] * sc, ep * ep) : make_double2(2.0, 0.0);
    }
  }
  __syncthreads();
  // ---- eigenvalues 0 .. LUMO by 5-section, four lanes per eigenvalue.  Every
  // lane runs the same rounds and steps (groups that have converged idle), so
  // the 4-lane shuffles always see a converged warp.
  {
    const int grp = tid >> 2, ln = tid & 3, base = tid & 31 & ~3;
    const double sc = S.scal[6];
    const double atol = 2.220446049250313e-16 * S.scal[7] + 1e-290;
    const int nlo = nz > 1 ? nz : 1;
    const int nev = nlo + 1 < n ? nlo + 1 : n;
    const int rounds = (nev + BT_T / 4 - 1) / (BT_T / 4);
    for (int rd = 0; rd < rounds; ++rd) {
      const int mm = rd * (BT_T / 4) + grp;
      const bool active = mm < nev;
      double lo = S.scal[4], hi = S.scal[5];
      bool done = !active;
      for (int it = 0; it < 100; ++it) {
        if (!done && hi - lo <= reltol * fmax(fabs(lo), fabs(hi)) + atol) done = true;
        const double x = lo + (hi - lo) * ((double)(ln + 1) / 5.0);
        const int cnt = done ? 0 : sturm(n, de, x * sc);
        const int flag = cnt > mm ? 1 : 0;
        int above = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) above |= __shfl_sync(0xffffffffu, flag, base + q) << q;
        double xs[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) xs[q] = __shfl_sync(0xffffffffu, x, base + q);
        if (!done) {
          double nl = lo, nh = hi;
          if (above == 0) {
            nl = xs[3];
          } else {
            const int firstl = __ffs(above) - 1;
            nh = xs[firstl];
            if (firstl > 0) nl = xs[firstl - 1];
          }
          if (!(nl > lo) && !(nh < hi)) done = true;
          lo = nl;
          hi = nh;
        }
        if (__all_sync(0xffffffffu, done)) break;
      }
      if (active && ln == 0) S.eig[mm] = 0.5 * (lo + hi);
    }
  }
  __syncthreads();
  ph_mark(ph, 3);
  if (!vectors) return;
  // ---- eigenvectors 0..nz-1 of T by inverse iteration (thread per cluster start)
  {
    const double tnorm = S.scal[7];
    // vectors whose eigenvalues lie closer than ortol are a cluster
    // (iterated together, re-orthogonalised); farther pairs converge apart in
    // two solves even from eigenvalues good to 1e-11 relative
    const double ortol = 1.0e-7 * tnorm;
    const double eps = 2.220446049250313e-16;
    const double tiny = eps * fmax(tnorm, 1e-300);
    double* Z = S.Z;
    for (int m0 = tid; m0 < nz; m0 += BT_T) {
      if (m0 > 0 && !(S.eig[m0] - S.eig[m0 - 1] > ortol)) continue;
      int m1 = m0 + 1;
      while (m1 < nz && !(S.eig[m1] - S.eig[m1 - 1] > ortol)) ++m1;
      double* u0 = scr + (long long)m0 * 5 * n;
      double* u1 = u0 + n;
      double* u2 = u1 + n;
      double* ul = u2 + n;
      double* us = ul + n;
      double lam_prev = 0.0;
      for (int mv = m0; mv < m1; ++mv) {
        double lam = S.eig[mv];
        if (mv > m0) {
          const double pertol = 10.0 * fabs(eps * lam) + tiny;
          if (lam - lam_prev < pertol) lam = lam_prev + pertol;
        }
        lam_prev = lam;
        double* x = Z + mv;  // stride nz
        // LU with partial pivoting of T - lam I, once per vector: 1 / pivot,
        // the two entries right of it, the multiplier, whether rows swapped
        {
          double dd = S.d[0] - lam, du = n > 1 ? S.e[0] : 0.0;
          for (int i = 0; i < n - 1; ++i) {
            const double sub = S.e[i], dn = S.d[i + 1] - lam, en = (i + 1 < n - 1) ? S.e[i + 1] : 0.0;
            if (fabs(dd) >= fabs(sub)) {
              double pv = dd;
              if (fabs(pv) < tiny) pv = copysign(tiny, pv == 0.0 ? 1.0 : pv);
              const double rp = recip_nr2(pv);
              const double l = sub * rp;
              u0[i] = rp; u1[i] = du; u2[i] = 0.0; ul[i] = l; us[i] = 0.0;
              dd = fma(-l, du, dn);
              du = en;
            } else {
              const double rs = recip_nr2(sub);
              const double l = dd * rs;
              u0[i] = rs; u1[i] = dn; u2[i] = en; ul[i] = l; us[i] = 1.0;
              dd = fma(-l, dn, du);
              du = -l * en;
            }
          }
          double last = dd;
          if (fabs(last) < tiny) last = copysign(tiny, last == 0.0 ? 1.0 : last);
          u0[n - 1] = recip_nr2(last);
        }
        const int nits = (m1 - m0 > 1) ? 4 : 2;
        for (int itr = 0; itr < nits; ++itr) {
          // forward (row swaps and multipliers) and back substitution; the
          // first pass starts from a pseudo-random vector made on the way
          unsigned long long rs = 0x9E3779B97F4A7C15ull ^ (unsigned long long)(mv + 1) * 0xBF58476D1CE4E5B9ull;
          auto rnd = [&]() {
            rs ^= rs >> 31; rs *= 0x94D049BB133111EBull; rs ^= rs >> 29;
            return ((double)(rs >> 11) * (1.0 / 9007199254740992.0)) - 0.5;
          };
          double xr = itr == 0 ? rnd() : x[0];
          for (int i = 0; i < n - 1; ++i) {
            const double xn = itr == 0 ? rnd() : x[(i + 1) * nz];
            if (us[i] != 0.0) {
              x[i * nz] = xn;
              xr = fma(-ul[i], xn, xr);
            } else {
              x[i * nz] = xr;
              xr = fma(-ul[i], xr, xn);
            }
          }
          double x1 = xr * u0[n - 1], x2 = 0.0;
          x[(n - 1) * nz] = x1;
          for (int i = n - 2; i >= 0; --i) {
            const double vv = fma(-u2[i], x2, fma(-u1[i], x1, x[i * nz])) * u0[i];
            x[i * nz] = vv;
            x2 = x1;
            x1 = vv;
          }
          for (int q = m0; q < mv; ++q) {  // re-orthogonalise against earlier members
            double dq = 0.0;
            for (int i = 0; i < n; ++i) dq = fma(Z[i * nz + q], x[i * nz], dq);
            for (int i = 0; i < n; ++i) x[i * nz] = fma(-dq, Z[i * nz + q], x[i * nz]);
          }
          // normalise (one solve from a unit vector grows it by at most
          // n / tiny, far inside the double range)
          double ss = 0.0;
          for (int i = 0; i < n; ++i) ss = fma(x[i * nz], x[i * nz], ss);
          const double sc = ss > 0.0 ? 1.0 / sqrt(ss) : 0.0;
          for (int i = 0; i < n; ++i) x[i * nz] *= sc;
        }
      }
    }
  }
  __syncthreads();
  ph_mark(ph, 4);
  // ---- back-transformation Z <- H_0 ... H_{n-3} Z in blocks of BT_NB
  // reflectors, each block as I - V T V^T (the compact WY form; T upper
  // triangular, T(0:c, c) = -tau_c T(0:c, 0:c) V(:, 0:c)^T v_c).  T of every
  // block first (a warp per block), then g lanes per column apply the blocks
  // from the last to the first with no barriers: a column belongs to one
  // lane group.
  {
    double* Z = S.Z;
    const int nr = n - 2;  // reflectors 0 .. n-3
    const int nblk = nr > 0 ? (nr + BT_NB - 1) / BT_NB : 0;
    auto vref = [&](int i, int kr) -> double {  // element i of reflector kr
      return i == kr + 1 ? 1.0 : (i > kr + 1 ? refl[i * (i + 1) / 2 + kr] : 0.0);
    };
    for (int blk = wp; blk < nblk; blk += BT_W) {
      double* T = S.tw + blk * BT_NB * BT_NB;
      const int kb = blk * BT_NB, nbb = min(BT_NB, nr - kb);
      for (int q = lane; q < BT_NB * BT_NB; q += 32) T[q] = 0.0;
      __syncwarp();
      // Gram entries V(:, j)^T v_c, j < c < nbb, one lane each
      for (int pq = lane; pq < BT_NB * (BT_NB - 1) / 2; pq += 32) {
        int c = 1, j = pq;
        while (j >= c) { j -= c; ++c; }
        if (c < nbb) {
          double g = 0.0;
          for (int i = kb + c + 1; i < n; ++i) g = fma(vref(i, kb + j), vref(i, kb + c), g);
          T[j * BT_NB + c] = g;
        }
      }
      __syncwarp();
      if (lane == 0) {
        for (int c = 0; c < nbb; ++c) {
          const double tc_ = S.tau[kb + c];
          double t[BT_NB];
#pragma unroll
          for (int j = 0; j < BT_NB; ++j) {
            double s = 0.0;
            if (j < c)
              for (int l = j; l < c; ++l) s = fma(T[j * BT_NB + l], T[l * BT_NB + c], s);
            t[j] = s;
          }
#pragma unroll
          for (int j = 0; j < BT_NB; ++j)
            if (j < c) T[j * BT_NB + c] = -tc_ * t[j];
          T[c * BT_NB + c] = tc_;
        }
      }
      __syncwarp();
    }
    __syncthreads();
    const int g = nz <= 32 ? 8 : (nz <= 64 ? 4 : 2);
    const int col = tid / g, gl = tid % g;
    const bool act = col < nz;
    for (int blk = nblk - 1; blk >= 0; --blk) {
      const double* T = S.tw + blk * BT_NB * BT_NB;
      const int kb = blk * BT_NB;
      double acc[BT_NB];
#pragma unroll
      for (int c = 0; c < BT_NB; ++c) acc[c] = 0.0;
      // rows kb+1 .. kb+BT_NB meet the reflectors' leading ones and zeros;
      // below them every element is a stored reflector entry.  Reflectors
      // past n-3 have zero T rows and columns and no stored entries here.
      if (act) {
        int i = kb + 1 + gl;
        for (; i < n && i <= kb + BT_NB; i += g) {
          const double z = Z[i * nz + col];
#pragma unroll
          for (int c = 0; c < BT_NB; ++c) acc[c] = fma(vref(i, kb + c), z, acc[c]);
        }
        for (; i < n; i += g) {
          const double z = Z[i * nz + col];
          const double* rr = refl + i * (i + 1) / 2 + kb;
#pragma unroll
          for (int c = 0; c < BT_NB; ++c) acc[c] = fma(rr[c], z, acc[c]);
        }
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1)
        if (o < g)
#pragma unroll
          for (int c = 0; c < BT_NB; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
      double wv[BT_NB];
#pragma unroll
      for (int c = 0; c < BT_NB; ++c) {
        double s = 0.0;
#pragma unroll
        for (int j = c; j < BT_NB; ++j) s = fma(T[c * BT_NB + j], acc[j], s);
        wv[c] = s;
      }
      if (act) {
        int i = kb + 1 + gl;
        for (; i < n && i <= kb + BT_NB; i += g) {
          double s = 0.0;
#pragma unroll
          for (int c = 0; c < BT_NB; ++c) s = fma(vref(i, kb + c), wv[c], s);
          Z[i * nz + col] -= s;
        }
        for (; i < n; i += g) {
          const double* rr = refl + i * (i + 1) / 2 + kb;
          double s = 0.0;
#pragma unroll
          for (int c = 0; c < BT_NB; ++c) s = fma(rr[c], wv[c], s);
          Z[i * nz + col] -= s;
        }
      }
    }
  }
  __syncthreads();
  ph_mark(ph, 5);
}

// cnvg (SCF/cnvg.F90:16-145) on the molecule's packed arrays; returns pl.
// The diagonal statistics run on thread 0 in the reference's order over
// copies staged in shared memory (S.d, S.e, S.e2, S.pv: free after the
// eigensolve); the off-diagonal extrapolation is elementwise.
__device__ double cta_cnvg(int n, double* pnew, double* p, double* p1, int niter, Smem& S) {
  double *xn = S.d, *xo = S.e, *x1 = S.e2, *pd = S.pv;
  for (int i = threadIdx.x; i < n; i += BT_T) {
    xn[i] = pnew[tri(i, i)];
    xo[i] = p[tri(i, i)];
    x1[i] = p1[i];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const bool extrap = (niter % 3) != 0;
    double pl = 0.0, faca = 0.0, facb = 0.0, sum1 = 0.0;
    for (int i = 0; i < n; ++i) {
      const double a = xn[i];
      sum1 = DADD(sum1, a);
      const double sa = fabs(DSUB(a, xo[i]));
      if (sa > pl) pl = sa;
      if (!extrap) {
        faca = DADD(faca, DMUL(sa, sa));
        const double t = DADD(DSUB(a, DMUL(2.0, xo[i])), x1[i]);
        facb = DADD(facb, DMUL(t, t));
      }
    }
    double fac = 0.0;
    if (facb > 1.0e-10 && faca < DMUL(100.0, facb)) fac = sqrt(faca / facb);
    // diagonal: damped extrapolation from the old diagonal (now P1), clamp, renormalise
    const double rhfuhf = 2.0;
    const double damp = (niter > 3) ? 0.05 : 1.0e10;
    double sum2 = 0.0;
    for (int i = 0; i < n; ++i) {
      double v = xn[i];
      const double dlt = DSUB(v, xo[i]);
      if (fabs(dlt) > damp) v = DADD(xo[i], copysign(damp, dlt));
      else v = DADD(v, DMUL(fac, dlt));
      const double t = v > 0.0 ? v : 0.0;
      v = t < rhfuhf ? t : rhfuhf;
      sum2 = DADD(sum2, v);
      pd[i] = v;
    }
    const double sum0 = sum1;
    for (int guard = 0; guard < 1000; ++guard) {
      const double sum = sum2 > 1.0e-3 ? sum1 / sum2 : 0.0;
      sum1 = sum0;
      if (sum2 < 1.0e-3 || fabs(DSUB(sum, 1.0)) < 1.0e-5) break;
      sum2 = 0.0;
      for (int i = 0; i < n; ++i) {
        double v = DADD(DMUL(pd[i], sum), 1.0e-20);
        v = v > 0.0 ? v : 0.0;
        if (v > rhfuhf) {
          v = rhfuhf;
          sum1 = DSUB(sum1, rhfuhf);
        } else {
          sum2 = DADD(sum2, v);
        }
        pd[i] = v;
      }
    }
    S.scal[8] = fac;
    S.scal[9] = pl;
  }
  __syncthreads();
  const double fac = S.scal[8];
  const int mp = n * (n + 1) / 2;
  for (int q = threadIdx.x; q < mp; q += BT_T) {
    int r, c;
    tri_rc(q, r, c);
    if (r == c) {
      p[q] = pd[r];
      pnew[q] = pd[r];
      p1[r] = xo[r];
    } else {
      const double a = pnew[q];
      const double v = DADD(a, DMUL(fac, DSUB(a, p[q])));
      p[q] = v;
      pnew[q] = v;
    }
  }
  __syncthreads();
  return S.scal[9];
}

// The molecule's F (packed, perturbed i*1e-10 in place as eigenvectors_LAPACK
// does) into S.A.
__device__ void load_perturbed(int n, double* f, Smem& S, bool in_place) {
  const int mp = n * (n + 1) / 2;
  if (in_place)
    for (int i = threadIdx.x; i < n; i += BT_T) {
      const long long k = tri(i, i);
      f[k] = DADD(f[k], DMUL((double)(i + 1), 1.0e-10));
    }
  __syncthreads();
  for (int q = threadIdx.x; q < mp; q += BT_T) {
    int r, c;
    tri_rc(q, r, c);
    S.A[q] = (r == c && !in_place) ? DADD(f[q], DMUL((double)(r + 1), 1.0e-10)) : f[q];
  }
  __syncthreads();
}

// P = 2 Z Z^T over the occupied vectors.
__device__ void cta_density(int n, int nz, const Smem& S, double* p) {
  const int mp = n * (n + 1) / 2;
  for (int q = threadIdx.x; q < mp; q += BT_T) {
    int r, c;
    tri_rc(q, r, c);
    double s = 0.0;
    for (int m = 0; m < nz; ++m) s = fma(S.Z[r * nz + m], S.Z[c * nz + m], s);
    p[q] = 2.0 * s;
  }
  __syncthreads();
}

template <int BT_NB>
__global__ void __launch_bounds__(BT_T, 2) scf_batch_kernel(BatchArgs B) {
  extern __shared__ double smem[];
  __shared__ int s_m, s_nitems;
  __shared__ long long s_ph[BT_PHASES + 1];
  const int tid = threadIdx.x;
  long long* ph = B.phase ? s_ph : nullptr;
  double* scr = B.scratch + (long long)blockIdx.x * BT_SCR;
  Smem S;
  S.A = smem;
  S.d = S.A + BT_AMAX;
  S.e = S.d + BT_NMAX;
  S.e2 = S.e + BT_NMAX;
  S.tau = S.e2 + BT_NMAX;
  S.pv = S.tau + BT_NMAX;
  S.v = S.pv + BT_NMAX;
  S.eig = S.v + BT_NMAX;
  S.red = S.eig + BT_NMAX + 2;
  S.scal = S.red + 2 * BT_W;
  S.tw = S.scal + 16;
  S.awrow = (long long*)(S.tw + bt_tw(BT_NB));
  S.afirst = (int*)(S.awrow + BT_NMAX);
  S.anor = S.afirst + BT_NMAX;
  S.acum = S.anor + BT_NMAX;
  S.orb_atom = S.acum + BT_NMAX;
  S.item = S.orb_atom + BT_NMAX;
  for (;;) {
    if (tid == 0) s_m = atomicAdd(B.next, 1);
    __syncthreads();
    const int m = s_m;
    __syncthreads();
    if (m >= B.nmol) break;
    const int mi = B.order[m];
    const Mol M = B.mol[mi];
    if (ph && tid == 0) {
      for (int q = 0; q < BT_PHASES; ++q) s_ph[q] = 0;
      s_ph[BT_PHASES] = clock64();
    }
    const int n = M.n, nclose = M.nclose;
    const int mp = n * (n + 1) / 2;
    S.Z = (n * nclose <= BT_AMAX) ? S.A : scr + BT_LU + BT_AMAX;
    // the molecule's atom tables
    for (int a = tid; a < M.numat; a += BT_T) {
      S.afirst[a] = B.first[M.aoff + a];
      S.anor[a] = B.nor[M.aoff + a];
      S.acum[a] = B.cum[M.aoff + a];
      S.awrow[a] = B.wrow[M.aoff + a];
    }
    __syncthreads();
    for (int a = tid; a < M.numat; a += BT_T)
      for (int o = 0; o < S.anor[a]; ++o) S.orb_atom[S.afirst[a] + o] = a;
    if (tid == 0) {
      int it = 0;
      for (int a = 0; a < M.numat; ++a) {
        const int nd = S.anor[a] * (S.anor[a] + 1) / 2;
        for (int q = 0; q < nd; ++q) S.item[it++] = (a << 4) | q;
      }
      s_nitems = it;
    }
    double* f = B.f + M.hoff;
    double* p = B.p + M.hoff;
    double* pold = B.pold + M.hoff;
    double* pold2 = B.pold2 + M.doff;
    const double* h = B.h + M.hoff;
    // ---- first-call setup (iter.F90:123-221): diagonal guess; PA = w1 * P
    const double w1 = (double)nclose / ((double)nclose + 1.0e-6 + (double)nclose);
    double cpa = w1;
    for (int q = tid; q < mp; q += BT_T) { p[q] = 0.0; pold[q] = 0.0; }
    __syncthreads();
    const int nitems = s_nitems;
    for (int i = tid; i < n; i += BT_T) {
      const long long j = tri(i, i);
      const double pd = B.pdiag[M.doff + i];
      p[j] = pd;
      pold[j] = DMUL(pd, w1);
      pold2[i] = pold[j];
    }
    __syncthreads();
    // control scalars: every thread holds the same copy
    double shift = 1.0, shfmax = 20.0, pl = 1.0, ten = -80.0, shfto = 0.0, shftbo = 0.0, shiftb = 0.0;
    const double bshift = -80.0, plchek = 0.005, trans = 0.2;
    bool newdg = false, oknewd = fabs(bshift) < 0.001;
    const double selcon = fmin(fmin(B.scfcrt * 100.0, 0.1), fmax(0.0, B.scfcrt));
    const double pltest = 0.05 * sqrt(fabs(selcon));
    int iredy = 1, niter = 0;
    double eold = 1.0e2, diff = 0.0, escf = 0.0, ee = 0.0, sellim = 0.0;
    bool ready = false, converged = false;
    double eig_homo = 0.0, eig_lumo = 0.0;
    const int ihomo = nclose > 1 ? nclose : 1;
    const double enrgy = PM7_FPC9;
    for (;;) {
      ++niter;
      if (niter > B.itrmax) break;
      bool use_shift = false;
      if (fabs(shift) > 1.0e-10 && bshift != 0.0) {
        if (niter > 1) {
          if (newdg) {
            if (diff > 0.0) { shift = 1.0; if (diff > 1) newdg = false; }
            else shift = -0.1;
          } else {
            shift = (ihomo < n) ? ten + eig_lumo - eig_homo + shift : 0.0;
          }
          if (diff > 0.0) {
            if (shift > 4.0) shfmax = 4.5;
            if (shift > shfmax) shfmax = fmax(shfmax - 0.5, 0.0);
          }
          shift = fmax(-20.0, fmin(shfmax, shift));
          if (fabs(shift - shfmax) < 1.0e-5) shfmax = shfmax + 0.01;
        }
        if (pl > plchek) { shftbo = shiftb; shfto = shift; }
        else { shiftb = shftbo; shift = shfto; }
        if (ihomo < n) eig_lumo = eig_lumo + shift;
        use_shift = true;
      }
      double cur_shift = shift;
      for (;;) {  // label 320
        ph_mark(ph, 7);
        cta_fock(B, M, S, nitems, cpa, cur_shift, use_shift, f, p, h);
        ph_mark(ph, 0);
        ee = cta_helect(n, p, cpa, h, f, S.red) * 2.0;
        escf = (ee + M.enuclr) * enrgy + M.atheat;
        diff = escf - eold;
        if (diff > 0) ten = ten - 1.0; else ten = ten * 0.975 + 0.05;
        sellim = fmax(selcon, 1.0e-15 * fmax(fabs(ee), 1.0));
        const bool conv = niter > 4 && (pl == 0.0 || (pl < pltest && fabs(diff) < sellim)) && ready;
        if (conv) {
          if (fabs(shift) < 1.0e-10) { converged = true; break; }
          shift = 0.0;
          shiftb = 0.0;
          use_shift = false;
          cur_shift = 0.0;
          continue;
        }
        break;
      }
      if (converged) break;
      ready = iredy > 0 && (fabs(diff) < sellim * 10.0 || pl == 0.0);
      ++iredy;
      eold = escf;
      ph_mark(ph, 1);
      load_perturbed(n, f, S, true);
      cta_eigh<BT_NB>(n, nclose, true, 1.0e-11, S, scr, ph);
      eig_homo = S.eig[ihomo - 1];
      eig_lumo = ihomo < n ? S.eig[ihomo] : 0.0;
      cta_density(n, nclose, S, p);
      ph_mark(ph, 6);
      pl = cta_cnvg(n, p, pold, pold2, niter, S);
      cpa = 0.5;
      if (!isfinite(pl)) break;
      oknewd = pl < sellim || oknewd;
      newdg = (pl < trans && oknewd) || newdg;
      if (pl < trans * 0.3333) oknewd = true;
    }
    // ---- label 600: final energy and the exit eigenvalues
    ph_mark(ph, 7);
    ee = cta_helect(n, p, cpa, h, f, S.red) * 2.0;
    load_perturbed(n, f, S, false);
    ph_mark(ph, 1);
    cta_eigh<BT_NB>(n, nclose, false, 4.4e-16, S, scr, ph);
    if (ph && tid == 0)
      for (int q = 0; q < BT_PHASES; ++q) atomicAdd(B.phase + q, (unsigned long long)s_ph[q]);
    if (tid == 0) {
      B.escf[mi] = (ee + M.enuclr) * enrgy + M.atheat;
      B.ee[mi] = ee;
      B.niter[mi] = niter;
      B.conv[mi] = converged ? 1 : 0;
      B.homo[mi] = S.eig[ihomo - 1];
      B.lumo[mi] = ihomo < n ? S.eig[ihomo] : 0.0;
    }
    __syncthreads();
  }
}

size_t batch_smem(int nb) {
  return sizeof(double) * ((size_t)BT_AMAX + 6 * BT_NMAX + BT_NMAX + 2 + 2 * BT_W + 16 + bt_tw(nb)) +
         sizeof(long long) * BT_NMAX + sizeof(int) * (4 * BT_NMAX + BT_IMAX);
}

// Kernel instance for a back-transformation block size (4, 8, 16).
const void* batch_kernel(int nb) {
  switch (nb) {
    case 4: return (const void*)scf_batch_kernel<4>;
    case 8: return (const void*)scf_batch_kernel<8>;
    case 16: return (const void*)scf_batch_kernel<16>;
    default: return nullptr;
  }
}

// Opts the instance into its dynamic shared memory and returns how many of
// its CTAs fit on one SM.
int batch_kernel_setup(int nb, int* per_sm) {
  const void* fn = batch_kernel(nb);
  if (!fn) return mb_set_error(MB_ERR_ARG, "batched SCF: block size must be 4, 8 or 16");
  const size_t smem = batch_smem(nb);
  MB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, fn, BT_T, smem));
  if (*per_sm < 1) return mb_set_error(MB_ERR_CUDA, "batched SCF kernel does not fit on an SM");
  return MB_OK;
}

}  // namespace

struct mb_batch {
  int nmol = 0;
  std::vector<Mol> hmol;
  Mol* mol = nullptr;
  int *order = nullptr, *first = nullptr, *nor = nullptr, *lim = nullptr, *cum = nullptr, *nat = nullptr, *next = nullptr,
      *niter = nullptr, *conv = nullptr, *status = nullptr;
  unsigned long long* phase = nullptr;
  bool timing = false;
  long long *wrow = nullptr, *offs = nullptr;  // offs: pair, atom prefixes (nmol + 1 each), hoff, woff
  double *coord = nullptr, *h = nullptr, *w = nullptr, *pdiag = nullptr, *f = nullptr, *p = nullptr,
         *pold = nullptr, *pold2 = nullptr, *scratch = nullptr, *escf = nullptr, *ee = nullptr, *homo = nullptr,
         *lumo = nullptr, *enuc = nullptr, *epairs = nullptr;
  long long tot_mp = 0, tot_w = 0;
  int tot_n = 0, tot_at = 0, grid = 0;
  int sms = 0, max_grid = 0;    // scratch is sized for max_grid CTAs
  int nb = 8, per_sm = 0;       // launch configuration (per_sm 0: as many as fit)
  // the run's launch sequence, captured once per configuration and replayed
  cudaGraphExec_t graph = nullptr;
  int g_nb = 0, g_grid = 0, g_timing = -1, g_itrmax = -1;
  double g_scfcrt = -1.0;
  cudaStream_t stream = nullptr;
};

static void batch_free(mb_batch* b) {
  if (!b) return;
  void* ptrs[] = {b->mol, b->order, b->first, b->nor, b->lim, b->cum, b->nat, b->next, b->niter, b->conv, b->status, b->wrow,
                  b->coord, b->h, b->w, b->pdiag, b->f, b->p, b->pold, b->pold2, b->scratch, b->escf, b->ee,
                  b->homo, b->lumo, b->enuc, b->epairs, b->phase, b->offs};
  if (b->graph) cudaGraphExecDestroy(b->graph);
  for (void* q : ptrs)
    if (q) cudaFree(q);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
}

extern "C" int mb_batch_create(int nmol, const int* numat, const int* nat, const double* coord, mb_batch** out) {
  if (nmol <= 0 || !numat || !nat || !coord || !out) return mb_set_error(MB_ERR_ARG, "mb_batch_create: bad args");
  *out = nullptr;
  static Pm7Params P;
  static bool pinit = false;
  if (!pinit) { pm7_init(&P); pinit = true; }
  mb_batch* b = new mb_batch();
  b->nmol = nmol;
  b->hmol.resize(nmol);
  std::vector<int> first, nor, lim, cum;
  std::vector<long long> wrow;
  std::vector<double> pdiag;
  long long hoff = 0, woff = 0, npair = 0;
  std::vector<long long> offs(4 * (size_t)nmol + 2);  // pair_off, atom_off, hoff, woff
  int aoff = 0, doff = 0;
  for (int m = 0; m < nmol; ++m) {
    Mol& M = b->hmol[m];
    const int na = numat[m];
    int ia = 0, nelec = 0, ncum = 0;
    double atheat = 0.0, eat = 0.0;
    long long wr = 0;
    std::vector<int> lm(na);
    for (int a = 0; a < na; ++a) {
      const int z = nat[aoff + a];
      if (!pm7_supported(z)) { batch_free(b); return mb_set_error(MB_ERR_UNSUPPORTED, "element outside H, C, O"); }
      const Pm7Elem& e = P.el[z];
      first.push_back(ia);
      nor.push_back(e.natorb);
      lm[a] = e.natorb == 1 ? 1 : 10;
      lim.push_back(lm[a]);
      cum.push_back(ncum);
      ncum += lm[a];
      for (int q = 0; q < e.natorb; ++q) pdiag.push_back(e.natorb == 1 ? e.tore : e.tore * 0.25);
      ia += e.natorb;
      nelec += (int)e.tore;
      atheat += e.eheat;
      eat += e.eisol;
    }
    // W: for atom a, its pair blocks with lower atoms (lim[a] x lim[b]) then its own block
    for (int a = 0; a < na; ++a) {
      wrow.push_back(wr);
      wr += (long long)lm[a] * (cum[aoff + a] + lm[a]);
    }
    if (nelec % 2 || ia > BT_NMAX || (long long)ia * (nelec / 2) > BT_ZMAX) {
      batch_free(b);
      return mb_set_error(MB_ERR_UNSUPPORTED, "batched SCF: closed shell, n <= 128 and n * nocc <= 11008 only");
    }
    M.n = ia;
    M.nclose = nelec / 2;
    M.numat = na;
    M.aoff = aoff;
    M.hoff = hoff;
    M.woff = woff;
    M.doff = doff;
    M.enuclr = 0.0;
    M.atheat = atheat - eat * PM7_FPC9;
    offs[m] = npair;
    offs[nmol + 1 + m] = aoff;
    offs[2 * nmol + 2 + m] = hoff;
    offs[3 * nmol + 2 + m] = woff;
    npair += (long long)na * (na - 1) / 2;
    hoff += (long long)ia * (ia + 1) / 2;
    woff += wr;
    doff += ia;
    aoff += na;
  }
  offs[nmol] = npair;
  offs[2 * nmol + 1] = aoff;
  b->tot_mp = hoff;
  b->tot_w = woff;
  b->tot_n = doff;
  b->tot_at = aoff;
  cudaError_t e = cudaSuccess;
#define BALLOC(ptr, bytes) if (e == cudaSuccess) e = cudaMalloc((void**)&(ptr), (bytes))
  BALLOC(b->mol, sizeof(Mol) * nmol);
  BALLOC(b->order, sizeof(int) * nmol);
  BALLOC(b->first, sizeof(int) * aoff);
  BALLOC(b->nor, sizeof(int) * aoff);
  BALLOC(b->lim, sizeof(int) * aoff);
  BALLOC(b->cum, sizeof(int) * aoff);
  BALLOC(b->wrow, sizeof(long long) * aoff);
  BALLOC(b->nat, sizeof(int) * aoff);
  BALLOC(b->coord, sizeof(double) * 3 * aoff);
  BALLOC(b->h, sizeof(double) * hoff);
  BALLOC(b->w, sizeof(double) * woff);
  BALLOC(b->pdiag, sizeof(double) * doff);
  BALLOC(b->f, sizeof(double) * hoff);
  BALLOC(b->p, sizeof(double) * hoff);
  BALLOC(b->pold, sizeof(double) * hoff);
  BALLOC(b->pold2, sizeof(double) * doff);
  BALLOC(b->escf, sizeof(double) * nmol);
  BALLOC(b->ee, sizeof(double) * nmol);
  BALLOC(b->homo, sizeof(double) * nmol);
  BALLOC(b->lumo, sizeof(double) * nmol);
  BALLOC(b->enuc, sizeof(double) * nmol);
  BALLOC(b->niter, sizeof(int) * nmol);
  BALLOC(b->conv, sizeof(int) * nmol);
  BALLOC(b->next, sizeof(int));
  BALLOC(b->status, sizeof(int));
  BALLOC(b->phase, sizeof(unsigned long long) * BT_PHASES);
  BALLOC(b->epairs, sizeof(double) * (npair + 1));
  BALLOC(b->offs, sizeof(long long) * offs.size());
#undef BALLOC
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMemcpy(b->first, first.data(), sizeof(int) * aoff, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->nor, nor.data(), sizeof(int) * aoff, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->lim, lim.data(), sizeof(int) * aoff, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->cum, cum.data(), sizeof(int) * aoff, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->wrow, wrow.data(), sizeof(long long) * aoff, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->nat, nat, sizeof(int) * aoff, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->coord, coord, sizeof(double) * 3 * aoff, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->pdiag, pdiag.data(), sizeof(double) * doff, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->offs, offs.data(), sizeof(long long) * offs.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    int r = mb_set_cuda_error(e, "mb_batch_create", __FILE__, __LINE__);
    batch_free(b);
    return r;
  }
  // integrals of every molecule on the GPU in three launches, then E_nuc
  {
    MbHcoreBatch hb;
    hb.nmol = nmol;
    hb.npair_tot = npair;
    hb.natom_tot = aoff;
    hb.pair_off = b->offs;
    hb.atom_off = b->offs + nmol + 1;
    hb.hoff = b->offs + 2 * nmol + 2;
    hb.woff = b->offs + 3 * nmol + 2;
    hb.nat = b->nat;
    hb.coord = b->coord;
    hb.first = b->first;
    hb.nor = b->nor;
    hb.lim = b->lim;
    hb.wrow = b->wrow;
    hb.cum = b->cum;
    hb.h = b->h;
    hb.w = b->w;
    hb.enuc_pairs = b->epairs;
    hb.enuclr = b->enuc;
    const int rc = mb_hcore_batch_dev(&hb, b->stream);
    if (rc != MB_OK) { batch_free(b); return rc; }
  }
  std::vector<double> en(nmol);
  e = cudaMemcpyAsync(en.data(), b->enuc, sizeof(double) * nmol, cudaMemcpyDeviceToHost, b->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
  if (e != cudaSuccess) {
    int r = mb_set_cuda_error(e, "mb_batch_create integrals", __FILE__, __LINE__);
    batch_free(b);
    return r;
  }
  for (int m = 0; m < nmol; ++m) b->hmol[m].enuclr = en[m];
  // molecules largest first, so the last wave is not a long one
  std::vector<int> order(nmol);
  for (int m = 0; m < nmol; ++m) order[m] = m;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return b->hmol[x].n > b->hmol[y].n; });
  e = cudaMemcpy(b->mol, b->hmol.data(), sizeof(Mol) * nmol, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->order, order.data(), sizeof(int) * nmol, cudaMemcpyHostToDevice);
  int dev = 0, sms = 0, per = 0, maxper = 0;
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) {
    int r = mb_set_cuda_error(e, "mb_batch_create kernel setup", __FILE__, __LINE__);
    batch_free(b);
    return r;
  }
  for (int nb : {4, 16, 8}) {  // the default (8) last: its attribute stays set
    int rc = batch_kernel_setup(nb, &per);
    if (rc != MB_OK) {
      batch_free(b);
      return rc;
    }
    maxper = std::max(maxper, per);
  }
  b->sms = sms;
  b->nb = 8;
  b->grid = std::min(nmol, sms * per);
  b->max_grid = std::min(nmol, sms * maxper);
  e = cudaMalloc((void**)&b->scratch, sizeof(double) * BT_SCR * (size_t)b->max_grid);
  if (e != cudaSuccess) {
    int r = mb_set_cuda_error(e, "mb_batch_create scratch", __FILE__, __LINE__);
    batch_free(b);
    return r;
  }
  *out = b;
  return MB_OK;
}

extern "C" int mb_batch_destroy(mb_batch* b) {
  if (b) {
    cudaStreamSynchronize(b->stream);
    batch_free(b);
  }
  return MB_OK;
}

extern "C" int mb_batch_nmol(const mb_batch* b) { return b ? b->nmol : 0; }

extern "C" int mb_batch_run(mb_batch* b, const mb_scf_opts* opts_in, double* escf, int* niter, int* converged,
                            double* t_ms) {
  if (!b) return mb_set_error(MB_ERR_ARG, "mb_batch_run: null batch");
  mb_scf_opts o;
  if (opts_in) o = *opts_in; else mb_scf_opts_default(&o);
  BatchArgs A;
  A.mol = b->mol;
  A.order = b->order;
  A.nmol = b->nmol;
  A.first = b->first;
  A.nor = b->nor;
  A.h = b->h;
  A.w = b->w;
  A.wrow = b->wrow;
  A.cum = b->cum;
  A.pdiag = b->pdiag;
  A.f = b->f;
  A.p = b->p;
  A.pold = b->pold;
  A.pold2 = b->pold2;
  A.scratch = b->scratch;
  A.escf = b->escf;
  A.ee = b->ee;
  A.niter = b->niter;
  A.conv = b->conv;
  A.homo = b->homo;
  A.lumo = b->lumo;
  A.next = b->next;
  A.phase = b->timing ? b->phase : nullptr;
  if (b->timing) MB_CUDA(cudaMemsetAsync(b->phase, 0, sizeof(unsigned long long) * BT_PHASES, b->stream));
  A.itrmax = o.itrmax;
  A.scfcrt = o.scfcrt;
  // The launch sequence (clear the work counter, the persistent kernel) is
  // captured into a CUDA graph once per configuration and replayed.
  const int timing = b->timing ? 1 : 0;
  if (!b->graph || b->g_nb != b->nb || b->g_grid != b->grid || b->g_timing != timing || b->g_itrmax != o.itrmax ||
      b->g_scfcrt != o.scfcrt) {
    if (b->graph) {
      cudaGraphExecDestroy(b->graph);
      b->graph = nullptr;
    }
    void* args[] = {&A};
    cudaGraph_t g = nullptr;
    MB_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    cudaError_t ce = cudaMemsetAsync(b->next, 0, sizeof(int), b->stream);
    if (ce == cudaSuccess)
      ce = cudaLaunchKernel(batch_kernel(b->nb), dim3(b->grid), dim3(BT_T), args, batch_smem(b->nb), b->stream);
    cudaError_t ee = cudaStreamEndCapture(b->stream, &g);
    if (ce == cudaSuccess) ce = ee;
    if (ce == cudaSuccess) ce = cudaGraphInstantiate(&b->graph, g, 0);
    if (g) cudaGraphDestroy(g);
    if (ce != cudaSuccess) {
      b->graph = nullptr;
      return mb_set_cuda_error(ce, "mb_batch_run graph capture", __FILE__, __LINE__);
    }
    b->g_nb = b->nb;
    b->g_grid = b->grid;
    b->g_timing = timing;
    b->g_itrmax = o.itrmax;
    b->g_scfcrt = o.scfcrt;
  }
  cudaEvent_t e0, e1;
  MB_CUDA(cudaEventCreate(&e0));
  MB_CUDA(cudaEventCreate(&e1));
  MB_CUDA(cudaEventRecord(e0, b->stream));
  MB_CUDA(cudaGraphLaunch(b->graph, b->stream));
  MB_LAUNCH_CHECK();
  MB_CUDA(cudaEventRecord(e1, b->stream));
  MB_CUDA(cudaEventSynchronize(e1));
  float ms = 0.f;
  MB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (t_ms) *t_ms = ms;
  if (escf) MB_CUDA(cudaMemcpy(escf, b->escf, sizeof(double) * b->nmol, cudaMemcpyDeviceToHost));
  if (niter) MB_CUDA(cudaMemcpy(niter, b->niter, sizeof(int) * b->nmol, cudaMemcpyDeviceToHost));
  if (converged) MB_CUDA(cudaMemcpy(converged, b->conv, sizeof(int) * b->nmol, cudaMemcpyDeviceToHost));
  return MB_OK;
}

extern "C" int mb_batch_set_config(mb_batch* b, int nb, int per_sm) {
  if (!b) return mb_set_error(MB_ERR_ARG, "mb_batch_set_config: null batch");
  int per = 0;
  MB_TRY(batch_kernel_setup(nb, &per));
  if (per_sm < 0) return mb_set_error(MB_ERR_ARG, "mb_batch_set_config: per_sm < 0");
  const int use = per_sm == 0 ? per : std::min(per_sm, per);
  b->nb = nb;
  b->per_sm = per_sm;
  b->grid = std::min({b->nmol, b->sms * use, b->max_grid});
  return MB_OK;
}

extern "C" int mb_batch_get_config(const mb_batch* b, int* nb, int* grid) {
  if (!b) return mb_set_error(MB_ERR_ARG, "mb_batch_get_config: null batch");
  if (nb) *nb = b->nb;
  if (grid) *grid = b->grid;
  return MB_OK;
}

// Times every configuration (block size 4, 8, 16 x one or as many CTAs per
// SM as fit) on this batch -- one untimed and one timed run each -- and keeps
// the fastest.  Every configuration computes the same SCFs (the block size
// only regroups the back-transformation's FP64 sums).
extern "C" int mb_batch_autotune(mb_batch* b, const mb_scf_opts* opts, int* nb_out, int* per_sm_out,
                                 double* ms_out) {
  if (!b) return mb_set_error(MB_ERR_ARG, "mb_batch_autotune: null batch");
  double best = 1e300;
  int bnb = 8, bper = 0;
  for (int nb : {4, 8, 16})
    for (int per : {1, 0}) {
      MB_TRY(mb_batch_set_config(b, nb, per));
      double ms = 0.0;
      MB_TRY(mb_batch_run(b, opts, nullptr, nullptr, nullptr, &ms));
      MB_TRY(mb_batch_run(b, opts, nullptr, nullptr, nullptr, &ms));
      if (ms < best) {
        best = ms;
        bnb = nb;
        bper = per;
      }
    }
  MB_TRY(mb_batch_set_config(b, bnb, bper));
  if (nb_out) *nb_out = bnb;
  if (per_sm_out) *per_sm_out = bper;
  if (ms_out) *ms_out = best;
  return MB_OK;
}

extern "C" int mb_batch_set_phase_timing(mb_batch* b, int on) {
  if (!b) return mb_set_error(MB_ERR_ARG, "mb_batch_set_phase_timing: null batch");
  b->timing = on != 0;
  return MB_OK;
}

extern "C" int mb_batch_phase_cycles(mb_batch* b, unsigned long long* out) {
  if (!b || !out) return mb_set_error(MB_ERR_ARG, "mb_batch_phase_cycles: bad args");
  MB_CUDA(cudaMemcpy(out, b->phase, sizeof(unsigned long long) * BT_PHASES, cudaMemcpyDeviceToHost));
  return MB_OK;
}

extern "C" int mb_batch_get_density(mb_batch* b, int m, double* p) {
  if (!b || m < 0 || m >= b->nmol || !p) return mb_set_error(MB_ERR_ARG, "mb_batch_get_density: bad args");
  const Mol& M = b->hmol[m];
  MB_CUDA(cudaMemcpy(p, b->p + M.hoff, sizeof(double) * (size_t)M.n * (M.n + 1) / 2, cudaMemcpyDeviceToHost));
  return MB_OK;
}

extern "C" int mb_batch_get_hw(mb_batch* b, int m, double* h, double* w, double* enuclr) {
  if (!b || m < 0 || m >= b->nmol) return mb_set_error(MB_ERR_ARG, "mb_batch_get_hw: bad args");
  const Mol& M = b->hmol[m];
  const long long wlen = (m + 1 < b->nmol ? b->hmol[m + 1].woff : b->tot_w) - M.woff;
  if (h) MB_CUDA(cudaMemcpy(h, b->h + M.hoff, sizeof(double) * (size_t)M.n * (M.n + 1) / 2, cudaMemcpyDeviceToHost));
  if (w) MB_CUDA(cudaMemcpy(w, b->w + M.woff, sizeof(double) * (size_t)wlen, cudaMemcpyDeviceToHost));
  if (enuclr) *enuclr = M.enuclr;
  return MB_OK;
}
