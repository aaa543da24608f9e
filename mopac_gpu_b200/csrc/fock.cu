// Two- and one-centre Fock build for the dense NDDO SCF (sp basis).
//
// Replaces fock2 (SCF/fock2.F90:16-374, sp branches :149-298), jab
// (integrals/jab.F90), kab (integrals/kab.F90) and fock1 (SCF/fock1.F90) as
// called from iter (SCF/iter.F90:553), including iter's level-shifted start
// value F = H + shift*PA + 1e-16*i, F_ii -= shift (SCF/iter.F90:317-324).
//
// Result is bit-identical to the reference loop order: every element of F
// receives its contributions in the same sequence (partner atoms in ascending
// order with the one-centre term at the atom's own position), each
// contribution is formed with the same term order, and no FMA is used.
//
// Design: two passes over a staging array.
//
// Pass 1 (fock2_pairs) evaluates every atom pair once, one pair per lane: its
// exchange block goes straight to F, and the Coulomb contributions that need a
// sum over a heavy atom's density go to the staging array.  Work is a queue of
// warp items, taken with an atomic counter:
//   HH  heavy A, 32 heavy partners below it: the 10 x 10 W blocks stream
//       through the warp as ten row tiles, used in the order of jab's density gather
//       (row pair(x, y) at step 4x + y).  That order is also kab's (mu, lam)
//       order and that of the terms of the partner's elements, so the exchange
//       sums and both atoms' Coulomb sums keep the reference's term sequence
//       with one W row live per lane.
//   HX  heavy A, 128 light partners, four tiles of one ten-double block per lane.
//   LL  light A, the light partners below it: exchange only.
// A tile (32 lanes x ten doubles) is copied with cp.async by the whole
// warp over the concatenated blocks -- consecutive lanes copy consecutive
// addresses -- into per-lane slots of 11 doubles (odd, so the lanes' reads
// hit distinct banks), all of an item's tiles at once.
//
// Pass 2 (fock2_fold) runs one CTA per atom: it streams the contributions of
// the atom's partners through shared memory in partner order, and up to ten
// owner threads fold them into iter's start value, adding fock1's one-centre
// term at the atom's own position.  A light partner's contribution is its
// density times its W block, which is read in place of a staged record of the
// same size.  A light atom's two values per partner are fock2's one or two
// additions; an absent second addition is -0.0, which leaves every sum unchanged
// bit for bit.
//
// Bound by sectors through L1: blocks, density and F in runs of 8 to 80 bytes.
// (H2O)333, one B200: 65 us for the pairs and 30 for the fold; with every ordered
// pair evaluated and staged, 122 and 19, and 5 for the lists in one CTA.
#include <cstdint>
#include <mutex>

#include "mb_common.cuh"

namespace {

constexpr int kWarps = 2;          // warps per CTA of the pair pass, four CTAs an SM
constexpr int kRows = 10;          // tiles per warp: the rows of a W block
constexpr int kSlot = 11;          // doubles per lane slot in a tile
constexpr int kTile = 32 * kSlot;  // doubles per tile
constexpr int kStageW = 10;        // staged doubles per (A, heavy B) record of a heavy A (a light A uses 2)
constexpr int kFoldThreads = 128;  // pass 2: threads per CTA; one warp folds, the others fetch
constexpr int kChunk = kFoldThreads - 32;  // pass 2: partners per chunk, one a fetching thread
constexpr int kFoldDepth = 3;      // pass 2: chunk buffers: one folded, two on their way

__host__ __device__ constexpr int pair1(int a, int b) {  // 1-based pair index of orbitals a, b (1..4)
  return a > b ? a * (a - 1) / 2 + b : b * (b - 1) / 2 + a;
}

// jab's density gather: term m uses pair index pair1(m / 4 + 1, m % 4 + 1).
__host__ __device__ constexpr int pidx(int m) { return pair1(m / 4 + 1, m % 4 + 1); }
// How many rows the gather visits first before term m (m / 4 <= m % 4).
__host__ __device__ constexpr int first_visit(int m) {
  int n = 0;
  for (int k = 0; k < m; ++k) n += k / 4 <= k % 4;
  return n;
}

__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

// Wait until at most N of this thread's committed groups are pending.
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
// The same for an n known after unrolling, n < kRows.
__device__ __forceinline__ void cp_async_wait(int n) {
  switch (n) {
    case 0: cp_async_wait<0>(); break;
    case 1: cp_async_wait<1>(); break;
    case 2: cp_async_wait<2>(); break;
    case 3: cp_async_wait<3>(); break;
    case 4: cp_async_wait<4>(); break;
    case 5: cp_async_wait<5>(); break;
    case 6: cp_async_wait<6>(); break;
    case 7: cp_async_wait<7>(); break;
    case 8: cp_async_wait<8>(); break;
    default: cp_async_wait<9>(); break;
  }
}

struct FockArgs {
  MbAtoms at;
  double* f;
  const double* h;
  const double* ptot;
  const double* pa;
  const double* w;
  double shift;
  int use_shift;
};

// Workspace: counts (heavy atoms, light atoms, item counter), the heavy and
// light atom lists (ascending), and the staging array.
struct FockWs {
  int* counts;
  int* hlist;
  int* llist;
  double* stage;
};

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

FockWs carve(void* ws, int numat) {
  char* p = (char*)ws;
  FockWs r;
  r.counts = (int*)p;
  p += 256;
  r.hlist = (int*)p;
  p += align256(sizeof(int) * (size_t)numat);
  r.llist = (int*)p;
  p += align256(sizeof(int) * (size_t)numat);
  r.stage = (double*)p;
  return r;
}

// Staged record of the rank-th heavy atom for atom A: a heavy A's ten values or a
// light A's two.
__device__ __forceinline__ long long rec_off(int A, int numat, int rank, bool heavy) {
  return (long long)A * numat * kStageW + (long long)rank * (heavy ? kStageW : 2);
}

// Heavy atoms below atom A: cum counts ten pairs for each of them and one for a
// light atom.  (first is no measure of it: orbitals may begin anywhere and leave gaps.)
__device__ __forceinline__ int heavy_below(const MbAtoms& at, int A) { return (__ldg(at.cum + A) - A) / 9; }

__device__ __forceinline__ double f_start(const FockArgs& a, long long idx, bool diag) {
  if (!a.use_shift) return __ldg(a.h + idx);
  double v = DADD(DADD(__ldg(a.h + idx), DMUL(a.shift, __ldg(a.pa + idx))), DMUL((double)(idx + 1), 1.0e-16));
  if (diag) v = DSUB(v, a.shift);
  return v;
}

// f_start with PA(idx) already in a register.
__device__ __forceinline__ double f_start_pa(const FockArgs& a, long long idx, double pa_idx) {
  if (!a.use_shift) return __ldg(a.h + idx);
  return DADD(DADD(__ldg(a.h + idx), DMUL(a.shift, pa_idx)), DMUL((double)(idx + 1), 1.0e-16));
}

// Heavy atom B's diagonal density block in jab's 4 x 4 gather order,
// pjb[x*4 + y] = P(max, min).
__device__ __forceinline__ void diag_block(const FockArgs& a, int fB, double* pjb) {
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const int r = fB + (x > y ? x : y), cc = fB + (x < y ? x : y);
      pjb[x * 4 + y] = __ldg(a.ptot + mb_tri(r, cc));
    }
}

// Warp-cooperative tile copy: 32 windows of ten doubles, window i at
// src[i] + add, land in slots 0..31.  Flat element q = 32r + lane of round r
// is element q % 10 of window q / 10, so consecutive lanes copy consecutive
// addresses of one window or the next.  Called by all 32 lanes.
__device__ __forceinline__ void issue_win10(double* tile, const unsigned long long* src, long long add, int lane) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const int q = 32 * r + lane;
    const int i = q / 10, e = q - 10 * i;
    cp_async8(tile + i * kSlot + e, (const double*)src[i] + add + e);
  }
}

// W block of the ordered pair (A, B): for B < A the lA x lB block of row A
// (B's pair index fastest), else the lB x lA block of row B.
__device__ __forceinline__ const double* w_block(const FockArgs& a, int A, int lA, long long wrowA, int B,
                                                 int lB) {
  return B < A ? a.w + wrowA + (long long)lA * __ldg(a.at.cum + B)
               : a.w + __ldg(a.at.wrow + B) + (long long)lB * __ldg(a.at.cum + A);
}

// The light atoms' densities, in their order: atom 0's staged records leave the
// room behind the heavy atoms' ten free.
__device__ __forceinline__ double* light_density(const FockWs& ws, int nh) { return ws.stage + (long long)nh * kStageW; }

// Heavy and light atom lists (ascending), their lengths, the light atoms'
// densities, and a zero item counter for the pair pass.
__global__ void fock2_lists(MbAtoms at, const double* __restrict__ ptot, FockWs ws) {
  const int A = blockIdx.x * blockDim.x + threadIdx.x;
  if (A >= at.numat) return;
  const int nh = heavy_below(at, A);
  const bool heavy = at.nor[A] == 4;
  if (heavy) ws.hlist[nh] = A;
  else ws.llist[A - nh] = A;
  if (!heavy) {
    const int last = at.numat - 1, all = heavy_below(at, last) + (at.nor[last] == 4), f = __ldg(at.first + A);
    light_density(ws, all)[A - nh] = __ldg(ptot + mb_tri(f, f));
  }
  if (A == at.numat - 1) {
    ws.counts[0] = nh + heavy;
    ws.counts[1] = at.numat - nh - heavy;
    ws.counts[2] = 0;
  }
}

__global__ void __launch_bounds__(32 * kWarps, 4) fock2_pairs(FockArgs a, FockWs ws) {
  extern __shared__ double s_tiles[];  // kWarps x kRows tiles
  __shared__ unsigned long long s_src[kWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* tiles = s_tiles + (size_t)warp * kRows * kTile;
  const int numat = a.at.numat;
  const int nh = ws.counts[0], nl = ws.counts[1];
  const int th = (nh + 31) / 32, tl = (nl + 127) / 128;
  const long long r1 = (long long)th * (th + 1) / 2 * 32, r2 = r1 + (long long)nh * tl, total = r2 + nl;

  for (;;) {
    long long item = 0;
    if (lane == 0) item = atomicAdd(&ws.counts[2], 1);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= total) break;

    // HH items and the others in turn, so that loading and computing warps share an
    // SM: (H2O)333 78 -> 67 us
    const long long both = 2 * min(r1, total - r1);
    if (item < both) item = (item & 1) ? r1 + (item >> 1) : item >> 1;
    else if (2 * r1 > both) item = item - (both >> 1);
    if (item < r1) {
      // HH: heavy atom i = 32 I + item % 32 and its partners 32 J + lane < i, J <= I;
      // W rows through the tile ring
      const int tile = (int)(item / 32);
      int I = (int)((sqrtf(8.0f * (float)tile + 1.0f) - 1.0f) * 0.5f);
      while (I * (I + 1) / 2 > tile) --I;
      while ((I + 1) * (I + 2) / 2 <= tile) ++I;
      const int J = tile - I * (I + 1) / 2;
      const int i = 32 * I + (int)(item % 32), j = 32 * J + lane;
      if (i >= nh || 32 * J >= i) continue;
      const bool act = j < i;
      const int A = __ldg(ws.hlist + i), B = act ? __ldg(ws.hlist + j) : A;
      const int fA = __ldg(a.at.first + A), fB = __ldg(a.at.first + B);
      s_src[warp][lane] =
          (unsigned long long)(act ? a.w + __ldg(a.at.wrow + A) + 10LL * __ldg(a.at.cum + B) : a.w);
      __syncwarp();
#pragma unroll
      for (int m = 0; m < 16; ++m)
        if (m / 4 <= m % 4) {  // a row at its first visit
          issue_win10(tiles + (pidx(m) - 1) * kTile, s_src[warp], (pidx(m) - 1) * 10, lane);
          cp_async_commit();
        }
      double* recA = ws.stage + rec_off(A, numat, j, true);
      double pj[16], pk[16], hm[4], sa[4], sb[10];
      // A's density block in jab's gather order, term m on lane m
      const int gx = (lane & 15) / 4, gy = lane & 3;
      const double pi = __ldg(a.ptot + mb_tri(fA + max(gx, gy), fA + min(gx, gy)));
      if (act) {
        diag_block(a, fB, pj);
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int y = 0; y < 4; ++y) pk[x * 4 + y] = __ldg(a.pa + (mb_tri(fA + x, fB + y)));
      }
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const int x = m / 4, y = m % 4;
        if (act && y == 0) {
#pragma unroll
          for (int nu = 0; nu < 4; ++nu) hm[nu] = __ldg(a.h + (mb_tri(fA + x, fB + nu)));
        }
        if (x <= y) {
          cp_async_wait(kRows - 1 - first_visit(m));
          __syncwarp();
        }
        const double* row = tiles + (pidx(m) - 1) * kTile + lane * kSlot;  // row pidx(m) of the block
        const double pim = __shfl_sync(0xffffffffu, pi, m);
        if (act) {
          double w[10];
#pragma unroll
          for (int q = 0; q < 10; ++q) w[q] = row[q];
          if (x <= y) {  // first visit of row pidx(m): A's Coulomb term for that pair index
            double sum = DMUL(pj[0], w[pidx(0) - 1]);
#pragma unroll
            for (int mm = 1; mm < 16; ++mm) sum = DADD(sum, DMUL(pj[mm], w[pidx(mm) - 1]));
            recA[pidx(m) - 1] = sum;
          }
          // term m of each of B's ten elements
#pragma unroll
          for (int q = 0; q < 10; ++q) {
            const double tt = DMUL(pim, w[q]);
            sb[q] = m == 0 ? tt : DADD(sb[q], tt);
          }
          // kab: this row is pair(mu, lam) with mu = x + 1, lam = y + 1
#pragma unroll
          for (int nu = 1; nu <= 4; ++nu)
#pragma unroll
            for (int sig = 1; sig <= 4; ++sig) {
              const double tt = DMUL(pk[y * 4 + sig - 1], w[pair1(nu, sig) - 1]);
              sa[nu - 1] = (y == 0 && sig == 1) ? tt : DADD(sa[nu - 1], tt);
            }
          if (y == 3) {
#pragma unroll
            for (int nu = 0; nu < 4; ++nu) {
              const long long idx = mb_tri(fA + x, fB + nu);
              const double st = a.use_shift
                                    ? DADD(DADD(hm[nu], DMUL(a.shift, pk[x * 4 + nu])), DMUL((double)(idx + 1), 1.0e-16))
                                    : hm[nu];
              a.f[idx] = DSUB(st, sa[nu]);
            }
          }
        }
      }
      __syncwarp();
      if (act) {
        double2* recB = (double2*)(ws.stage + rec_off(B, numat, i, true));
#pragma unroll
        for (int q = 0; q < 5; ++q) recB[q] = make_double2(sb[2 * q], sb[2 * q + 1]);
      }
    } else if (item < r2) {
      // HX: heavy A, light partners llist[128 t + 32 g + lane]; one ten-double block each
      const long long k = item - r1;
      const int rank = (int)(k / tl), A = __ldg(ws.hlist + rank);
      const int base = (int)(k % tl) * 128;
      const int fA = __ldg(a.at.first + A);
      const long long wrowA = __ldg(a.at.wrow + A);
      unsigned long long* src = (unsigned long long*)(tiles + 4 * kTile);
      int Bs[4];
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int idx = base + 32 * g + lane;
        const int B = idx < nl ? __ldg(ws.llist + idx) : -1;
        Bs[g] = B;
        // the last tiles of an HX item are free: the windows' addresses
        src[g * 32 + lane] = (unsigned long long)(B >= 0 ? w_block(a, A, 10, wrowA, B, 1) : a.w);
      }
      __syncwarp();
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        issue_win10(tiles + g * kTile, src + g * 32, 0, lane);
        cp_async_commit();
      }
      double pi[10];  // A's diagonal density block, packed
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y <= x; ++y) pi[x * (x + 1) / 2 + y] = __ldg(a.ptot + mb_tri(fA + x, fA + y));
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int B = Bs[g];
        double pj[4], hs[4];
        long long idx[4];
        if (B >= 0) {
          const int fB = __ldg(a.at.first + B);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            idx[q] = B < A ? mb_tri(fA + q, fB) : mb_tri(fB, fA + q);
            pj[q] = __ldg(a.pa + idx[q]);
            hs[q] = f_start_pa(a, idx[q], pj[q]);
          }
        }
        cp_async_wait(3 - g);
        __syncwarp();
        if (B >= 0) {
          const double* wk = tiles + g * kTile + lane * kSlot;
          // B's two additions (fock2's "ib - ia >= 3" / "jb - ja >= 3" branches)
          double sumoff = 0.0, sumdia = 0.0;
#pragma unroll
          for (int x = 0; x < 4; ++x) {
#pragma unroll
            for (int y = 0; y < x; ++y) sumoff = DADD(sumoff, DMUL(pi[x * (x + 1) / 2 + y], wk[x * (x + 1) / 2 + y]));
            sumdia = DADD(sumdia, DMUL(pi[x * (x + 1) / 2 + x], wk[x * (x + 1) / 2 + x]));
          }
          *(double2*)(ws.stage + rec_off(B, numat, rank, false)) = make_double2(DMUL(sumoff, 2.0), sumdia);
          // kab on the 4 x 1 or 1 x 4 block
#pragma unroll
          for (int x = 1; x <= 4; ++x) {
            double sum = 0.0;
#pragma unroll
            for (int y = 1; y <= 4; ++y) sum = DADD(sum, DMUL(pj[y - 1], wk[pair1(x, y) - 1]));
            a.f[idx[x - 1]] = DSUB(hs[x - 1], sum);
          }
        }
      }
      __syncwarp();
    } else {
      // LL: light A, the light partners below it
      const int k = (int)(item - r2), A = __ldg(ws.llist + k);
      const double* row = a.w + __ldg(a.at.wrow + A);
      const long long f0 = mb_tri(__ldg(a.at.first + A), 0);
#pragma unroll 4
      for (int l = lane; l < k; l += 32) {
        const int B = __ldg(ws.llist + l);
        const long long idx = f0 + __ldg(a.at.first + B);
        const double pab = __ldg(a.pa + idx);
        a.f[idx] = DSUB(f_start_pa(a, idx, pab), DMUL(pab, __ldg(row + __ldg(a.at.cum + B))));
      }
    }
  }
}

// Pass 2: one CTA per atom; owners e < lim[A] fold in partner order, the chain of
// additions being the least time this takes.  In step k, one warp folds chunk
// k - 2 while the other warps copy chunk k, whose addresses they found in step k - 1,
// and find those of chunk k + 1.
__global__ void __launch_bounds__(kFoldThreads) fock2_fold(FockArgs a, FockWs ws) {
  extern __shared__ double s_buf[];  // kFoldDepth chunks of kChunk records
  __shared__ const double* s_src[2][kChunk];
  __shared__ double s_fac[kFoldDepth][kChunk];  // a light partner's density, 1 for a staged record
  const int A = blockIdx.x, tid = threadIdx.x, pt = tid - 32;
  const int numat = a.at.numat;
  const int fA = __ldg(a.at.first + A), nA = __ldg(a.at.nor + A), lA = __ldg(a.at.lim + A);
  const bool heavy = nA == 4;
  const long long wrowA = __ldg(a.at.wrow + A);
  const int cA = __ldg(a.at.cum + A);
  const double* pl = light_density(ws, ws.counts[0]);

  double run = 0.0, f1 = 0.0;
  long long own_idx = 0;
  if (tid < lA) {
    int iw = 1, jw = 1;  // local (row, col), 1-based, from packed element tid
    {
      int e = tid, r = 1;
      while (e >= r) { e -= r; ++r; }
      iw = r; jw = e + 1;
    }
    own_idx = mb_tri(fA + iw - 1, fA + jw - 1);
    run = f_start(a, own_idx, iw == jw);
    // fock1 (SCF/fock1.F90): one-centre Coulomb and exchange for element (iw, jw)
    const double* w1 = a.w + wrowA + (long long)lA * cA;
    const int ilim = lA;
    const int ijw = iw * (iw - 1) / 2 + jw;
    double sum = 0.0;
#pragma unroll
    for (int kw = 1; kw <= 4; ++kw)
#pragma unroll
      for (int lw = 1; lw <= 4; ++lw) {
        if (kw > nA || lw > nA) continue;
        int ip = kw > lw ? kw : lw, jp = kw < lw ? kw : lw;
        long long ijp = mb_tri(fA + ip - 1, fA + jp - 1);
        int klw = ip * (ip - 1) / 2 + jp;
        int im = kw > jw ? kw : jw, jm = kw < jw ? kw : jw;
        int ikw = im * (im - 1) / 2 + jm;
        im = lw > iw ? lw : iw; jm = lw < iw ? lw : iw;
        int jlw = im * (im - 1) / 2 + jm;
        sum = DSUB(DADD(sum, DMUL(__ldg(a.ptot + ijp), w1[(ijw - 1) + ilim * (klw - 1)])),
                   DMUL(__ldg(a.pa + ijp), w1[(ikw - 1) + ilim * (jlw - 1)]));
      }
    f1 = sum;
  }

  const int nchunk = (numat + kChunk - 1) / kChunk;
  const double* src = a.w;  // this thread's partner of chunk k, and its factor
  double fac = 1.0;
  bool staged = false;
  auto find = [&](int k) {
    const int B = k * kChunk + pt;
    src = a.w;
    fac = 1.0;
    staged = false;
    if (k < nchunk && B < numat && B != A) {
      const int hB = heavy_below(a.at, B);
      staged = __ldg(a.at.nor + B) == 4;
      if (staged) src = ws.stage + rec_off(A, numat, hB, heavy);
      else src = B < A ? a.w + wrowA + (long long)lA * __ldg(a.at.cum + B) : a.w + __ldg(a.at.wrow + B) + cA;
      if (!staged) fac = __ldg(pl + (B - hB));
    }
    s_src[k & 1][pt] = src;
  };
  if (pt >= 0) find(0);
  __syncthreads();
  for (int k = 0; k < nchunk + 2; ++k) {
    if (pt >= 0) {
      if (k < nchunk) {
        double* dst = s_buf + (k % kFoldDepth) * kChunk * kStageW;
        s_fac[k % kFoldDepth][pt] = fac;
        if (heavy) {
          const int n = min(kChunk, numat - k * kChunk) * kStageW;
          for (int q = pt; q < n; q += kChunk) cp_async8(dst + q, s_src[k & 1][q / kStageW] + q % kStageW);
        } else {
          cp_async8(dst + 2 * pt, src);
          if (staged) cp_async8(dst + 2 * pt + 1, src + 1);
          else dst[2 * pt + 1] = -0.0;
        }
      }
      cp_async_commit();
      find(k + 1);
      cp_async_wait(1);  // chunk k - 1 is here
    } else if (k >= 2 && tid < lA) {
      const int c = k - 2;
      const double* buf = s_buf + (c % kFoldDepth) * kChunk * kStageW;
      const double* fc = s_fac[c % kFoldDepth];
      const int b0 = c * kChunk;
      const int nb = min(kChunk, numat - b0);
      const int tA = (A >= b0 && A < b0 + nb) ? A - b0 : nb;
      auto fold = [&](int t0, int t1) {
        if (heavy) {
          int t = t0;
          for (; t + 8 <= t1; t += 8) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = DMUL(fc[t + u], buf[(t + u) * kStageW + tid]);
#pragma unroll
            for (int u = 0; u < 8; ++u) run = DADD(run, v[u]);
          }
          for (; t < t1; ++t) run = DADD(run, DMUL(fc[t], buf[t * kStageW + tid]));
        } else {
          int t = t0;
          for (; t + 8 <= t1; t += 8) {
            double v[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) v[u] = buf[2 * t + u];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[2 * u] = DMUL(fc[t + u], v[2 * u]);
#pragma unroll
            for (int u = 0; u < 16; ++u) run = DADD(run, v[u]);
          }
          for (; t < t1; ++t) run = DADD(DADD(run, DMUL(fc[t], buf[2 * t])), buf[2 * t + 1]);
        }
      };
      fold(0, tA);
      if (tA < nb) {
        run = DADD(run, f1);
        fold(tA + 1, nb);
      }
    }
    __syncthreads();
  }
  if (tid < lA) a.f[own_idx] = run;
}

int fock_attrs() {
  static std::mutex mu;
  static bool done[64] = {};
  int dev = 0;
  MB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return mb_set_error(MB_ERR_UNSUPPORTED, "Fock build: device index out of range");
  std::lock_guard<std::mutex> lock(mu);
  if (!done[dev]) {
    MB_CUDA(cudaFuncSetAttribute(fock2_pairs, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double) * kWarps * kRows * kTile)));
    MB_CUDA(cudaFuncSetAttribute(fock2_pairs, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared));
    MB_CUDA(cudaFuncSetAttribute(fock2_fold, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double) * kFoldDepth * kChunk * kStageW)));
    done[dev] = true;
  }
  return MB_OK;
}

}  // namespace

extern "C" size_t mb_fock2_ws_bytes(int numat) {
  if (numat <= 0) return 0;
  return 256 + 2 * align256(sizeof(int) * (size_t)numat) + sizeof(double) * kStageW * (size_t)numat * numat;
}

extern "C" int mb_fock2_ws(const MbAtomsDev* atoms, double* f, const double* h, const double* ptot,
                           const double* pa, const double* w, double shift, int use_shift, void* ws,
                           size_t ws_bytes, cudaStream_t stream) {
  if (!atoms || atoms->numat <= 0) return mb_set_error(MB_ERR_ARG, "mb_fock2_ws: no atoms");
  if (!ws || ws_bytes < mb_fock2_ws_bytes(atoms->numat))
    return mb_set_error(MB_ERR_ARG, "mb_fock2_ws: workspace smaller than mb_fock2_ws_bytes(numat)");
  if (((uintptr_t)ws & 255) != 0) return mb_set_error(MB_ERR_ARG, "mb_fock2_ws: workspace not 256-byte aligned");
  MB_TRY(fock_attrs());
  FockArgs a;
  a.at.numat = atoms->numat;
  a.at.first = atoms->first;
  a.at.nor = atoms->nor;
  a.at.lim = atoms->lim;
  a.at.wrow = atoms->wrow;
  a.at.cum = atoms->cum;
  a.f = f;
  a.h = h;
  a.ptot = ptot;
  a.pa = pa;
  a.w = w;
  a.shift = shift;
  a.use_shift = use_shift;
  const FockWs fw = carve(ws, atoms->numat);
  int dev = 0, sms = 0;
  MB_CUDA(cudaGetDevice(&dev));
  MB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  mb_kstat_mark(MB_KSTAT_FOCK, stream, true);
  fock2_lists<<<(atoms->numat + 127) / 128, 128, 0, stream>>>(a.at, ptot, fw);
  MB_LAUNCH_CHECK();
  fock2_pairs<<<sms * 4, 32 * kWarps, sizeof(double) * kWarps * kRows * kTile, stream>>>(a, fw);
  MB_LAUNCH_CHECK();
  fock2_fold<<<atoms->numat, kFoldThreads, sizeof(double) * kFoldDepth * kChunk * kStageW, stream>>>(a, fw);
  MB_LAUNCH_CHECK();
  mb_kstat_mark(MB_KSTAT_FOCK, stream, false);
  return MB_OK;
}

extern "C" int mb_fock2_dev(const MbAtomsDev* atoms, double* f, const double* h, const double* ptot,
                            const double* pa, const double* w, double shift, int use_shift,
                            cudaStream_t stream) {
  if (!atoms || atoms->numat <= 0) return mb_set_error(MB_ERR_ARG, "mb_fock2_dev: no atoms");
  const size_t bytes = mb_fock2_ws_bytes(atoms->numat);
  void* ws = nullptr;
  MB_CUDA(mb_malloc_async(&ws, bytes, stream));
  const int rc = mb_fock2_ws(atoms, f, h, ptot, pa, w, shift, use_shift, ws, bytes, stream);
  const cudaError_t fe = cudaFreeAsync(ws, stream);
  if (rc != MB_OK) return rc;
  if (fe != cudaSuccess) return mb_set_cuda_error(fe, "cudaFreeAsync", __FILE__, __LINE__);
  return MB_OK;
}
