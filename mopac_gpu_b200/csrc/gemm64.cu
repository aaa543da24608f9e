// FP64 GEMM / packed SYRK (column-major, LAPACK argument conventions).
//
// Two tile engines:
//  * DMMA: 128 x 128 or 64 x 64 per CTA on mma.sync m16n8k8 f64, used for every
//    product whose output has more than 64 rows and columns.
//  * FFMA: 64 x 64 per CTA, 4 x 4 outputs per thread, double-buffered through
//    registers; its 8 shared loads per 16 FMAs bind it at half the FP64 rate,
//    so it only serves skinny outputs.
// The split-precision tensor-core path lives in gemm_tc.cu.
#include "mb_common.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16, NT = 256;
constexpr int TM = 4, TN = 4;  // per-thread outputs: rows ty + 16*i, cols tx + 16*j

template <bool TA>
__device__ __forceinline__ double load_a(const double* a, int lda, int m, int k, int r, int kk) {
  if (r >= m || kk >= k) return 0.0;
  return TA ? a[(long long)r * lda + kk] : a[(long long)kk * lda + r];
}
template <bool TB>
__device__ __forceinline__ double load_b(const double* b, int ldb, int n, int k, int kk, int c) {
  if (c >= n || kk >= k) return 0.0;
  return TB ? b[(long long)kk * ldb + c] : b[(long long)c * ldb + kk];
}

// C tile (bm, bn) accumulation, shared by dgemm and packed syrk.
template <bool TA, bool TB>
__device__ __forceinline__ void tile_mma(const double* __restrict__ a, int lda, const double* __restrict__ b,
                                         int ldb, int m, int n, int kbeg, int kend, int bm, int bn,
                                         double acc[TM][TN]) {
  const int k = kend;
  __shared__ double As[2][BK][BM + 1];
  __shared__ double Bs[2][BK][BN + 1];
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0;
  // staging: A tile 64x16 and B tile 16x64, 4 elements per thread each
  double ra[4], rb[4];
  auto gload = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int e = tid + q * NT;
      int r, kk;
      if (TA) { kk = e % BK; r = e / BK; } else { r = e % BM; kk = e / BM; }
      ra[q] = load_a<TA>(a, lda, m, k, bm + r, k0 + kk);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int e = tid + q * NT;
      int c, kk;
      if (TB) { c = e % BN; kk = e / BN; } else { kk = e % BK; c = e / BK; }
      rb[q] = load_b<TB>(b, ldb, n, k, k0 + kk, bn + c);
    }
  };
  auto sstore = [&](int buf) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int e = tid + q * NT;
      int r, kk;
      if (TA) { kk = e % BK; r = e / BK; } else { r = e % BM; kk = e / BM; }
      As[buf][kk][r] = ra[q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int e = tid + q * NT;
      int c, kk;
      if (TB) { c = e % BN; kk = e / BN; } else { kk = e % BK; c = e / BK; }
      Bs[buf][kk][c] = rb[q];
    }
  };
  const int nk = (kend - kbeg + BK - 1) / BK;
  gload(kbeg);
  sstore(0);
  __syncthreads();
  for (int t = 0; t < nk; ++t) {
    const int cur = t & 1;
    if (t + 1 < nk) gload(kbeg + (t + 1) * BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      double av[TM], bv[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) av[i] = As[cur][kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < TN; ++j) bv[j] = Bs[cur][kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fma(av[i], bv[j], acc[i][j]);
    }
    if (t + 1 < nk) sstore(cur ^ 1);
    __syncthreads();
  }
}

template <bool TA, bool TB>
__global__ void __launch_bounds__(NT) dgemm_kernel(int m, int n, int k, double alpha, const double* __restrict__ a,
                                                   int lda, const double* __restrict__ b, int ldb, double beta,
                                                   double* __restrict__ c, int ldc) {
  // split-K: slice z of gridDim.z covers k in [z*kchunk, min(k, (z+1)*kchunk))
  // and, when gridDim.z > 1, writes its raw partial sum to c + z*m*n (ld = m)
  const int bm = blockIdx.y * BM, bn = blockIdx.x * BN;
  const int kchunk = (k + gridDim.z - 1) / gridDim.z;
  const int kb = blockIdx.z * kchunk, ke = min(k, kb + kchunk);
  double acc[TM][TN];
  tile_mma<TA, TB>(a, lda, b, ldb, m, n, kb, ke, bm, bn, acc);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const bool partial = gridDim.z > 1;
  double* cz = partial ? c + (long long)blockIdx.z * m * n : c;
  const int ldz = partial ? m : ldc;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    int r = bm + ty + 16 * i;
    if (r >= m) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      int cc = bn + tx + 16 * j;
      if (cc >= n) continue;
      double* p = cz + (long long)cc * ldz + r;
      if (partial) *p = acc[i][j];
      else *p = (beta == 0.0) ? alpha * acc[i][j] : alpha * acc[i][j] + beta * (*p);
    }
  }
}

// ------------------------------------------------------------------ DMMA
// Tiles of TILE x TILE per CTA, TILE 128 (8 warps of 64 x 32) or 64 (4 warps of
// 32 x 32), k in blocks of DBK through a ring of DSTG shared-memory stages
// filled by cp.async; the next fragments of eight k are read while the 4 x 4 or
// 2 x 4 m16n8k8 products of the current ones run.  An operand is staged as it lies in
// memory, [k][m] or (transposed) [m][k]; both strides are 4 modulo 16 doubles, so
// a fragment's lanes hit distinct banks.
//
// FP64 products run at the rate of the FP64 pipe either way, so the tile is
// chosen by how evenly its tiles divide over the SMs (dmma_tile below).  Every
// output is summed over k in ascending order whatever the tile: both give the
// same bits.  One B200, us (before: 128-tiles of m8n8k4 in two register-staged
// buffers): 3072^3 1863 (2058), 3072 x 1024 x 3072 730 (1035), 1024 x 2048 x 3072
// 518 (546), 2046 x 682 x 2046 259 (354), 682 x 1364 x 2046 174 (369), 1026^3 97
// (187), 600^3 52 (115); packed SYRK of 3072 x 2048 630 (1043), 1026 x 684 64
// (128), 600 x 400 34 (81), 144 x 96 16 (27).
constexpr int DBK = 16, DSTG = 3;

template <int TILE>
struct Dmma {
  static constexpr int THREADS = TILE * 2;                  // 8 or 4 warps
  static constexpr int MI = TILE == 128 ? 8 : 4, NJ = 4;    // fragments of a warp
  static constexpr int WM = 8 * MI, WROWS = TILE / WM;      // rows of a warp, warps along m
  static constexpr int LDM = TILE + 4, LDK = DBK + 4;       // strides of [k][m] and [m][k]
  static constexpr int STAGE = TILE * LDK > DBK * LDM ? TILE * LDK : DBK * LDM;  // doubles, one operand
  static constexpr int SMEM = (int)sizeof(double) * 2 * DSTG * STAGE;
};

// A 16 x 8 block over eight k: bit for bit eight multiply-adds in ascending k.
__device__ __forceinline__ void dmma(double (&c0)[2], double (&c1)[2], const double (&a0)[2], const double (&a1)[2],
                                     const double (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+d"(c0[0]), "+d"(c0[1]), "+d"(c1[0]), "+d"(c1[1])
      : "d"(a0[0]), "d"(a1[0]), "d"(a0[1]), "d"(a1[1]), "d"(b[0]), "d"(b[1]));
}

// Rows r0 .. r0 + TILE - 1, k0 .. k0 + DBK - 1 of an operand X(r, k), zero
// outside R x K.  KC: k is the contiguous index (stage [r][k]), else r is
// ([k][r]).  V: doubles per copy, 2 when pairs are 16-byte aligned.
template <int TILE, bool KC, int V>
__device__ __forceinline__ void dmma_stage(double* t, const double* __restrict__ x, int ld, int r0, int R, int k0,
                                           int K) {
  using D = Dmma<TILE>;
  constexpr int W = KC ? DBK : TILE, H = KC ? TILE : DBK, LD = KC ? D::LDK : D::LDM;
#pragma unroll
  for (int c = threadIdx.x; c < H * W / V; c += D::THREADS) {
    const int row = c / (W / V), w = V * (c % (W / V));
    const int r = r0 + (KC ? row : w), k = k0 + (KC ? w : row);
    const bool row_in = KC ? r < R : k < K;
    const int left = KC ? K - k : R - r;  // of the contiguous index
    const int bytes = !row_in || left <= 0 ? 0 : (left >= V ? 8 * V : 8);
    const double* src = bytes ? x + (KC ? (long long)r * ld + k : (long long)k * ld + r) : x;
    const unsigned d = (unsigned)__cvta_generic_to_shared(t + row * LD + w);
    if (V == 2)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
    else
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
  }
}

// TILE x TILE tile of op(A) op(B) over k in [kbeg, kend).  Warp w covers rows
// (w % WROWS) * WM .. and columns (w / WROWS) * 32 ..; fragment (i, j) of a
// lane holds C(row0 + 8 i + lane / 4, col0 + 8 j + 2 (lane % 4) + {0, 1}).
template <int TILE, bool TA, bool TB, int V>
__device__ __forceinline__ void tile_dmma(const double* __restrict__ a, int lda, const double* __restrict__ b,
                                          int ldb, int m, int n, int kbeg, int kend, int bm, int bn,
                                          double (&acc)[Dmma<TILE>::MI][Dmma<TILE>::NJ][2]) {
  using D = Dmma<TILE>;
  extern __shared__ __align__(16) double dmma_sh[];  // D::SMEM bytes: DSTG stages of A, then of B
  double* As = dmma_sh;
  double* Bs = dmma_sh + DSTG * D::STAGE;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = (warp % D::WROWS) * D::WM, wn = (warp / D::WROWS) * 32;
#pragma unroll
  for (int i = 0; i < D::MI; ++i)
#pragma unroll
    for (int j = 0; j < D::NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int nk = (kend - kbeg + DBK - 1) / DBK;
  auto stage = [&](int t) {
    if (t < nk) {
      dmma_stage<TILE, TA, V>(As + (t % DSTG) * D::STAGE, a, lda, bm, m, kbeg + t * DBK, kend);
      dmma_stage<TILE, !TB, V>(Bs + (t % DSTG) * D::STAGE, b, ldb, bn, n, kbeg + t * DBK, kend);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  const int fr = lane >> 2, fk = lane & 3;
  // this lane's first element of a k4 fragment, and the step to the next row block
  const int a0 = TA ? (wm + fr) * D::LDK + fk : fk * D::LDM + wm + fr, ai = TA ? 8 * D::LDK : 8, ak = TA ? 4 : 4 * D::LDM;
  const int b0 = TB ? fk * D::LDM + wn + fr : (wn + fr) * D::LDK + fk, bj = TB ? 8 : 8 * D::LDK, bk = TB ? 4 * D::LDM : 4;
  for (int t = 0; t < DSTG - 1; ++t) stage(t);
  for (int t = 0; t < nk; ++t) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(DSTG - 2) : "memory");
    __syncthreads();  // stage t has landed; every warp has left stage t - 1
    stage(t + DSTG - 1);
    const double* at = As + (t % DSTG) * D::STAGE + a0;
    const double* bt = Bs + (t % DSTG) * D::STAGE + b0;
    double av[2][D::MI][2], bv[2][D::NJ][2];  // fragments of eight k, as two of four
    auto load = [&](int q) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int i = 0; i < D::MI; ++i) av[q & 1][i][h] = at[(2 * q + h) * ak + i * ai];
#pragma unroll
        for (int j = 0; j < D::NJ; ++j) bv[q & 1][j][h] = bt[(2 * q + h) * bk + j * bj];
      }
    };
    load(0);
#pragma unroll
    for (int q = 0; q < DBK / 8; ++q) {
      if (q + 1 < DBK / 8) load(q + 1);
#pragma unroll
      for (int i = 0; i < D::MI; i += 2)
#pragma unroll
        for (int j = 0; j < D::NJ; ++j)
          dmma(acc[i][j], acc[i + 1][j], av[q & 1][i], av[q & 1][i + 1], bv[q & 1][j]);
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

template <int TILE, bool TA, bool TB, int V>
__global__ void __launch_bounds__(Dmma<TILE>::THREADS)
    dgemm_dmma_kernel(int m, int n, int k, double alpha, const double* __restrict__ a, int lda,
                      const double* __restrict__ b, int ldb, double beta, double* __restrict__ c, int ldc) {
  using D = Dmma<TILE>;
  const int bm = blockIdx.y * TILE, bn = blockIdx.x * TILE;
  const int kchunk = (k + gridDim.z - 1) / gridDim.z;
  const int kb = blockIdx.z * kchunk, ke = min(k, kb + kchunk);
  double acc[D::MI][D::NJ][2];
  tile_dmma<TILE, TA, TB, V>(a, lda, b, ldb, m, n, kb, ke, bm, bn, acc);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r0 = bm + (warp % D::WROWS) * D::WM + (lane >> 2), c0 = bn + (warp / D::WROWS) * 32 + 2 * (lane & 3);
  const bool partial = gridDim.z > 1;
  double* cz = partial ? c + (long long)blockIdx.z * m * n : c;
  const int ldz = partial ? m : ldc;
#pragma unroll
  for (int i = 0; i < D::MI; ++i) {
    const int r = r0 + 8 * i;
    if (r >= m) continue;
#pragma unroll
    for (int j = 0; j < D::NJ; ++j)
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int cc = c0 + 8 * j + t;
        if (cc >= n) continue;
        double* p = cz + (long long)cc * ldz + r;
        if (partial) *p = acc[i][j][t];
        else *p = (beta == 0.0) ? alpha * acc[i][j][t] : alpha * acc[i][j][t] + beta * (*p);
      }
  }
}

// Packed lower P = occ * A A^T (+ P when acc) on the DMMA engine (tiles meeting the lower triangle).
template <int TILE, int V>
__global__ void __launch_bounds__(Dmma<TILE>::THREADS)
    syrk_packed_dmma_kernel(int n, int k, double occ, const double* __restrict__ a, int lda, double* __restrict__ p,
                            int acc_p) {
  using D = Dmma<TILE>;
  // block b of the lower triangle of tiles, row by row
  const long long b = blockIdx.x;
  int tr = (int)((sqrt(8.0 * (double)b + 1.0) - 1.0) * 0.5);
  while ((long long)tr * (tr + 1) / 2 > b) --tr;
  while ((long long)(tr + 1) * (tr + 2) / 2 <= b) ++tr;
  const int bm = tr * TILE, bn = (int)(b - (long long)tr * (tr + 1) / 2) * TILE;
  double acc[D::MI][D::NJ][2];
  tile_dmma<TILE, false, true, V>(a, lda, a, lda, n, n, 0, k, bm, bn, acc);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r0 = bm + (warp % D::WROWS) * D::WM + (lane >> 2), c0 = bn + (warp / D::WROWS) * 32 + 2 * (lane & 3);
#pragma unroll
  for (int i = 0; i < D::MI; ++i) {
    const int r = r0 + 8 * i;
    if (r >= n) continue;
#pragma unroll
    for (int j = 0; j < D::NJ; ++j)
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int cc = c0 + 8 * j + t;
        if (cc > r) continue;
        const long long q = mb_tri(r, cc);
        p[q] = acc_p ? occ * acc[i][j][t] + p[q] : occ * acc[i][j][t];
      }
  }
}

// 128 or 64, by the time of the fullest SM in tenths of a 64-tile's time at the
// full rate.  Three 64-tile CTAs share an SM and cover each other's barriers;
// one or two alone run at half and at 0.8 of the rate.  A 128-tile runs alone on
// its SM at 0.9.  (3072^3: 31.1 TFLOP/s with 64, 28.2 with 128; 1024 x 2048 x 3072,
// four 64-tiles or one 128-tile an SM: 21.5 and 24.9; 682 x 1364 x 2046, two or
// one: 21.9 and 10.3.)
int dmma_tile(long long tiles128, long long tiles64) {
  const long long c = (tiles64 + 147) / 148, r = c % 3;
  const long long t64 = 30 * (c / 3) + (r == 0 ? 0 : r == 1 ? 20 : 24), t128 = 44 * ((tiles128 + 147) / 148);
  return t64 <= t128 ? 64 : 128;
}

// The tile of an m x n product in nz slices of k, and of a packed SYRK of order n.
int gemm_tile(int m, int n, int nz) {
  auto tiles = [&](int t) { return (long long)nz * ((m + t - 1) / t) * ((n + t - 1) / t); };
  return dmma_tile(tiles(128), tiles(64));
}
int syrk_tile(int n) {
  auto tiles = [&](int t) {
    const long long q = (n + t - 1) / t;
    return q * (q + 1) / 2;
  };
  return dmma_tile(tiles(128), tiles(64));
}

bool dmma_pairs(const double* x, int ld) { return ((uintptr_t)x & 15) == 0 && ld % 2 == 0; }

template <int TILE, bool TA, bool TB, int V>
int dmma_launch(int m, int n, int k, int nz, double alpha, const double* a, int lda, const double* b, int ldb,
                double beta, double* out, int ldc, cudaStream_t stream) {
  MB_TRY(mb_smem_optin((const void*)dgemm_dmma_kernel<TILE, TA, TB, V>, Dmma<TILE>::SMEM));
  const dim3 grid((n + TILE - 1) / TILE, (m + TILE - 1) / TILE, nz);
  dgemm_dmma_kernel<TILE, TA, TB, V><<<grid, Dmma<TILE>::THREADS, Dmma<TILE>::SMEM, stream>>>(m, n, k, alpha, a, lda, b,
                                                                                              ldb, beta, out, ldc);
  MB_LAUNCH_CHECK();
  return MB_OK;
}

template <bool TA, bool TB>
int dmma_gemm(int m, int n, int k, int nz, double alpha, const double* a, int lda, const double* b, int ldb,
              double beta, double* out, int ldc, cudaStream_t stream) {
  const bool small = gemm_tile(m, n, nz) == 64;
  // a slice starts at an even k, or its pairs along k are off their boundary
  const bool even = nz == 1 || (k + nz - 1) / nz % 2 == 0;
  const bool pairs = even && dmma_pairs(a, lda) && dmma_pairs(b, ldb);
  if (small) {
    if (pairs) return dmma_launch<64, TA, TB, 2>(m, n, k, nz, alpha, a, lda, b, ldb, beta, out, ldc, stream);
    return dmma_launch<64, TA, TB, 1>(m, n, k, nz, alpha, a, lda, b, ldb, beta, out, ldc, stream);
  }
  if (pairs) return dmma_launch<128, TA, TB, 2>(m, n, k, nz, alpha, a, lda, b, ldb, beta, out, ldc, stream);
  return dmma_launch<128, TA, TB, 1>(m, n, k, nz, alpha, a, lda, b, ldb, beta, out, ldc, stream);
}

template <int TILE, int V>
int syrk_launch(int n, int k, double alpha, const double* a, int lda, double* p, int acc, cudaStream_t stream) {
  MB_TRY(mb_smem_optin((const void*)syrk_packed_dmma_kernel<TILE, V>, Dmma<TILE>::SMEM));
  const long long t = (n + TILE - 1) / TILE;
  syrk_packed_dmma_kernel<TILE, V>
      <<<(unsigned)(t * (t + 1) / 2), Dmma<TILE>::THREADS, Dmma<TILE>::SMEM, stream>>>(n, k, alpha, a, lda, p, acc);
  MB_LAUNCH_CHECK();
  return MB_OK;
}

int dmma_syrk(int n, int k, double alpha, const double* a, int lda, double* p, int acc, cudaStream_t stream) {
  const bool small = syrk_tile(n) == 64, pairs = dmma_pairs(a, lda);
  if (small) return pairs ? syrk_launch<64, 2>(n, k, alpha, a, lda, p, acc, stream)
                          : syrk_launch<64, 1>(n, k, alpha, a, lda, p, acc, stream);
  return pairs ? syrk_launch<128, 2>(n, k, alpha, a, lda, p, acc, stream)
               : syrk_launch<128, 1>(n, k, alpha, a, lda, p, acc, stream);
}

// C = alpha * sum_z part[z] + beta * C, slices summed in order (deterministic).
__global__ void splitk_reduce(int m, int n, int nz, double alpha, const double* __restrict__ part, double beta,
                              double* __restrict__ c, int ldc) {
  const long long mn = (long long)m * n;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < mn; q += (long long)gridDim.x * blockDim.x) {
    double s = part[q];
    for (int z = 1; z < nz; ++z) s += part[z * mn + q];
    const int r = (int)(q % m), cc = (int)(q / m);
    double* p = c + (long long)cc * ldc + r;
    *p = (beta == 0.0) ? alpha * s : alpha * s + beta * (*p);
  }
}

// P(packed lower) = occ * A A^T (+ P when acc) with A = c[:, 0:k] (n x k,
// column-major).  Grid over 64x64 tiles intersecting the lower triangle.
__global__ void __launch_bounds__(NT) syrk_packed_kernel(int n, int k, double occ, const double* __restrict__ a,
                                                         int lda, double* __restrict__ p, int ntn, int acc_p) {
  const int bm = blockIdx.y * BM, bn = blockIdx.x * BN;
  if (bn > bm + BM - 1) return;  // tile entirely above the diagonal
  double acc[TM][TN];
  tile_mma<false, true>(a, lda, a, lda, n, n, 0, k, bm, bn, acc);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    int r = bm + ty + 16 * i;
    if (r >= n) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      int cc = bn + tx + 16 * j;
      if (cc > r) continue;
      const long long q = mb_tri(r, cc);
      p[q] = acc_p ? occ * acc[i][j] + p[q] : occ * acc[i][j];
    }
  }
}

// P_ii = cst + P_ii (the constant of the positron-equivalent density).
__global__ void add_diag_kernel(int n, double cst, double* __restrict__ p) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[mb_tri(i, i)] = cst + p[mb_tri(i, i)];
}

// DMMA engine for all but skinny outputs.
bool gemm_wide(int m, int n) { return m > BM && n > BN; }

// Slices of k, counted in 128- or 64-wide tiles, whatever tile then runs: the sums'
// order stays the same.
int gemm_slices(int m, int n, int k, size_t ws_elems) {
  const bool wide = gemm_wide(m, n);
  const int t = wide ? 128 : BM;
  const int tiles = ((n + t - 1) / t) * ((m + t - 1) / t);
  const int target = wide ? 148 : 296;
  int nz = 1;
  if (k >= 512 && tiles < target) {
    nz = (target + tiles - 1) / tiles;
    if (nz > k / 128) nz = k / 128;
    if (nz > 32) nz = 32;
    while (nz > 1 && (size_t)nz * m * n > ws_elems) --nz;
  }
  return nz;
}

}  // namespace

// Which tile a product takes, given the elements of its workspace (0: none), and a
// packed SYRK: 64 or 128, 0 for the FFMA engine.
extern "C" int mb_dgemm_tile(int m, int n, int k, size_t ws_elems) {
  return gemm_wide(m, n) ? gemm_tile(m, n, gemm_slices(m, n, k, ws_elems)) : 0;
}
extern "C" int mb_syrk_tile(int n) { return n > BM ? syrk_tile(n) : 0; }

// GEMM with optional split-K: when the output has too few 64x64 tiles to fill
// the GPU and k is long, the k loop is cut into slices whose partial sums go to
// ws (nsplit * m * n doubles) and are reduced in a fixed order.
extern "C" int mb_dgemm_ws(char transa, char transb, int m, int n, int k, double alpha, const double* a, int lda,
                           const double* b, int ldb, double beta, double* c, int ldc, double* ws, size_t ws_elems,
                           cudaStream_t stream) {
  if (m < 0 || n < 0 || k < 0) return mb_set_error(MB_ERR_ARG, "mb_dgemm: negative size");
  if (m == 0 || n == 0) return MB_OK;
  bool ta = (transa == 'T' || transa == 't' || transa == 'C' || transa == 'c');
  bool tb = (transb == 'T' || transb == 't' || transb == 'C' || transb == 'c');
  const bool wide = gemm_wide(m, n);
  const int nz = ws ? gemm_slices(m, n, k, ws_elems) : 1;
  double* out = nz > 1 ? ws : c;
  if (wide) {
    if (!ta && !tb) MB_TRY((dmma_gemm<false, false>(m, n, k, nz, alpha, a, lda, b, ldb, beta, out, ldc, stream)));
    else if (!ta && tb) MB_TRY((dmma_gemm<false, true>(m, n, k, nz, alpha, a, lda, b, ldb, beta, out, ldc, stream)));
    else if (ta && !tb) MB_TRY((dmma_gemm<true, false>(m, n, k, nz, alpha, a, lda, b, ldb, beta, out, ldc, stream)));
    else MB_TRY((dmma_gemm<true, true>(m, n, k, nz, alpha, a, lda, b, ldb, beta, out, ldc, stream)));
  } else {
    const dim3 grid((n + BN - 1) / BN, (m + BM - 1) / BM, nz);
    if (!ta && !tb) dgemm_kernel<false, false><<<grid, NT, 0, stream>>>(m, n, k, alpha, a, lda, b, ldb, beta, out, ldc);
    else if (!ta && tb) dgemm_kernel<false, true><<<grid, NT, 0, stream>>>(m, n, k, alpha, a, lda, b, ldb, beta, out, ldc);
    else if (ta && !tb) dgemm_kernel<true, false><<<grid, NT, 0, stream>>>(m, n, k, alpha, a, lda, b, ldb, beta, out, ldc);
    else dgemm_kernel<true, true><<<grid, NT, 0, stream>>>(m, n, k, alpha, a, lda, b, ldb, beta, out, ldc);
    MB_LAUNCH_CHECK();
  }
  if (nz > 1) {
    long long mn = (long long)m * n;
    int blocks = (int)((mn + 255) / 256);
    if (blocks > 148 * 8) blocks = 148 * 8;
    splitk_reduce<<<blocks, 256, 0, stream>>>(m, n, nz, alpha, ws, beta, c, ldc);
    MB_LAUNCH_CHECK();
  }
  return MB_OK;
}

extern "C" int mb_dgemm_dev(char transa, char transb, int m, int n, int k, double alpha, const double* a,
                            int lda, const double* b, int ldb, double beta, double* c, int ldc,
                            cudaStream_t stream) {
  return mb_dgemm_ws(transa, transb, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, nullptr, 0, stream);
}

namespace {

// P = alpha * C[:, k0:k1] C[:, k0:k1]^T (+ P when acc), packed lower.  An
// empty column range gives alpha * 0 (+ P), as a GEMM with k = 0 does.
int syrk_range(int n, int k0, int k1, double alpha, const double* c, int ldc, double* p, bool acc,
               cudaStream_t stream) {
  const int k = k1 > k0 ? k1 - k0 : 0;
  const double* a = c + (long long)(k > 0 ? k0 : 0) * ldc;
  if (n > BM) return dmma_syrk(n, k, alpha, a, ldc, p, acc ? 1 : 0, stream);
  dim3 grid((n + BN - 1) / BN, (n + BM - 1) / BM);
  syrk_packed_kernel<<<grid, NT, 0, stream>>>(n, k, alpha, a, ldc, p, grid.x, acc ? 1 : 0);
  MB_LAUNCH_CHECK();
  return MB_OK;
}

}  // namespace

extern "C" int mb_density_dev(int n, int nocc, double occ, const double* c, int ldc, double* p,
                              cudaStream_t stream) {
  if (n <= 0 || nocc < 0 || nocc > n) return mb_set_error(MB_ERR_ARG, "mb_density_dev: bad size");
  if (nocc == 0) {
    MB_CUDA(cudaMemsetAsync(p, 0, sizeof(double) * (size_t)n * (n + 1) / 2, stream));
    return MB_OK;
  }
  mb_kstat_mark(MB_KSTAT_DENSITY, stream, true);
  const int rc = syrk_range(n, 0, nocc, occ, c, ldc, p, false, stream);
  mb_kstat_mark(MB_KSTAT_DENSITY, stream, false);
  return rc;
}

// density_for_GPU (matrix/density_for_GPU.F90:16-130) and densit
// (matrix/densit.F90): closed-shell, fractional and UHF occupations.
// iopc 2, 3: the DGEMM form; 4: occ * C_d C_d^T; 5: that below fract 0.01,
// else the explicit sums; 6 (no reference iopc): densit, the explicit sums
// at any fract.
extern "C" int mb_density_occ_dev(int n, int ndubl, int nsingl, double occ, double fract, int mode, int iopc,
                                  const double* c, int ldc, double* p, cudaStream_t stream) {
  if (n <= 0 || ldc < n || ndubl < 0 || ndubl > n || nsingl < 0 || nsingl > n || !c || !p)
    return mb_set_error(MB_ERR_ARG, "mb_density_occ_dev: bad size");
  if (iopc < 2 || iopc > 6) return mb_set_error(MB_ERR_ARG, "mb_density_occ_dev: iopc must be 2..6");
  // iopc 4 (and 5 below fract 0.01): the closed-shell product occ * C_d C_d^T
  if (iopc == 4 || (iopc == 5 && fract < 1.0e-2)) return mb_density_dev(n, ndubl, occ, c, ldc, p, stream);
  // electron or positron equivalent (density_for_GPU.F90:32-54, densit.F90:19-36)
  double sign = 1.0, frac = fract, cst = 0.0;
  int nl2 = 1, nu2 = ndubl, nl1 = ndubl + 1, nu1 = nsingl;
  if (ndubl != 0 && nsingl > n / 2 && mode != 2) {
    sign = -1.0;
    frac = occ - fract;
    cst = occ;
    nl2 = nsingl + 1;
    nu2 = n;
    nl1 = ndubl + 1;
    nu1 = nsingl;
  }
  // iopc 2/3 (the DGEMM form): 2*sign*G2, then + frac*sign*G1; iopc 5/6 (the
  // explicit sums, densit): sign*(occ*G2 + frac*G1).  G = C C^T over the
  // 1-based column ranges [nl, nu]; then P_ii = cst + P_ii.
  const double a2 = (iopc <= 3 ? 2.0 : occ) * sign, a1 = frac * sign;
  mb_kstat_mark(MB_KSTAT_DENSITY, stream, true);
  int rc = syrk_range(n, nl2 - 1, nu2, a2, c, ldc, p, false, stream);
  if (rc == MB_OK) rc = syrk_range(n, nl1 - 1, nu1, a1, c, ldc, p, true, stream);
  mb_kstat_mark(MB_KSTAT_DENSITY, stream, false);
  if (rc != MB_OK) return rc;
  if (cst != 0.0) {
    add_diag_kernel<<<(n + 255) / 256, 256, 0, stream>>>(n, cst, p);
    MB_LAUNCH_CHECK();
  }
  return MB_OK;
}
