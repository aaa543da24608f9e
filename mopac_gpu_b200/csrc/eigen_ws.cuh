// Workspace of one eigensolve, shared by eigen.cu and eigen_panel.cu.
#pragma once
#include "mb_common.cuh"

namespace eigh {

constexpr int NB = 32;    // panel width
constexpr int TCH = 16;   // row chunks per dot product of the panels
constexpr int BT = 64;    // reflectors per back-transformation block

struct Ws {
  double *A, *V, *Z, *X, *U0, *U1, *U2;  // n x n each
  double* vwv;                           // [V | W | V] panel columns
  double *d, *e, *e2, *tau, *wvec;       // n each
  double *tvec, *tpart, *part;
  double *S, *Tm;                        // every back-transformation block's V^T V and T factor
  double* Y;                             // BT x n
  double* bnd;
};

inline size_t ws_doubles(int n) {
  const size_t nn = (size_t)n * n;
  return 7 * nn + 3 * (size_t)n * NB + 5 * (size_t)n + 2 * NB + 2 * NB * TCH + 4096 +
         (size_t)BT * BT * 2 * (size_t)((n + BT - 1) / BT) + (size_t)BT * n;
}

inline Ws carve(int n, void* ws) {
  const size_t nn = (size_t)n * n, tb = (size_t)BT * BT * (size_t)((n + BT - 1) / BT);
  double* b = (double*)ws;
  auto take = [&](size_t count) {
    double* p = b;
    b += count;
    return p;
  };
  Ws w;
  w.A = take(nn);
  w.V = take(nn);
  w.Z = take(nn);
  w.X = take(nn);
  w.U0 = take(nn);
  w.U1 = take(nn);
  w.U2 = take(nn);
  w.vwv = take((size_t)n * 3 * NB);
  w.d = take(n);
  w.e = take(n);
  w.e2 = take(n);
  w.tau = take(n);
  w.wvec = take(n);
  w.tvec = take(2 * NB);
  w.tpart = take(2 * NB * TCH);
  w.part = take(4096);
  w.S = take(tb);
  w.Tm = take(tb);
  w.Y = take((size_t)BT * n);
  w.bnd = w.part + 2048;
  return w;
}

}  // namespace eigh

// eigen.cu: the caller's return code for a solve's status word, with its message.
// The word holds the first failure: MB_ERR_TIMEOUT (a bounded wait gave up) or
// MB_ERR_NUMERIC.
extern "C" int mb_eigh_status(int status);
// eigen_panel.cu
extern "C" int mb_eigh_panels(int n, int cols, const eigh::Ws* w, cudaStream_t stream, int* done);
extern "C" int mb_eigh_back(int n, const eigh::Ws* w, double* c, cudaStream_t stream);
// tridiag.cu
extern "C" int mb_tridiag_cluster_orders(int clusters16);
extern "C" int mb_tridiag_cluster_max(void);
extern "C" int mb_tridiag_cluster(int n, double* pk, int perturb, double* vall, double* d, double* e, double* tau,
                                  int* status, cudaStream_t stream);
extern "C" int mb_tridiag_grid_max(int ctas);
extern "C" int mb_tridiag_grid(int m, int ctas, const double* a, long long lda, double* vall, double* d, double* e,
                               double* tau, void* scratch, int* status, cudaStream_t stream);
extern "C" int mb_unpack_dev(int n, const double* pk, double* a, int lda, int perturb, double* pk_mut,
                             cudaStream_t stream);
