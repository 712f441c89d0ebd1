// Pressure-correction / momentum Krylov solve on the device: BiCGStab
// (van der Vorst 1992) right-preconditioned by point or 3x3 block Jacobi, or
// for scalar systems by the aggregation-AMG V-cycle of oa_amg.cu; for scalar
// AMG-preconditioned systems also GCR(2), one V-cycle per iteration.
//
// The reference hands its systems to liblinsolve (PETSc / Trilinos / HYPRE,
// src/equation/linearSystem.h:416-462), which is absent from the reference
// checkout; the algorithm here is the published one. All scalars live on the
// device and every reduction is a fixed two-stage tree (block partials, which
// every block of the kernel that needs the sum adds in one order; segments of a
// batch close in the last block, in chunk order), so results are bitwise
// reproducible run to run. A device "done" flag lets chunks of iterations be launched without
// host round trips; kernels after convergence return immediately.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>

#include <algorithm>
#include <climits>
#include <cmath>
#include <vector>
#include <type_traits>

#include "oa_internal.h"
#include "oa_krylov.h"
#include "oa_ell.cuh"

namespace oa {

constexpr int KB = 256;        // threads per block for vector kernels
// Blocks of the kernels that reduce; they loop over the rows, so that the
// kernel which uses a sum can add the partials itself, in every block. The
// number and the order of the tree below fix the sums' last bits, which
// BiCGStab in FP32 carries on: with 8 blocks per SM (1184) and the warps added
// first, twenty momentum iterations ended 1e-7 away in U, and p, whose level
// hangs on one node, 7e-5.
constexpr int MAX_PARTIALS = 2048;
// of a solver: two sets of two values
constexpr int KRYLOV_PARTIALS = 4 * MAX_PARTIALS;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Fixed-order two-stage reductions: a partial per block, and every block of
// the kernel that needs the sum adds the partials in the same order. On a
// 16^3 cavity (20 partials) this costs 0.1 to 0.2 us per kernel; a ticket with the
// last block adding up cost 1.6 us, a kernel of one block for the sum 3 to 4. With
// all 2,048 partials it costs what it replaces: on 129^3 rows in FP32 k_gcr_orth,
// k_gcr_update and k_end_iter take 18.9, 23.9 and 4.4 us, with kernels of one
// block between them they took 18.1, 16.5 and 3 x 4.3.
template <int NV>
__device__ __forceinline__ void block_partials(double (&v)[NV], double* partials) {
  __shared__ double sh[NV][KB / 32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const double s = warp_sum(v[k]);
    if (l == 0) sh[k][w] = s;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < KB / 32; ++i) s += sh[threadIdx.x][i];
    partials[threadIdx.x * MAX_PARTIALS + blockIdx.x] = s;
  }
}

// Sum of nb partials per value in a fixed tree, in every thread: the eight warps
// first, by halves, then the lanes
template <int NV>
__device__ __forceinline__ void sum_partials(const double* __restrict__ partials, int nb, double (&out)[NV]) {
  __shared__ double sh[NV][KB];
  const int l = threadIdx.x & 31;
  double t[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) t[k] = 0.0;
  for (int i = threadIdx.x; i < nb; i += KB)
#pragma unroll
    for (int k = 0; k < NV; ++k) t[k] += __ldg(partials + k * MAX_PARTIALS + i);
#pragma unroll
  for (int k = 0; k < NV; ++k) sh[k][threadIdx.x] = t[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double s[KB / 32];
#pragma unroll
    for (int i = 0; i < KB / 32; ++i) s[i] = sh[k][32 * i + l];
#pragma unroll
    for (int h = KB / 64; h > 0; h >>= 1)
#pragma unroll
      for (int i = 0; i < h; ++i) s[i] += s[i + h];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
    out[k] = s[0];
  }
}

// The done flag for a kernel whose first block may set it (a breakdown) while
// other blocks of the same grid start: one answer for the whole block. With a
// test by each thread a block could lose some warps to the flag, and the others
// would add the sums those never wrote and go on with a wrong coefficient. A
// block that still sees the flag clear finds the same breakdown in the sums.
__device__ __forceinline__ bool block_done(const KScal* sc) { return __syncthreads_or(sc->done); }

static int reduce_grid(long long n) { return (int)std::min<long long>((n + KB - 1) / KB, MAX_PARTIALS); }

// Product of row component m of block row [a, e) with x: U entries at a time
// with every load in flight before the first use, summed in entry order.
template <int B, class TM, class TV>
__device__ __forceinline__ double row_product(const int* __restrict__ cols, const TM* __restrict__ A,
                                              const TV* __restrict__ x, int a, int e, int m) {
  constexpr int U = B == 1 ? 4 : (sizeof(TM) == 8 ? 2 : 4);
  double s = 0.0;
  for (int k = a; k < e; k += U) {
    int j[U];
    TM v[U][B];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int q = min(k + u, e - 1);
      j[u] = __ldg(cols + q);
#pragma unroll
      for (int c = 0; c < B; ++c) v[u][c] = __ldg(A + (size_t)q * B * B + B * m + c);
    }
    TV xv[U][B];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int c = 0; c < B; ++c) xv[u][c] = __ldg(x + (size_t)B * j[u] + c);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k + u < e)
#pragma unroll
        for (int c = 0; c < B; ++c) s += double(v[u][c]) * double(xv[u][c]);
  }
  return s;
}

template <int B, class TM, class TP>
__global__ void k_build_minv(int nn, const int* __restrict__ rp, const int* __restrict__ dg, const TM* __restrict__ A,
                             TP* Minv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nn) return;
  const TM* d = A + (size_t)(rp[i] + dg[i]) * B * B;
  if (B == 1) {
    Minv[i] = TP(1.0 / double(d[0]));
  } else {
    double a[9];
    for (int k = 0; k < 9; ++k) a[k] = double(d[k]);
    const double det = a[0] * (a[4] * a[8] - a[5] * a[7]) - a[1] * (a[3] * a[8] - a[5] * a[6]) +
                       a[2] * (a[3] * a[7] - a[4] * a[6]);
    const double id = 1.0 / det;
    TP* r = Minv + 9 * (size_t)i;
    r[0] = TP((a[4] * a[8] - a[5] * a[7]) * id);
    r[1] = TP((a[2] * a[7] - a[1] * a[8]) * id);
    r[2] = TP((a[1] * a[5] - a[2] * a[4]) * id);
    r[3] = TP((a[5] * a[6] - a[3] * a[8]) * id);
    r[4] = TP((a[0] * a[8] - a[2] * a[6]) * id);
    r[5] = TP((a[2] * a[3] - a[0] * a[5]) * id);
    r[6] = TP((a[3] * a[7] - a[4] * a[6]) * id);
    r[7] = TP((a[1] * a[6] - a[0] * a[7]) * id);
    r[8] = TP((a[0] * a[4] - a[1] * a[3]) * id);
  }
}

// x = 0, r = b, and for BiCGStab rh = b (the directions start with the first
// iteration, which reads none); partial ||b||^2
template <class TV, class TB>
__global__ void __launch_bounds__(KB) k_init(int n, const TB* __restrict__ b, TV* x, TV* r, TV* rh, double* partials) {
  double s[1] = {0.0};
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const TV bv = TV(b[t]);
    x[t] = TV(0);
    r[t] = bv;
    if (rh) rh[t] = bv;
    s[0] += double(bv) * double(bv);
  }
  block_partials<1>(s, partials);
}

// rtol_dev / maxit_dev (when not null) replace rtol / maxit: the inner solves
// of a graph-captured iterative refinement take them from the refinement state
__global__ void __launch_bounds__(KB) k_init_scalars(KScal* sc, const double* partials, int nb, double rtol,
                                                      int maxit, const double* rtol_dev, const int* maxit_dev) {
  double o[1];
  sum_partials<1>(partials, nb, o);
  if (threadIdx.x == 0) {
    sc->rtol = rtol_dev ? *rtol_dev : rtol;
    sc->maxit = maxit_dev ? *maxit_dev : maxit;
    sc->bnorm = sqrt(o[0]);
    sc->rnorm = sc->bnorm;
    sc->rho = sc->alpha = sc->omega = 1.0;
    sc->d0 = o[0];  // rh.r for the first iteration equals ||b||^2
    sc->iters = 0;
    sc->status = 0;
    sc->seg_rel = 0.0;
    sc->done = (sc->bnorm == 0.0 || !(sc->bnorm < INFINITY)) ? 1 : 0;
    if (!(sc->bnorm < INFINITY)) sc->status = 2;
  }
}

// z = Minv v of row i (point or 3x3 block Jacobi); the inverse is stored in
// the precision of the Krylov vectors (FP32 in the mixed form's inner solves)
template <int B, class TV>
__device__ __forceinline__ void jacobi_row(const TV* __restrict__ Minv, int i, const TV (&v)[B], TV* z) {
  if (B == 1) {
    z[i] = TV(double(__ldg(Minv + i)) * double(v[0]));
  } else {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const TV* M = Minv + 9 * (size_t)i + 3 * m;
      z[3 * (size_t)i + m] = TV(double(__ldg(M)) * double(v[0]) + double(__ldg(M + 1)) * double(v[1 % B]) +
                                double(__ldg(M + 2)) * double(v[2 % B]));
    }
  }
}

// p = r + beta (p - omega v), beta = (rho1/rho)(alpha/omega), rho1 = sc->d0
// (p = r in the first iteration), and with Jacobi ph = Minv p; one thread per
// row
template <int B, class TV>
__global__ void __launch_bounds__(KB) k_p_update(int nn, TV* p, const TV* __restrict__ r, const TV* __restrict__ v,
                                                  const TV* __restrict__ Minv, TV* ph, const KScal* sc) {
  if (sc->done) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nn) return;
  const bool first = sc->iters == 0;
  const double omega = sc->omega, beta = (sc->d0 / sc->rho) * (sc->alpha / omega);
  TV q[B];
#pragma unroll
  for (int c = 0; c < B; ++c) {
    const size_t t = (size_t)B * i + c;
    q[c] = first ? r[t] : TV(double(r[t]) + beta * (double(p[t]) - omega * double(v[t])));
    p[t] = q[c];
  }
  if (Minv) jacobi_row<B, TV>(Minv, i, q, ph);
}

// alpha = rho1 / (rh.v) from the product's partials (a zero or non-finite rh.v
// is a breakdown), s = r - alpha v (stored in r), and with Jacobi sh = Minv s
template <int B, class TV>
__global__ void __launch_bounds__(KB) k_s_update(int nn, TV* r, const TV* __restrict__ v,
                                                  const TV* __restrict__ Minv, TV* sh,
                                                  const double* __restrict__ partials, int nb, KScal* sc) {
  if (block_done(sc)) return;
  double o[1];
  sum_partials<1>(partials, nb, o);
  const bool broken = o[0] == 0.0 || !(fabs(o[0]) < INFINITY);
  const double alpha = broken ? 0.0 : sc->d0 / o[0];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (broken) {
      sc->done = 1;
      sc->status = 1;
    } else {
      sc->alpha = alpha;
    }
  }
  if (broken) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
    TV q[B];
#pragma unroll
    for (int c = 0; c < B; ++c) {
      const size_t t = (size_t)B * i + c;
      q[c] = TV(double(r[t]) - alpha * double(v[t]));
      r[t] = q[c];
    }
    if (Minv) jacobi_row<B, TV>(Minv, i, q, sh);
  }
}

// Row i of a scalar matrix times x
template <class TM>
struct ScalarMat {
  const int *rp, *cols;  // CSR
  const TM* A;
  EllMat<TM> ell;        // fixed-width storage
};
template <int FORMAT, class TM, class TX>
__device__ __forceinline__ double scalar_row(const ScalarMat<TM>& m, int i, const TX* __restrict__ x) {
  if constexpr (FORMAT >= ELL)
    return ell_row<FORMAT, TM>(m.ell, i, [&](int j) { return double(__ldg(x + j)); });
  else
    return row_product<1, TM, TX>(m.cols, m.A, x, __ldg(m.rp + i), __ldg(m.rp + i + 1), 0);
}

// a kernel template over the formats of a scalar matrix
#define OA_FORMAT(format, call)        \
  switch (format) {                    \
    case ELL + 7: call(ELL + 7); break;                \
    case ELL + 15: call(ELL + 15); break;              \
    case ELL_STREAM + 7: call(ELL_STREAM + 7); break;  \
    case ELL_STREAM + 15: call(ELL_STREAM + 15); break;\
    default: call(1);                  \
  }

// y = A x for a BSR matrix with BxB row-major blocks. The scalar row products run
// 8 blocks per SM (32 registers): a pass of the mixed 128^3 cavity takes 39.1 ms,
// with 6 blocks 39.7. In FP64 width 7 spills 68 to 80 B per thread at 8, and 6 is
// the faster one (16^3 3.78 against 3.69 ms, 96^3 22.7 against 21.8).
// STEP 1: partial w.y with w = rh; STEP 2: partials y.w and y.y with w = s.
template <int B, class TM, class TV, int STEP, int FORMAT>
__global__ void __launch_bounds__(KB, B == 1 ? 8 : 1) k_spmv(int nn, ScalarMat<TM> M, const TV* __restrict__ x, TV* __restrict__ y,
                                              const TV* __restrict__ w, double* partials, const KScal* sc) {
  if (sc->done) return;
  double v[STEP];
#pragma unroll
  for (int k = 0; k < STEP; ++k) v[k] = 0.0;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nn * B; t += gridDim.x * blockDim.x) {
    const double wt = double(w[t]);
    double s;
    if (B == 1) {
      s = scalar_row<FORMAT, TM, TV>(M, t, x);
    } else {
      const int i = t / B, m = t - i * B;
      s = row_product<B, TM, TV>(M.cols, M.A, x, __ldg(M.rp + i), __ldg(M.rp + i + 1), m);
    }
    const TV ys = TV(s);
    y[t] = ys;
    v[0] += double(ys) * wt;
    if (STEP > 1) v[STEP - 1] += double(ys) * double(ys);
  }
  block_partials<STEP>(v, partials);
}

// End of a BiCGStab iteration: rho <- rho1; rho1 <- rh.r; convergence test
// (per segment for batched systems)
__device__ __forceinline__ void bicgstab_end(KScal* sc, double rr, double rhr, double segmax, int nseg) {
  sc->seg_rel = segmax;
  sc->rho = sc->d0;
  sc->d0 = rhr;
  sc->rnorm = sqrt(rr);
  sc->iters += 1;
  if (!(sc->rnorm < INFINITY)) {
    sc->done = 1;
    sc->status = 2;
  } else if (sc->rnorm > 1e3 * sc->bnorm) {
    sc->done = 1;  // diverging (seen with FP32 vectors on stiff systems)
    sc->status = 3;
  } else if ((nseg > 1 ? segmax <= sc->rtol : sc->rnorm <= sc->rtol * sc->bnorm) || sc->iters >= sc->maxit) {
    sc->done = 1;
  } else if (sc->omega == 0.0 || sc->d0 == 0.0) {
    sc->done = 1;
    sc->status = 1;
  }
}

// End of a GCR iteration: residual norm and convergence test; an iteration that
// leaves the residual where it was (truncated GCR can stagnate when the
// preconditioned operator's symmetric part is not definite) ends the solve
// with status 1, and the caller falls back to BiCGStab
__device__ __forceinline__ void gcr_end(KScal* sc, double rr, double segmax, int nseg) {
  sc->seg_rel = segmax;
  const double prev = sc->rnorm;
  sc->rnorm = sqrt(rr);
  sc->iters += 1;
  if (!(sc->rnorm < INFINITY)) {
    sc->done = 1;
    sc->status = 2;
  } else if ((nseg > 1 ? segmax <= sc->rtol : sc->rnorm <= sc->rtol * sc->bnorm) || sc->iters >= sc->maxit) {
    sc->done = 1;
  } else if (sc->rnorm > 0.9999 * prev) {
    sc->done = 1;
    sc->status = 1;
  }
}

// the partials of an iteration's last kernel close it
template <bool GCR>
__global__ void __launch_bounds__(KB) k_end_iter(KScal* sc, const double* partials, int nb) {
  if (sc->done) return;
  double o[2];
  if (GCR) {
    double p[1];
    sum_partials<1>(partials, nb, p);
    o[0] = p[0];
  } else {
    sum_partials<2>(partials, nb, o);
  }
  if (threadIdx.x) return;
  if (GCR) gcr_end(sc, o[0], 0.0, 0);
  else bicgstab_end(sc, o[0], o[1], 0.0, 0);
}

// omega = (t.s)/(t.t) from the product's partials, x += alpha ph + omega sh,
// r = s - omega t; partials r.r, rh.r
template <class TV>
__global__ void __launch_bounds__(KB) k_x_update(int n, TV* x, TV* r, const TV* __restrict__ ph,
                                                  const TV* __restrict__ sh, const TV* __restrict__ t,
                                                  const TV* __restrict__ rh, const double* __restrict__ in, int nb,
                                                  double* partials, KScal* sc) {
  if (sc->done) return;
  double o[2];
  sum_partials<2>(in, nb, o);
  const double alpha = sc->alpha, omega = o[1] > 0.0 ? o[0] / o[1] : 0.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) sc->omega = omega;
  double v[2] = {0.0, 0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    x[i] = TV(double(x[i]) + alpha * double(ph[i]) + omega * double(sh[i]));
    const TV rn = TV(double(r[i]) - omega * double(t[i]));
    r[i] = rn;
    v[0] += double(rn) * double(rn);
    v[1] += double(rh[i]) * double(rn);
  }
  block_partials<2>(v, partials);
}

// Segments of a batch: one block per chunk of a segment's rows sums squares,
// and the last block adds each segment's chunks in order into out[] and takes
// the largest sqrt(out[s] / b2[s]) (0 where b2 = 0). END 0: sums only (b2 may be
// null); 1, 2: the convergence test that closes a BiCGStab / GCR iteration;
// 3: the ratio into *ratio.
template <class T, int END>
__global__ void __launch_bounds__(KB) k_segments(Segments sg, const T* __restrict__ v, double* out, const double* b2,
                                                  KScal* sc, double* ratio, const double* __restrict__ partials,
                                                  int nb) {
  if (END == 1 || END == 2)
    if (sc->done) return;
  __shared__ double sh[KB / 32];
  __shared__ bool last;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int q1 = sg.chunk[blockIdx.x + 1];
  double a = 0.0;
  for (int q = sg.chunk[blockIdx.x] + threadIdx.x; q < q1; q += KB) {
    const double x = double(v[__ldg(sg.rows + q)]);
    a += x * x;
  }
  a = warp_sum(a);
  if (l == 0) sh[w] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int i = 0; i < KB / 32; ++i) s += sh[i];
    sg.part[blockIdx.x] = s;
    __threadfence();
    last = atomicInc(sg.ticket, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double m = 0.0;
  for (int s = threadIdx.x; s < sg.nseg; s += KB) {
    double t = 0.0;
    for (int c = sg.chunk_ptr[s]; c < sg.chunk_ptr[s + 1]; ++c) t += __ldcg(sg.part + c);
    out[s] = t;
    if (END) {
      const double b = b2[s];
      if (b > 0.0) m = fmax(m, sqrt(t / b));
    }
  }
  if (!END) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (l == 0) sh[w] = m;
  double o[2] = {0.0, 0.0};
  if (END == 1) sum_partials<2>(partials, nb, o);
  if (END == 2) {
    double p[1];
    sum_partials<1>(partials, nb, p);
    o[0] = p[0];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < KB / 32; ++i) m = fmax(m, sh[i]);
    if (END == 1) bicgstab_end(sc, o[0], o[1], m, sg.nseg);
    if (END == 2) gcr_end(sc, o[0], m, sg.nseg);
    if (END == 3) *ratio = m;
  }
}

// ---------------------------------------------------------------------------
// GCR(2) for scalar systems with a variable-free right preconditioner (Eisenstat,
// Elman and Schultz 1983, truncated to the two latest directions): z = M^-1 r,
// q = A z, orthogonalised against the stored A-images Q0, Q1 (orthonormal)
// with the same combination applied to z, normalised, then x += alpha P,
// r -= alpha Q with alpha = r.Q. One preconditioner application and one SpMV
// per iteration instead of BiCGStab's two of each; the residual norm is
// monotone. Iteration k stores its direction in slot k mod 2; the first two
// iterations find one or both slots empty and leave them out (the coefficients
// of an empty slot are zero).

// q = A z; partials q.Q0, q.Q1
template <class TM, class TV, int FORMAT>
__global__ void __launch_bounds__(KB, 8) k_spmv_gcr(int nn, ScalarMat<TM> M, const TV* __restrict__ z,
                                                  TV* __restrict__ q, const TV* __restrict__ Q0,
                                                  const TV* __restrict__ Q1, double* partials, const KScal* sc) {
  if (sc->done) return;
  const int have = sc->iters;
  double v[2] = {0.0, 0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
    const double q0 = have > 0 ? double(Q0[i]) : 0.0, q1 = have > 1 ? double(Q1[i]) : 0.0;
    const TV qs = TV(scalar_row<FORMAT, TM, TV>(M, i, z));
    q[i] = qs;
    v[0] += double(qs) * q0;
    v[1] += double(qs) * q1;
  }
  block_partials<2>(v, partials);
}

// beta_j = q.Q_j from the product's partials, z -= beta0 P0 + beta1 P1, q -=
// beta0 Q0 + beta1 Q1; partials q.q, r.q
template <class TV>
__global__ void __launch_bounds__(KB) k_gcr_orth(int n, TV* z, TV* q, const TV* __restrict__ P0,
                                                  const TV* __restrict__ P1, const TV* __restrict__ Q0,
                                                  const TV* __restrict__ Q1, const TV* __restrict__ r,
                                                  const double* __restrict__ in, int nb, double* partials,
                                                  const KScal* sc) {
  if (sc->done) return;
  const int have = sc->iters;
  double be[2];
  sum_partials<2>(in, nb, be);
  const double b0 = be[0], b1 = be[1];
  double v[2] = {0.0, 0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double zi = double(z[i]), qi = double(q[i]);
    if (have > 0) {
      zi -= b0 * double(P0[i]);
      qi -= b0 * double(Q0[i]);
    }
    if (have > 1) {
      zi -= b1 * double(P1[i]);
      qi -= b1 * double(Q1[i]);
    }
    if (have > 0) z[i] = TV(zi);
    const TV qn = TV(qi);
    if (have > 0) q[i] = qn;
    v[0] += double(qn) * double(qn);
    v[1] += double(r[i]) * double(qn);
  }
  block_partials<2>(v, partials);
}

// 1/|q| and alpha = r.q / |q| from the partials (a vanishing q is a breakdown),
// P = z / |q|, Q = q / |q| into the oldest slot, x += alpha P, r -= alpha Q;
// partial r.r
template <class TV>
__global__ void __launch_bounds__(KB) k_gcr_update(int n, TV* x, TV* r, const TV* __restrict__ z,
                                                    const TV* __restrict__ q, TV* __restrict__ P, TV* __restrict__ Q,
                                                    const double* __restrict__ in, int nb, double* partials,
                                                    KScal* sc) {
  if (block_done(sc)) return;
  double o[2];
  sum_partials<2>(in, nb, o);
  const double nq = sqrt(o[0]);
  if (!(nq > 0.0) || !(nq < INFINITY)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      sc->done = 1;
      sc->status = nq < INFINITY ? 1 : 2;
    }
    return;
  }
  const double inv = 1.0 / nq, al = o[1] / nq;
  double v[1] = {0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const TV pi = TV(double(z[i]) * inv), qi = TV(double(q[i]) * inv);
    P[i] = pi;
    Q[i] = qi;
    x[i] = TV(double(x[i]) + al * double(pi));
    const TV rn = TV(double(r[i]) - al * double(qi));
    r[i] = rn;
    v[0] += double(rn) * double(rn);
  }
  block_partials<1>(v, partials);
}

// ---------------------------------------------------------------------------
template <int B, class TM, class TV>
int KrylovSolver<B, TM, TV>::setup(int nn_, const int* rp_, const int* cols_, const int* dg_, cudaStream_t st_) {
  if (nn == nn_ && rp == rp_) return OA_OK;
  release();
  nn = nn_;
  rp = rp_;
  cols = cols_;
  dg = dg_;
  st = st_;
  const size_t n = (size_t)B * nn;
  for (int k = 0; k < 8; ++k) OA_CUDA(cudaMalloc(&vec[k], sizeof(TV) * n));
  OA_CUDA(cudaMalloc(&Minv, sizeof(double) * (size_t)B * B * nn));
  OA_CUDA(cudaMalloc(&partials, sizeof(double) * KRYLOV_PARTIALS));
  OA_CUDA(cudaMalloc(&scal, sizeof(KScal)));
  OA_CUDA(cudaMallocHost(&hscal, sizeof(KScal)));
  return OA_OK;
}

template <int B, class TM, class TV>
size_t KrylovSolver<B, TM, TV>::storage_bytes(int nn_) {
  const size_t n = (size_t)B * nn_;
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  return 8 * up(sizeof(TV) * n) + up(sizeof(double) * (size_t)B * B * nn_) + up(sizeof(double) * KRYLOV_PARTIALS) +
         up(sizeof(KScal));
}

template <int B, class TM, class TV>
int KrylovSolver<B, TM, TV>::attach(int nn_, const int* rp_, const int* cols_, const int* dg_, cudaStream_t st_,
                                    void* storage, size_t bytes) {
  release();
  if (bytes < storage_bytes(nn_)) return fail(OA_ERR_ARG, "Krylov: caller storage too small");
  nn = nn_;
  rp = rp_;
  cols = cols_;
  dg = dg_;
  st = st_;
  external = true;
  const size_t n = (size_t)B * nn;
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  char* p = static_cast<char*>(storage);
  for (int k = 0; k < 8; ++k) {
    vec[k] = p;
    p += up(sizeof(TV) * n);
  }
  Minv = reinterpret_cast<double*>(p);
  p += up(sizeof(double) * (size_t)B * B * nn);
  partials = reinterpret_cast<double*>(p);
  p += up(sizeof(double) * KRYLOV_PARTIALS);
  scal = p;
  return OA_OK;
}

template <int B, class TM, class TV>
void KrylovSolver<B, TM, TV>::release() {
  if (!external) {
    for (auto& v : vec)
      if (v) cudaFree(v);
    if (Minv) cudaFree(Minv);
    if (partials) cudaFree(partials);
    if (scal) cudaFree(scal);
  }
  for (auto& v : vec) v = nullptr;
  external = false;
  if (hscal) cudaFreeHost(hscal);
  if (graph_exec) cudaGraphExecDestroy(graph_exec);
  graph_exec = nullptr;
  graph_A = nullptr;
  graph_amg = nullptr;
  Minv = nullptr;
  partials = nullptr;
  scal = nullptr;
  hscal = nullptr;
  nn = 0;
  rp = nullptr;
}

template <int B, class TM, class TV>
bool KrylovSolver<B, TM, TV>::uses_amg() const {
  return B == 1 && std::is_same<TM, TV>::value && amg != nullptr;
}

template <int B, class TM, class TV>
int KrylovSolver<B, TM, TV>::precond(const TV* in, TV* out) {
  if constexpr (B == 1 && std::is_same<TM, TV>::value)
    if (amg) return amg->apply(in, out, &static_cast<KScal*>(scal)->done, st);
  return OA_OK;
}

// x = 0, r = b (rh = b), the inverse (block) diagonal of the Jacobi
// preconditioner, device scalars
template <int B, class TM, class TV>
template <class TB>
int KrylovSolver<B, TM, TV>::prologue(const TM* A, const TB* b, double rtol, int maxit, const double* rtol_dev,
                                      const int* maxit_dev, bool use_gcr) {
  const int n = B * nn;
  KScal* sc = static_cast<KScal*>(scal);
  const int gv = reduce_grid(n);
  if (!uses_amg()) {
    k_build_minv<B, TM, TV><<<(nn + KB - 1) / KB, KB, 0, st>>>(nn, rp, dg, A, reinterpret_cast<TV*>(Minv));
    count_launches(1);
  }
  k_init<TV, TB><<<gv, KB, 0, st>>>(n, b, static_cast<TV*>(vec[0]), static_cast<TV*>(vec[1]),
                                    use_gcr ? nullptr : static_cast<TV*>(vec[2]), partials);
  k_init_scalars<<<1, KB, 0, st>>>(sc, partials, gv, rtol, maxit, rtol_dev, maxit_dev);
  count_launches(2);
  if (seg.on()) {
    k_segments<TB, 0><<<seg.nchunk, KB, 0, st>>>(seg, b, seg.b2, nullptr, nullptr, nullptr, nullptr, 0);
    count_launches(1);
  }
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}

// one chunk of check_every iterations; every kernel reads its scalars and the
// tolerance from device memory, so a chunk can be captured once and replayed
template <int B, class TM, class TV>
int KrylovSolver<B, TM, TV>::chunk(const TM* A, int check_every, bool use_gcr) {
  const int n = B * nn;
  TV *x = static_cast<TV*>(vec[0]), *r = static_cast<TV*>(vec[1]), *rh = static_cast<TV*>(vec[2]),
     *p = static_cast<TV*>(vec[3]), *v = static_cast<TV*>(vec[4]), *ph = static_cast<TV*>(vec[5]),
     *sh = static_cast<TV*>(vec[6]), *t = static_cast<TV*>(vec[7]);
  KScal* sc = static_cast<KScal*>(scal);
  const int gv = reduce_grid(n);
  // two sets of partials: a kernel reads the one and writes the other
  double *pa = partials, *pb = partials + 2 * MAX_PARTIALS;
  const ScalarMat<TM> M = {rp, cols, A, ell_mat(ell, static_cast<const TM*>(ell_val))};
  const int format = B == 1 && ell_val ? ell_format(ell.w, ell.slots, sizeof(TM)) : 1;
  if (use_gcr) {
    // GCR(2) work vectors in the same buffers: x r z q P0 P1 Q0 Q1
    TV *gz = rh, *gq = p, *gP[2] = {v, ph}, *gQ[2] = {sh, t};
    for (int it = 0; it < check_every; ++it) {
      const int slot = it & 1;  // the older of the two stored directions
      if (int s = precond(r, gz)) return s;
#define OA_CALL(F) k_spmv_gcr<TM, TV, F><<<gv, KB, 0, st>>>(nn, M, gz, gq, gQ[0], gQ[1], pa, sc)
      OA_FORMAT(format, OA_CALL)
#undef OA_CALL
      k_gcr_orth<TV><<<gv, KB, 0, st>>>(n, gz, gq, gP[0], gP[1], gQ[0], gQ[1], r, pa, gv, pb, sc);
      k_gcr_update<TV><<<gv, KB, 0, st>>>(n, x, r, gz, gq, gP[slot], gQ[slot], pb, gv, pa, sc);
      if (seg.on())
        k_segments<TV, 2><<<seg.nchunk, KB, 0, st>>>(seg, r, seg.r2, seg.b2, sc, nullptr, pa, gv);
      else
        k_end_iter<true><<<1, KB, 0, st>>>(sc, pa, gv);
      count_launches(4);
    }
    OA_CUDA(cudaGetLastError());
    return OA_OK;
  }
  const TV* Mi = uses_amg() ? nullptr : reinterpret_cast<const TV*>(Minv);
  const int gr = (nn + KB - 1) / KB;
  for (int it = 0; it < check_every; ++it) {
    k_p_update<B, TV><<<gr, KB, 0, st>>>(nn, p, r, v, Mi, ph, sc);
    if (int s = precond(p, ph)) return s;
#define OA_CALL(F) k_spmv<B, TM, TV, 1, B == 1 ? F : 1><<<gv, KB, 0, st>>>(nn, M, ph, v, rh, pa, sc)
    OA_FORMAT(format, OA_CALL)
#undef OA_CALL
    k_s_update<B, TV><<<reduce_grid(nn), KB, 0, st>>>(nn, r, v, Mi, sh, pa, gv, sc);
    if (int s = precond(r, sh)) return s;
#define OA_CALL(F) k_spmv<B, TM, TV, 2, B == 1 ? F : 1><<<gv, KB, 0, st>>>(nn, M, sh, t, r, pb, sc)
    OA_FORMAT(format, OA_CALL)
#undef OA_CALL
    k_x_update<TV><<<gv, KB, 0, st>>>(n, x, r, ph, sh, t, rh, pb, gv, pa, sc);
    if (seg.on())
      k_segments<TV, 1><<<seg.nchunk, KB, 0, st>>>(seg, r, seg.r2, seg.b2, sc, nullptr, pa, gv);
    else
      k_end_iter<false><<<1, KB, 0, st>>>(sc, pa, gv);
    count_launches(6);
  }
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}

template <int B, class TM, class TV>
template <class TB>
int KrylovSolver<B, TM, TV>::solve(const TM* A, const TB* b, TV*& xout, double rtol, int maxit, int* iters,
                                   double* res, int check_every, bool reuse_precond) {
  constexpr bool kAmgOk = (B == 1) && std::is_same<TM, TV>::value;
  KScal* sc = static_cast<KScal*>(scal);
  const bool use_gcr = gcr && B == 1;
  if (use_gcr && check_every % 2) return fail(OA_ERR_ARG, "GCR: iteration chunks must hold an even number of iterations");
  // OA_DEBUG: device time of the preconditioner set-up and of the whole solve
  const bool dbg = std::getenv("OA_DEBUG") != nullptr;
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
  if (dbg)
    for (auto& e : ev) {
      cudaEventCreate(&e);
    }
  if (dbg) cudaEventRecord(ev[0], st);
  if constexpr (kAmgOk) {
    if (amg && !reuse_precond) {
      if (int s = amg->numeric(reinterpret_cast<const TV*>(A), st)) return s;
    }
  }
  if (dbg) cudaEventRecord(ev[1], st);
  if (int s = prologue<TB>(A, b, rtol, maxit, nullptr, nullptr, use_gcr)) return s;
  if (use_graph && (graph_exec == nullptr || graph_A != (const void*)A || graph_chunk != check_every ||
                    graph_amg != (const void*)amg || graph_gcr != use_gcr)) {
    if (graph_exec) cudaGraphExecDestroy(graph_exec);
    graph_exec = nullptr;
    cudaGraph_t g;
    OA_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    const long long l0 = launch_total();
    const int cs = chunk(A, check_every, use_gcr);
    const long long per_chunk = launch_total() - l0;
    const cudaError_t ce = cudaStreamEndCapture(st, &g);
    if (cs) return cs;
    if (ce != cudaSuccess) return fail(OA_ERR_CUDA, std::string("Krylov chunk capture: ") + cudaGetErrorString(ce));
    OA_CUDA(cudaGraphInstantiate(&graph_exec, g, 0));
    cudaGraphDestroy(g);
    graph_A = A;
    graph_amg = amg;
    graph_chunk = check_every;
    graph_gcr = use_gcr;
    graph_launches = per_chunk;
    count_launches(-per_chunk);  // captured, not launched
  }
  int done_iters = 0;
  while (true) {
    if (use_graph) {
      OA_CUDA(cudaGraphLaunch(graph_exec, st));
      count_launches(graph_launches);
    } else if (int s = chunk(A, check_every, use_gcr)) {
      return s;
    }
    done_iters += check_every;
    // pinned staging when the solver owns its storage, else plain host memory
    void* hdst = hscal ? hscal : static_cast<void*>(hbuf);
    OA_CUDA(cudaMemcpyAsync(hdst, sc, sizeof(KScal), cudaMemcpyDeviceToHost, st));
    OA_CUDA(cudaStreamSynchronize(st));
    const KScal* h = static_cast<const KScal*>(hdst);
    if (h->done || done_iters >= maxit) break;
  }
  const KScal* h = static_cast<const KScal*>(hscal ? hscal : static_cast<void*>(hbuf));
  static_assert(sizeof(KScal) <= sizeof(hbuf), "host staging buffer too small");
  if (iters) *iters = h->iters;
  if (res) *res = seg.on() ? h->seg_rel : (h->bnorm > 0 ? h->rnorm / h->bnorm : 0.0);
  xout = static_cast<TV*>(vec[0]);
  last_status = h->status;
  if (dbg) {
    cudaEventRecord(ev[2], st);
    cudaEventSynchronize(ev[2]);
    float t_setup = 0.f, t_all = 0.f;
    cudaEventElapsedTime(&t_setup, ev[0], ev[1]);
    cudaEventElapsedTime(&t_all, ev[0], ev[2]);
    std::fprintf(stderr, "[oa] %s<%d,%s> n %d iters %d: precond set-up %.3f ms, solve %.3f ms\n",
                 use_gcr ? "GCR(2)" : "BiCGStab", B, sizeof(TV) == 4 ? "f32" : "f64", nn, h->iters, t_setup, t_all);
    for (auto& e : ev) cudaEventDestroy(e);
  }
  if (h->status == 2) return fail(OA_ERR_SOLVER, use_gcr ? "GCR: non-finite residual" : "BiCGStab: non-finite residual");
  return OA_OK;
}

template <int B, class TM, class TV>
template <class TB>
int KrylovSolver<B, TM, TV>::emit(GraphBuild& gb, cudaGraph_t g, Deps& d, int body, const TM* A, const TB* b,
                                  double rtol, int maxit, const double* rtol_dev, const int* maxit_dev, int maxit_cap,
                                  int check_every, bool gcr_mode, int branch_body) {
  const bool use_gcr = gcr_mode && B == 1;
  if (use_gcr && check_every % 2) return fail(OA_ERR_ARG, "GCR: iteration chunks must hold an even number of iterations");
  if (st != gb.st) return fail(OA_ERR_ARG, "Krylov graph: the solver's stream is not the capturing stream");
  const int lb = gb.new_body();
  if (lb < 0) return fail(OA_ERR_ARG, "Krylov graph: too many conditional bodies");
  cudaGraphConditionalHandle h;
  if (int s = gb.handle(g, &h)) return s;
  if (int s = gb.seg(g, d, body, [&]() -> int {
        if (int s2 = prologue<TB>(A, b, rtol, maxit, rtol_dev, maxit_dev, use_gcr)) return s2;
        return launch_loop_enter(gb, h, scal, lb, branch_body);
      }))
    return s;
  cudaGraph_t wb = nullptr;
  if (int s = gb.cond(g, d, h, cudaGraphCondTypeWhile, 1, &wb)) return s;
  Deps bd;
  const int cap = (maxit_cap + check_every - 1) / check_every + 2;
  return gb.seg(wb, bd, lb, [&]() -> int {
    if (int s2 = chunk(A, check_every, use_gcr)) return s2;
    return launch_loop_next(gb, h, scal, lb, cap);
  });
}

template struct KrylovSolver<1, double, double>;
template struct KrylovSolver<3, double, double>;
template struct KrylovSolver<1, float, float>;
template struct KrylovSolver<3, float, float>;
template int KrylovSolver<1, double, double>::solve<double>(const double*, const double*, double*&, double, int, int*, double*, int, bool);
template int KrylovSolver<3, double, double>::solve<double>(const double*, const double*, double*&, double, int, int*, double*, int, bool);
template int KrylovSolver<1, float, float>::solve<double>(const float*, const double*, float*&, double, int, int*, double*, int, bool);
template int KrylovSolver<1, float, float>::solve<float>(const float*, const float*, float*&, double, int, int*, double*, int, bool);
template int KrylovSolver<3, float, float>::solve<float>(const float*, const float*, float*&, double, int, int*, double*, int, bool);
#define OA_EMIT(B, TM, TV, TB)                                                                                   \
  template int KrylovSolver<B, TM, TV>::emit<TB>(GraphBuild&, cudaGraph_t, Deps&, int, const TM*, const TB*, double, \
                                                 int, const double*, const int*, int, int, bool, int);
OA_EMIT(1, double, double, double)
OA_EMIT(3, double, double, double)
OA_EMIT(1, float, float, float)
OA_EMIT(3, float, float, float)
#undef OA_EMIT

// ---------------------------------------------------------------------------
// fixed-width storage
// One warp per group. Its distances are merged from the rows' column lists, the
// smallest next one first, so that every row keeps its order.
__global__ void __launch_bounds__(32) k_ell_graph(int n, int w, const int* rp, const int* cols, int* out, int* delta,
                                                  uint16_t* mask) {
  const int i = blockIdx.x * 32 + threadIdx.x;
  const int a = i < n ? rp[i] : 0, len = i < n ? rp[i + 1] - a : 0;
  int* d = delta + (size_t)blockIdx.x * (w + 1);
  int at = 0;
  unsigned have = 0;
  for (int q = 0; q < w; ++q) {
    const int next = at < len ? cols[a + at] - i : INT_MAX;
    const int m = __reduce_min_sync(0xffffffffu, next);
    if (next == m && m != INT_MAX) {
      have |= 1u << q;
      ++at;
    }
    if (threadIdx.x == 0) d[q] = m == INT_MAX ? 0 : m;
  }
  const bool columns = w != ELL_DISTANCES || __any_sync(0xffffffffu, at < len);
  const int pad = len ? cols[a] : 0;
  if (threadIdx.x == 0) d[w] = columns;
  mask[i] = (uint16_t)(columns ? (1u << len) - 1 : have);
  for (int q = 0; q < w; ++q) out[(size_t)blockIdx.x * 32 * w + 32 * q + threadIdx.x] = q < len ? cols[a + q] : pad;
}

template <class T, int W>
__global__ void __launch_bounds__(256) k_ell_values(int n, const int* __restrict__ rp,
                                                    const uint16_t* __restrict__ mask, const T* __restrict__ csr,
                                                    T* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (n + 31) / 32 * 32) return;
  const int a = i < n ? __ldg(rp + i) : 0;
  const unsigned have = __ldg(mask + i);
  T v[W];
#pragma unroll
  for (int q = 0; q < W; ++q) v[q] = have >> q & 1 ? __ldg(csr + a + __popc(have & ((1u << q) - 1))) : T(0);
#pragma unroll
  for (int q = 0; q < W; ++q) out[(size_t)(i >> 5) * 32 * W + 32 * q + (i & 31)] = v[q];
}

// Bytes per row that stay free beside storage of this kind: more than a program
// takes from the mesh on. A 24^3 flow with its solvers holds 3.2 KB per row in
// FP64 and 2.6 in the mixed form, conduction on 17^3 nodes 3.0 and 2.5; the k
// and omega systems add 0.5, the autotuner 0.3.
constexpr size_t SPARE_BYTES_PER_ROW = 4096;

void* spare_alloc(size_t bytes, long long rows) {
  size_t free_bytes = 0, total = 0;
  if (cudaMemGetInfo(&free_bytes, &total) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  if (free_bytes < bytes || free_bytes - bytes < SPARE_BYTES_PER_ROW * (size_t)rows) return nullptr;
  void* p = nullptr;
  if (cudaMalloc(&p, bytes) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return p;
}

int ell_graph(int n, const int* h_rp, const int* rp, const int* cols, EllGraph* out, cudaStream_t st) {
  *out = EllGraph{};
  int longest = 0;
  for (int i = 0; i < n; ++i) longest = std::max(longest, h_rp[i + 1] - h_rp[i]);
  const int w = longest <= 7 ? 7 : 15;
  const long long groups = (n + 31LL) / 32, slots = groups * 32 * w;
  if (longest > w || slots > 2LL * h_rp[n] + 4096) return OA_OK;
  int* c = static_cast<int*>(spare_alloc(sizeof(int) * (slots + groups * (w + 1)) + sizeof(uint16_t) * groups * 32, n));
  if (!c) return OA_OK;
  int* delta = c + slots;
  uint16_t* mask = reinterpret_cast<uint16_t*>(delta + groups * (w + 1));
  out->w = w;
  out->cols = c;
  out->delta = delta;
  out->mask = mask;
  out->slots = slots;
  if (groups == 0) return OA_OK;
  k_ell_graph<<<(unsigned)groups, 32, 0, st>>>(n, w, rp, cols, c, delta, mask);
  count_launches(1);
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}

template <class T>
int ell_values(int n, const int* rp, const T* csr, const EllGraph& gr, T* out, cudaStream_t st) {
  const int g = ((n + 31) / 32 * 32 + 255) / 256;
  if (gr.w == 7) k_ell_values<T, 7><<<g, 256, 0, st>>>(n, rp, gr.mask, csr, out);
  else k_ell_values<T, 15><<<g, 256, 0, st>>>(n, rp, gr.mask, csr, out);
  count_launches(1);
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}
template int ell_values<float>(int, const int*, const float*, const EllGraph&, float*, cudaStream_t);
template int ell_values<double>(int, const int*, const double*, const EllGraph&, double*, cudaStream_t);

// ---------------------------------------------------------------------------
// FP64 residual for iterative refinement: r = b - A x (A in its stored
// precision, arithmetic in FP64), with partial ||r||^2.
template <class TM, int FORMAT>
__global__ void __launch_bounds__(KB) k_residual(int nn, ScalarMat<TM> M, const double* __restrict__ x,
                                                  const double* __restrict__ b, double* __restrict__ r,
                                                  double* partials) {
  double v[1] = {0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
    const double bi = b[i];
    const double ri = bi - scalar_row<FORMAT, TM, double>(M, i, x);
    r[i] = ri;
    v[0] += ri * ri;
  }
  block_partials<1>(v, partials);
}

template <bool ROOT, int NV>
__global__ void __launch_bounds__(KB) k_sums_out(const double* partials, int nb, double* out) {
  double o[NV];
  sum_partials<NV>(partials, nb, o);
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) out[k] = ROOT ? sqrt(o[k]) : o[k];
}

template <class TV>
__global__ void k_add_correction(int n, double* x, const TV* d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] += double(d[i]);
}

template <class TM>
int KrylovMatrix<TM>::residual(int nn, const double* x, const double* b, double* r, double* partials,
                               double* norm_dev, cudaStream_t st) const {
  const int g = reduce_grid(nn);
  const ScalarMat<TM> M = {rp, cols, A, ell_mat(ell, eval)};
#define OA_CALL(F) k_residual<TM, F><<<g, KB, 0, st>>>(nn, M, x, b, r, partials)
  OA_FORMAT(eval ? ell_format(ell.w, ell.slots, sizeof(TM)) : 1, OA_CALL)
#undef OA_CALL
  k_sums_out<true, 1><<<1, KB, 0, st>>>(partials, g, norm_dev);
  count_launches(2);
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}
template struct KrylovMatrix<float>;

__global__ void __launch_bounds__(KB) k_sumsq(int n, const double* __restrict__ v, double* partials) {
  double s[1] = {0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) s[0] += v[i] * v[i];
  block_partials<1>(s, partials);
}

int device_sumsq(int n, const double* v, double* out, double* partials, cudaStream_t st) {
  const int g = reduce_grid(n);
  k_sumsq<<<g, KB, 0, st>>>(n, v, partials);
  k_sums_out<false, 1><<<1, KB, 0, st>>>(partials, g, out);
  count_launches(2);
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}

int partials_size() { return 6 * MAX_PARTIALS; }

// per-component sums of squares of two [nn][3] vectors
template <class T>
__global__ void __launch_bounds__(KB) k_comp_sumsq3(int nn, const T* __restrict__ a, const T* __restrict__ b,
                                                     double* partials) {
  double s[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double p = double(a[3 * (size_t)i + k]), q = double(b[3 * (size_t)i + k]);
      s[k] += p * p;
      s[3 + k] += q * q;
    }
  block_partials<6>(s, partials);
}

template <class T>
int device_comp_sumsq3(int nn, const T* a, const T* b, double* out, double* partials, cudaStream_t st) {
  const int g = reduce_grid(nn);
  k_comp_sumsq3<T><<<g, KB, 0, st>>>(nn, a, b, partials);
  k_sums_out<false, 6><<<1, KB, 0, st>>>(partials, g, out);
  count_launches(2);
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}
template int device_comp_sumsq3<float>(int, const float*, const float*, double*, double*, cudaStream_t);
template int device_comp_sumsq3<double>(int, const double*, const double*, double*, double*, cudaStream_t);

template <class TV>
int add_correction(int n, double* x, const TV* d, cudaStream_t st) {
  k_add_correction<TV><<<(n + KB - 1) / KB, KB, 0, st>>>(n, x, d);
  count_launches(1);
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}
template int add_correction<float>(int, double*, const float*, cudaStream_t);
template int add_correction<double>(int, double*, const double*, cudaStream_t);

template <class T>
int segment_sumsq(const Segments& sg, const T* v, double* out, cudaStream_t st) {
  if (!sg.on()) return OA_OK;
  k_segments<T, 0><<<sg.nchunk, KB, 0, st>>>(sg, v, out, nullptr, nullptr, nullptr, nullptr, 0);
  count_launches(1);
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}
template int segment_sumsq<float>(const Segments&, const float*, double*, cudaStream_t);
template int segment_sumsq<double>(const Segments&, const double*, double*, cudaStream_t);

int segment_ratio(const Segments& sg, const double* v, double* out, cudaStream_t st) {
  k_segments<double, 3><<<sg.nchunk, KB, 0, st>>>(sg, v, sg.r2, sg.b2, nullptr, out, nullptr, 0);
  count_launches(1);
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}

// ---------------------------------------------------------------------------
// Control kernels of the conditional nodes of whole-iteration graphs (one
// thread each; the condition is set by the graph that holds the node, or by
// the node's own body).
namespace {
__global__ void k_set_if(cudaGraphConditionalHandle h, const int* flag, int negate) {
  cudaGraphSetConditional(h, ((*flag != 0) != (negate != 0)) ? 1u : 0u);
}
__global__ void k_count_body(BodyCounters* c, int body) { c->total[body] += 1; }
__global__ void k_loop_enter(cudaGraphConditionalHandle h, const KScal* sc, BodyCounters* c, int body,
                             int branch_body) {
  c->cur[body] = 0;
  if (branch_body >= 0) c->total[branch_body] += 1;
  cudaGraphSetConditional(h, sc->done ? 0u : 1u);
}
__global__ void k_loop_next(cudaGraphConditionalHandle h, const KScal* sc, BodyCounters* c, int body, int cap) {
  const int n = ++c->cur[body];
  c->total[body] += 1;
  cudaGraphSetConditional(h, (!sc->done && n < cap) ? 1u : 0u);
}
}  // namespace

int launch_set_if(GraphBuild& gb, cudaGraphConditionalHandle h, const int* flag, bool negate) {
  k_set_if<<<1, 1, 0, gb.st>>>(h, flag, negate ? 1 : 0);
  count_launches(1);
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}
int launch_count_body(GraphBuild& gb, int body) {
  k_count_body<<<1, 1, 0, gb.st>>>(gb.ctr, body);
  count_launches(1);
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}
int launch_loop_enter(GraphBuild& gb, cudaGraphConditionalHandle h, const void* kscal, int body, int branch_body) {
  k_loop_enter<<<1, 1, 0, gb.st>>>(h, static_cast<const KScal*>(kscal), gb.ctr, body, branch_body);
  count_launches(1);
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}
int launch_loop_next(GraphBuild& gb, cudaGraphConditionalHandle h, const void* kscal, int body, int cap) {
  k_loop_next<<<1, 1, 0, gb.st>>>(h, static_cast<const KScal*>(kscal), gb.ctr, body, cap);
  count_launches(1);
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}
int launch_counters_reset(GraphBuild& gb) {
  OA_CUDA(cudaMemsetAsync(gb.ctr, 0, sizeof(BodyCounters), gb.st));
  return OA_OK;
}

}  // namespace oa
