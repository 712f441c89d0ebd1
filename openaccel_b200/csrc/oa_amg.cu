// Aggregation AMG V-cycle for the pressure-correction system (see oa_amg.h).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <vector>

#include "oa_amg.h"
#include "oa_amg_symbolic.h"
#include "oa_internal.h"

namespace oa {

constexpr int AB = 256;          // threads per block
constexpr int COARSE_MAX = 256;  // coarsest level solved by a dense inverse
constexpr int MAX_CHEB = 6;      // highest Chebyshev smoothing degree

constexpr int CLUSTER_THREADS = 1024;
constexpr int CLUSTER_BLOCKS = 16;

// The V-cycle from a level of at most DENSE_ROWS rows down is one dense operator
// (see dense_operator below).
constexpr int DENSE_ROWS = 1024;
constexpr int DENSE_COLS = 512;  // columns formed at a time

// Lanes per row of the row-parallel kernels of a level with `rows` rows of
// `avg` entries: levels with many rows keep one lane per row for short rows
// and take 8 for long ones; smaller levels spread each row over a group of
// lanes so that the few rows still fill the SMs. OA_AMG_LANES_BIG overrides
// the choice for long rows on large levels. On smaller levels up to 64 entries
// take 8 lanes above 12,000 rows (20,352 rows of 29 on a 61x53x47 block, 38,000 on a
// 128x48x48 channel) and 32 below: with 32 from 24 entries on, whatever the rows, a
// pass takes 8.95 instead of 8.11 ms (61x53x47), 13.2 instead of 11.5 (channel) and
// 14.1 instead of 13.1 (16 cavities). 4 or 8 lanes up to 12 entries make no
// difference in any of these.
static int lanes_for(double avg, long long rows) {
  if (rows >= 100000) {
    if (avg <= 16.0) return 1;
    static const int big = [] {
      const char* e = std::getenv("OA_AMG_LANES_BIG");
      const int v = e ? std::atoi(e) : 0;
      return (v == 1 || v == 4 || v == 8 || v == 32) ? v : 0;
    }();
    if (big) return big;
    return 8;
  }
  return avg <= 4.0 ? 1 : (avg <= 12.0 ? 4 : (rows > 12000 && avg <= 64.0 ? 8 : 32));
}

// Lanes per row in the cluster of the power iteration (16,384 threads).
__device__ __forceinline__ int cluster_lanes(int n, int nnz) { return nnz <= 4 * n ? 1 : (nnz <= 24 * n ? 4 : 16); }

static unsigned grid_for(long long rows, int lpr) { return (unsigned)((rows * lpr + AB - 1) / AB); }


template <class T>
static int upload(T** d, const std::vector<T>& h) {
  if (cudaMalloc(d, sizeof(T) * std::max<size_t>(1, h.size())) != cudaSuccess)
    return fail(OA_ERR_CUDA, "AMG: device allocation failed");
  if (!h.empty() && cudaMemcpy(*d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice) != cudaSuccess)
    return fail(OA_ERR_CUDA, "AMG: upload failed");
  return OA_OK;
}

template <class T>
static int dalloc(T** d, size_t n) {
  if (cudaMalloc(d, sizeof(T) * std::max<size_t>(1, n)) != cudaSuccess)
    return fail(OA_ERR_CUDA, "AMG: device allocation failed");
  return OA_OK;
}

template <class T>
void Amg<T>::release() {
  for (size_t l = 0; l < L.size(); ++l) {
    AmgLevel<T>& v = L[l];
    if (l > 0) {
      cudaFree(v.rp);
      cudaFree(v.cols);
      cudaFree(v.diag);
    }
    if (v.own_A) cudaFree(v.A);
    void* p[] = {v.dinv,   v.agg,   v.mptr,   v.mlist, v.gptr,   v.glist, v.r,      v.t,    v.p_rp,
                 v.p_cols, v.p_diag, v.pg_ptr, v.pg_list, v.pv, v.ptv, v.pt_rp, v.pt_rows, v.pt_src, v.tv,
                 v.tt_ptr, v.tt_a,   v.tt_p,   v.ct_ptr, v.ct_p, v.ct_t, v.cr,      v.cd0,  v.cd1,
                 v.est,    v.coef,  v.pw_v, v.pw_w,   v.pw_part, v.pw_ticket};
    for (void* q : p)
      if (q) cudaFree(q);
    if (l > 0) {
      cudaFree(v.x);
      cudaFree(v.b);
    }
  }
  L.clear();
  if (dense_inv) cudaFree(dense_inv);
  if (dense_op) cudaFree(dense_op);
  operator_stale = false;
  dense_inv = nullptr;
  dense_op = nullptr;
  dense_work = nullptr;
  ready = false;
}

// ---------------------------------------------------------------------------
// kernels
template <class T>
__global__ void k_galerkin(int nnz_c, const int* __restrict__ gptr, const int* __restrict__ glist,
                           const T* __restrict__ Af, T* __restrict__ Ac) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nnz_c) return;
  double s = 0.0;
  for (int q = gptr[c]; q < gptr[c + 1]; ++q) s += double(Af[glist[q]]);
  Ac[c] = T(s);
}

template <class T>
__global__ void k_dinv(int n, const int* __restrict__ rp, const int* __restrict__ dg, const T* __restrict__ A,
                       T* __restrict__ dinv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dinv[i] = T(1.0 / double(A[rp[i] + dg[i]]));
}

// dense copy of the coarsest matrix, augmented with the identity: [A | I]
template <class T>
__global__ void k_dense_fill(int n, const int* __restrict__ rp, const int* __restrict__ cols, const T* __restrict__ A,
                             double* M) {
  const int i = blockIdx.x;
  for (int j = threadIdx.x; j < 2 * n; j += blockDim.x) M[(size_t)i * 2 * n + j] = (j - n == i) ? 1.0 : 0.0;
  __syncthreads();
  for (int k = rp[i] + threadIdx.x; k < rp[i + 1]; k += blockDim.x) M[(size_t)i * 2 * n + cols[k]] = double(A[k]);
}

// Gauss-Jordan elimination without pivoting (the coarse Galerkin operators of
// the grounded Rhie-Chow Laplacian are M-matrices), one block; leaves A^-1 in
// the right half. At step k the pivot row is zero left of column k (earlier
// steps cleared it) and right of column n + k (the identity's later columns
// are still untouched there), so only its n + 1 columns k .. n + k are
// normalised and used: the skipped updates would subtract exact zeros. Only for
// a coarsest level above 256 rows (a hierarchy cut off at its last level).
__global__ void k_gauss_jordan(int n, double* M) {
  const int w = 2 * n;
  for (int k = 0; k < n; ++k) {
    __syncthreads();
    const double piv = M[(size_t)k * w + k];
    __syncthreads();
    for (int j = k + threadIdx.x; j <= n + k; j += blockDim.x) M[(size_t)k * w + j] /= piv;
    __syncthreads();
    // columns k + 1 .. n + k of every other row (n of them)
    for (int idx = threadIdx.x; idx < n * n; idx += blockDim.x) {
      const int i = idx / n, j = k + 1 + (idx - i * n);
      if (i == k) continue;
      M[(size_t)i * w + j] -= M[(size_t)i * w + k] * M[(size_t)k * w + j];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x)
      if (i != k) M[(size_t)i * w + k] = 0.0;
  }
}

// The same elimination in place and in registers for n <= 128 (C = 1 block) or
// n <= 256 (C = 4 blocks of one cluster): every thread keeps 4 x 4 entries, and
// step k replaces column k, which the augmented form would clear, by the
// identity's column k, whose entries the same operations produce. The pivot
// row goes to every block's shared memory and the pivot column to its own
// rows' block, so a step is one barrier, n divisions and one multiply-add per
// entry instead of three passes over the matrix in L2.
template <int C>
__global__ void __launch_bounds__(1024, 1) k_invert(int n, double* M) {
  constexpr int CT = C == 1 ? 32 : 64, RT = 1024 / CT;  // column and row lanes of a block
  __shared__ double prow[2][4 * CT], pcol[2][4 * RT], pn[4 * CT];
  const int w = 2 * n, tc = threadIdx.x % CT, tr = threadIdx.x / CT, row0 = blockIdx.x * 4 * RT;
  double a[4][4];
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = row0 + tr + RT * p, c = tc + CT * q;
      a[p][q] = (r < n && c < n) ? M[(size_t)r * w + c] : 0.0;
    }
  auto publish = [&](int k) {
    double* pr = prow[k & 1];
    double* pc = pcol[k & 1];
#pragma unroll
    for (int p = 0; p < 4; ++p)
      if (row0 + tr + RT * p == k)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (C == 1) {
            pr[tc + CT * q] = a[p][q];
          } else {
            const unsigned at = (unsigned)__cvta_generic_to_shared(pr + tc + CT * q);
#pragma unroll
            for (int b = 0; b < C; ++b)
              asm volatile(
                  "{\n\t.reg .u32 ra;\n\tmapa.shared::cluster.u32 ra, %0, %1;\n\t"
                  "st.shared::cluster.f64 [ra], %2;\n\t}" ::"r"(at),
                  "r"(b), "d"(a[p][q])
                  : "memory");
          }
        }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (tc + CT * q == k)
#pragma unroll
        for (int p = 0; p < 4; ++p) pc[tr + RT * p] = a[p][q];
  };
  auto barrier = [] {
    if (C == 1)
      __syncthreads();
    else
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  };
  barrier();  // every block of the cluster has started before its shared memory is written
  publish(0);
  for (int k = 0; k < n; ++k) {
    barrier();
    const double* pr = prow[k & 1];
    const double* pc = pcol[k & 1];
    if (threadIdx.x < n) pn[threadIdx.x] = ((int)threadIdx.x == k ? 1.0 : pr[threadIdx.x]) / pr[k];
    __syncthreads();
    double f[4], m[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) f[p] = pc[tr + RT * p];
#pragma unroll
    for (int q = 0; q < 4; ++q) m[q] = pn[tc + CT * q];
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double old = tc + CT * q == k ? 0.0 : a[p][q];
        a[p][q] = row0 + tr + RT * p == k ? m[q] : old - f[p] * m[q];
      }
    if (k + 1 < n) publish(k + 1);
  }
  barrier();  // no block leaves while another writes into it
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = row0 + tr + RT * p, c = tc + CT * q;
      if (r < n && c < n) M[(size_t)r * w + n + c] = a[p][q];
    }
}

// Sum of one value per lane over a group of LPR consecutive lanes (a row's
// lanes), by a fixed xor butterfly: the same order every run.
template <int LPR>
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------------
// Row phases of the V-cycle above the dense operator, LPR lanes per row.
//
// A row's entries come in groups of U per lane whose index and value loads are
// all in flight before the first use: the phases are bound by the latency of
// the chain row pointer -> column -> vector, not by the arithmetic.
//
// A kernel reads its vectors through the read-only path; one that walks over a
// vector which other blocks write between two cluster barriers (SHARED) uses
// plain loads, which the barrier's acquire orders.
template <bool SHARED, class T>
__device__ __forceinline__ double ldv(const T* p) {
  return SHARED ? double(*p) : double(__ldg(p));
}

template <int LPR, class T, class G>
__device__ __forceinline__ double row_dot(const int* __restrict__ cols, const T* __restrict__ A, int a, int e,
                                          int lane, G get) {
  constexpr int U = LPR >= 8 ? 2 : 4;
  double s = 0.0;
  for (int k = a + lane; k < e; k += U * LPR) {
    int j[U];
    T v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int q = k + u * LPR < e ? k + u * LPR : k;
      j[u] = __ldg(cols + q);
      v[u] = __ldg(A + q);
    }
    double x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = get(j[u]);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k + u * LPR < e) s += double(v[u]) * x[u];
  }
  return group_sum<LPR>(s);
}

// f(row, lane) over the rows, whole warps together (rows past n included: f
// checks)
template <int FORMAT, class F>
__device__ __forceinline__ void for_rows(int n, F&& f) {
  constexpr int LPR = lanes_of(FORMAT);
  const unsigned total = (unsigned)n * LPR, stride = gridDim.x * blockDim.x;
  for (unsigned g0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); g0 < total; g0 += stride) {
    const unsigned g = g0 + (threadIdx.x & 31u);
    f((int)(g / LPR), (int)(g % LPR));
  }
}

// LPR of ELL or above (finest level): one thread per row over the fixed-width storage.
template <class T>
struct RowMat {
  int n;
  const int *rp, *cols;
  const T* A;
  EllMat<T> ell;
};

template <int LPR, class T, class G>
__device__ __forceinline__ double mat_row(const RowMat<T>& m, int i, int lane, G get) {
  if constexpr (LPR >= ELL) return i < m.n ? ell_row<LPR, T>(m.ell, i, get) : 0.0;
  int a = 0, e = 0;
  if (i < m.n) {
    a = __ldg(m.rp + i);
    e = __ldg(m.rp + i + 1);
  }
  return row_dot<lanes_of(LPR), T>(m.cols, m.A, a, e, lane, get);
}

// Downward step: pre-smooth from zero, xs_i = w Dinv_i b_i, and the residual
// r_i = b_i - sum_j a_ij xs_j (neighbours' xs formed from b).
template <int LPR, class T>
__device__ __forceinline__ void ph_smooth_resid(const RowMat<T>& m, const T* dinv, const T* b, T* xs, T* r, double w) {
  for_rows<LPR>(m.n, [&](int i, int lane) {
    double bi = 0.0, di = 0.0;
    if (i < m.n && lane == 0) {
      bi = ldv<false>(b + i);
      di = double(__ldg(dinv + i));
    }
    const double s = mat_row<LPR>(m, i, lane, [&](int j) { return w * double(__ldg(dinv + j)) * ldv<false>(b + j); });
    if (i >= m.n || lane) return;
    xs[i] = T(w * di * bi);
    r[i] = T(bi - s);
  });
}

// residual r = b - A x
template <int LPR, class T>
__device__ __forceinline__ void ph_resid(const RowMat<T>& m, const T* b, const T* x, T* r) {
  for_rows<LPR>(m.n, [&](int i, int lane) {
    double bi = 0.0;
    if (i < m.n && lane == 0) bi = ldv<false>(b + i);
    const double s = mat_row<LPR>(m, i, lane, [&](int j) { return ldv<false>(x + j); });
    if (i < m.n && lane == 0) r[i] = T(bi - s);
  });
}

// restriction bc = P^T r over the coarse rows (m: P^T)
template <int LPR, class T>
__device__ __forceinline__ void ph_restrict(const RowMat<T>& m, const T* r, T* bc) {
  for_rows<LPR>(m.n, [&](int i, int lane) {
    const double s = mat_row<LPR>(m, i, lane, [&](int j) { return ldv<false>(r + j); });
    if (i < m.n && lane == 0) bc[i] = T(s);
  });
}

// coarse correction in place: t_i += alpha (P xc)_i (m: P)
template <int LPR, class T>
__device__ __forceinline__ void ph_prolong_add(const RowMat<T>& m, const T* xc, T* t, double alpha) {
  for_rows<LPR>(m.n, [&](int i, int lane) {
    double ti = 0.0;
    if (i < m.n && lane == 0) ti = double(t[i]);
    const double s = mat_row<LPR>(m, i, lane, [&](int j) { return ldv<false>(xc + j); });
    if (i < m.n && lane == 0) t[i] = T(ti + alpha * s);
  });
}

// post-smooth out of place: x_i = t_i + w Dinv_i (b_i - sum_j a_ij t_j)
template <int LPR, class T>
__device__ __forceinline__ void ph_post_smooth(const RowMat<T>& m, const T* dinv, const T* b, const T* t, T* x,
                                               double w) {
  for_rows<LPR>(m.n, [&](int i, int lane) {
    double bi = 0.0, di = 0.0, ti = 0.0;
    if (i < m.n && lane == 0) {
      bi = ldv<false>(b + i);
      di = double(__ldg(dinv + i));
      ti = ldv<false>(t + i);
    }
    const double s = mat_row<LPR>(m, i, lane, [&](int j) { return ldv<false>(t + j); });
    if (i < m.n && lane == 0) x[i] = T(ti + w * di * (bi - s));
  });
}

// Chebyshev smoothing (Saad, Iterative Methods for Sparse Linear Systems,
// 2nd ed., Algorithm 12.1, applied to Dinv A) over [lambda / ratio, lambda]:
// with theta and delta the interval's centre and half width, sigma = theta /
// delta and rho_0 = 1 / sigma, step k >= 1 takes rho_k = 1 / (2 sigma -
// rho_{k-1}), r_k = r_{k-1} - Dinv A d_{k-1}, d_k = rho_k rho_{k-1} d_{k-1} +
// (2 rho_k / delta) r_k and x += d_k, from r_0 = Dinv (b - A x), d_0 = r_0 /
// theta. The coefficients are formed once per estimate of lambda (formed in
// every row of every step, their divisions were a serial chain of up to 0.6 us
// at the end of each kernel).
__device__ __forceinline__ void cheb_coefficients(double lmax, double ratio, double* coef) {
  const double lmin = lmax / ratio, theta = 0.5 * (lmax + lmin), delta = 0.5 * (lmax - lmin);
  const double sigma = theta / delta;
  double rho = 1.0 / sigma;
  coef[0] = 1.0 / theta;
  for (int j = 1; j < MAX_CHEB; ++j) {
    const double rho1 = 1.0 / (2.0 * sigma - rho);
    coef[2 * j - 1] = rho1 * rho;
    coef[2 * j] = 2.0 * rho1 / delta;
    rho = rho1;
  }
}

// Pre-smoothing from a zero iterate, steps 0 and 1 together: d_0 = Dinv b /
// theta (formed for the neighbours from b), r_1 = Dinv b - Dinv A d_0, d_1 and
// x = d_0 + d_1.
template <int LPR, class T>
__device__ __forceinline__ void ph_cheb_first(const RowMat<T>& m, const T* dinv, const T* b, const double* coef, T* cr,
                                              T* d1, T* x) {
  const double inv_theta = __ldg(coef), c1 = __ldg(coef + 1), c2 = __ldg(coef + 2);
  for_rows<LPR>(m.n, [&](int i, int lane) {
    double bi = 0.0, di = 0.0;
    if (i < m.n && lane == 0) {
      bi = ldv<false>(b + i);
      di = double(__ldg(dinv + i));
    }
    const double s = mat_row<LPR>(m, i, lane, [&](int j) { return double(__ldg(dinv + j)) * ldv<false>(b + j); });
    if (i >= m.n || lane) return;
    const double db = di * bi;
    const double r1 = db - di * s * inv_theta, d0 = db * inv_theta;
    const double dn = c1 * d0 + c2 * r1;
    cr[i] = T(r1);
    d1[i] = T(dn);
    x[i] = T(d0 + dn);
  });
}

// Post-smoothing, step 0 from the iterate t: r_0 = Dinv (b - A t), d_0 = r_0 /
// theta, x = t + d_0.
template <int LPR, class T>
__device__ __forceinline__ void ph_cheb_start(const RowMat<T>& m, const T* dinv, const T* b, const T* t,
                                              const double* coef, T* cr, T* d0, T* x) {
  const double inv_theta = __ldg(coef);
  for_rows<LPR>(m.n, [&](int i, int lane) {
    double bi = 0.0, di = 0.0, ti = 0.0;
    if (i < m.n && lane == 0) {
      bi = ldv<false>(b + i);
      di = double(__ldg(dinv + i));
      ti = ldv<false>(t + i);
    }
    const double s = mat_row<LPR>(m, i, lane, [&](int j) { return ldv<false>(t + j); });
    if (i >= m.n || lane) return;
    const double r0 = di * (bi - s), d = r0 * inv_theta;
    cr[i] = T(r0);
    d0[i] = T(d);
    x[i] = T(ti + d);
  });
}

// Step k >= 1: r -= Dinv A d_in, d_out = c1 d_in + c2 r, x += d_out (each row
// updates only its own r and x; the neighbours are read from d_in)
template <int LPR, class T>
__device__ __forceinline__ void ph_cheb_next(const RowMat<T>& m, const T* dinv, const T* d_in, const double* coef,
                                             int step, T* cr, T* d_out, T* x) {
  const double c1 = __ldg(coef + 2 * step - 1), c2 = __ldg(coef + 2 * step);
  for_rows<LPR>(m.n, [&](int i, int lane) {
    double di = 0.0, dd = 0.0, ri = 0.0, xi = 0.0;
    if (i < m.n && lane == 0) {
      di = double(__ldg(dinv + i));
      dd = ldv<false>(d_in + i);
      ri = double(cr[i]);
      xi = double(x[i]);
    }
    const double s = mat_row<LPR>(m, i, lane, [&](int j) { return ldv<false>(d_in + j); });
    if (i >= m.n || lane) return;
    const double r = ri - di * s;
    const double dn = c1 * dd + c2 * r;
    cr[i] = T(r);
    d_out[i] = T(dn);
    x[i] = T(xi + dn);
  });
}

// restriction by the piecewise-constant prolongation: bc_c = sum of the
// members' residuals, in member order
template <class T>
__device__ __forceinline__ void ph_restrict_pc(int nc, const int* mptr, const int* mlist, const T* r, T* bc) {
  for_rows<1>(nc, [&](int c, int) {
    if (c >= nc) return;
    double s = 0.0;
    for (int m = __ldg(mptr + c); m < __ldg(mptr + c + 1); ++m) s += ldv<false>(r + __ldg(mlist + m));
    bc[c] = T(s);
  });
}

// Fused upward step of the piecewise-constant prolongation: t = xs + alpha P xc
// formed on the fly for each neighbour, then x_i = t_i + w Dinv_i (b_i - sum_j
// a_ij t_j). Reads xs, writes x: out of place, no race between rows.
template <class T>
__device__ __forceinline__ void ph_up(const RowMat<T>& m, const T* dinv, const int* agg, const T* b, const T* xs,
                                      const T* xc, T* x, double w, double alpha) {
  for_rows<1>(m.n, [&](int i, int) {
    auto t = [&](int j) { return ldv<false>(xs + j) + alpha * ldv<false>(xc + __ldg(agg + j)); };
    const double s = mat_row<1>(m, i, 0, t);
    if (i >= m.n) return;
    x[i] = T(t(i) + w * double(__ldg(dinv + i)) * (ldv<false>(b + i) - s));
  });
}

// ---- one kernel per phase
#define OA_PHASE_KERNEL(name, params, args)                                              \
  template <class T, int LPR>                                                            \
  __global__ void __launch_bounds__(AB, 8) k_##name params {                                \
    if (*done) return;                                                                   \
    ph_##name<LPR, T> args;                                                       \
  }
OA_PHASE_KERNEL(smooth_resid, (RowMat<T> m, const T* dinv, const T* b, T* xs, T* r, double w, const int* done),
                (m, dinv, b, xs, r, w))
OA_PHASE_KERNEL(resid, (RowMat<T> m, const T* b, const T* x, T* r, const int* done), (m, b, x, r))
OA_PHASE_KERNEL(restrict, (RowMat<T> m, const T* r, T* bc, const int* done), (m, r, bc))
OA_PHASE_KERNEL(prolong_add, (RowMat<T> m, const T* xc, T* t, double alpha, const int* done), (m, xc, t, alpha))
OA_PHASE_KERNEL(post_smooth, (RowMat<T> m, const T* dinv, const T* b, const T* t, T* x, double w, const int* done),
                (m, dinv, b, t, x, w))
OA_PHASE_KERNEL(cheb_first,
                (RowMat<T> m, const T* dinv, const T* b, const double* coef, T* cr, T* d1, T* x, const int* done),
                (m, dinv, b, coef, cr, d1, x))
OA_PHASE_KERNEL(cheb_start,
                (RowMat<T> m, const T* dinv, const T* b, const T* t, const double* coef, T* cr, T* d0, T* x,
                 const int* done),
                (m, dinv, b, t, coef, cr, d0, x))
OA_PHASE_KERNEL(cheb_next,
                (RowMat<T> m, const T* dinv, const T* d_in, const double* coef, int step, T* cr, T* d_out, T* x,
                 const int* done),
                (m, dinv, d_in, coef, step, cr, d_out, x))
#undef OA_PHASE_KERNEL

template <class T>
__global__ void k_restrict_pc(int nc, const int* mptr, const int* mlist, const T* r, T* bc, const int* done) {
  if (*done) return;
  ph_restrict_pc<T>(nc, mptr, mlist, r, bc);
}

template <class T>
__global__ void __launch_bounds__(AB) k_up(RowMat<T> m, const T* dinv, const int* agg, const T* b, const T* xs,
                                           const T* xc, T* x, double w, double alpha, const int* done) {
  if (*done) return;
  ph_up<T>(m, dinv, agg, b, xs, xc, x, w, alpha);
}

// x = M b with the dense operator of a level (rows ld apart), one warp per row
template <class T>
__global__ void __launch_bounds__(AB) k_dense_apply(int n, const double* __restrict__ M, int ld,
                                                    const T* __restrict__ b, T* __restrict__ x, const int* done) {
  if (*done) return;
  for_rows<32>(n, [&](int i, int lane) {
    double s = 0.0;
    if (i < n) {
      const double* row = M + (size_t)i * ld;
#pragma unroll 4
      for (int j = lane; j < n; j += 32) s += __ldg(row + j) * double(__ldg(b + j));
    }
    s = group_sum<32>(s);
    if (i < n && lane == 0) x[i] = T(s);
  });
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A launch as one cluster of CLUSTER_BLOCKS blocks, more than the portable 8.
struct ClusterLaunch {
  cudaLaunchConfig_t c = {};
  cudaLaunchAttribute at[1];
  explicit ClusterLaunch(cudaStream_t st) {
    c.gridDim = CLUSTER_BLOCKS;
    c.blockDim = CLUSTER_THREADS;
    c.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CLUSTER_BLOCKS;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = 1;
  }
};

// Opts a kernel in on the current device; false where such a cluster cannot be
// placed there (a slice of a GPU).
template <class K>
static bool cluster_fits(K kernel) {
  const ClusterLaunch l(nullptr);
  int n = 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kernel, &l.c) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return n > 0;
}

template <class K, class... A>
static int launch_cluster(K kernel, cudaStream_t st, const A&... args) {
  const ClusterLaunch l(st);
  OA_CUDA(cudaLaunchKernelEx(&l.c, kernel, args...));
  count_launches(1);
  return OA_OK;
}

// ---------------------------------------------------------------------------
// numeric phase

// Smoothed prolongation: P_iJ = [J == agg(i)] - wp Dinv_i sum of the row's A
// entries whose column lies in aggregate J; LPR lanes share a row's entries.
template <class T, int LPR>
__global__ void __launch_bounds__(AB) k_sa_prolongator(int n, const int* __restrict__ p_rp,
                                                       const int* __restrict__ p_diag, const int* __restrict__ pg_ptr,
                                                       const int* __restrict__ pg_list, const T* __restrict__ A,
                                                       const T* __restrict__ dinv, double wp, T* __restrict__ pv) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = g / LPR, lane = g % LPR;
  if (i >= n) return;
  const double di = double(dinv[i]);
  const int e0 = p_rp[i];
  for (int e = e0 + lane; e < p_rp[i + 1]; e += LPR) {
    double s = 0.0;
    for (int q = pg_ptr[e]; q < pg_ptr[e + 1]; ++q) s += double(A[pg_list[q]]);
    pv[e] = T((e - e0 == p_diag[i] ? 1.0 : 0.0) - wp * di * s);
  }
}

// out_e = sum over the entry's term list of a[ia] * b[ib], LPR lanes per entry.
template <class T, int LPR>
__global__ void __launch_bounds__(AB) k_pair_sum(int n_out, const int* __restrict__ ptr, const int* __restrict__ ia,
                                                 const int* __restrict__ ib, const T* __restrict__ a,
                                                 const T* __restrict__ b, T* __restrict__ out) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const int e = g / LPR, lane = g % LPR;
  double s = 0.0;
  if (e < n_out)
    for (int q = ptr[e] + lane; q < ptr[e + 1]; q += LPR) s += double(a[ia[q]]) * double(b[ib[q]]);
  s = group_sum<LPR>(s);
  if (e < n_out && lane == 0) out[e] = T(s);
}

// P^T values in coarse-row order (contiguous for the restriction)
template <class T>
__global__ void k_gather(int n, const int* __restrict__ idx, const T* __restrict__ src, T* __restrict__ dst) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) dst[q] = src[idx[q]];
}

// Spectral radius of Dinv A by power iteration from a fixed pseudo-random
// vector: POWER_STEPS products w = Dinv A (v / |v|) in FP64, each followed by
// an ordered reduction of |w|^2; the last |w|, times a safety factor of 1.1,
// bounds the smoothing interval.
constexpr int POWER_STEPS = 15;
// One cluster pays off while a sweep of the matrix by its 16 SMs (about 0.45 us
// per MB from L2) costs no more than a kernel of its own per product.
constexpr size_t POWER_CLUSTER_BYTES = 4u << 20;

__device__ __forceinline__ double power_start(int i) {
  unsigned h = (unsigned)i * 2654435761u;
  h ^= h >> 15;
  h *= 2246822519u;
  h ^= h >> 13;
  return double(h) * (2.0 / 4294967296.0) - 1.0;
}

__global__ void k_power_init(int n, double* v, double* est) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] = power_start(i);
  if (i == 0) est[0] = 1.0;
}

// sum over a block of at most 1024 threads, in a fixed order; every thread of
// warp 0 gets it
__device__ __forceinline__ double block_sum(double v, double* sh) {
  v = group_sum<32>(v);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x < 32) s = group_sum<32>(threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0);
  return s;
}

template <bool SHARED, int LPR, class T>
__device__ __forceinline__ double ph_power(const RowMat<T>& m, const T* dinv, const double* v, double inv, double* w) {
  double q = 0.0;
  for_rows<LPR>(m.n, [&](int i, int lane) {
    const double s = mat_row<LPR>(m, i, lane, [&](int j) { return ldv<SHARED>(v + j); });
    if (i >= m.n || lane) return;
    const double wi = double(__ldg(dinv + i)) * s * inv;
    w[i] = wi;
    q += wi * wi;
  });
  return q;
}

// One product over a large level; the last block to finish sums the
// block partials in order and closes the step.
template <class T, int LPR>
__global__ void __launch_bounds__(AB) k_power_step(RowMat<T> m, const T* dinv, const double* v, double* est, double* w,
                                                   double* partials, unsigned* ticket, double ratio, double* coef) {
  __shared__ double sh[32];
  __shared__ bool mine;
  const double q = ph_power<false, LPR, T>(m, dinv, v, est[0], w);
  const double s = block_sum(q, sh);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = s;
    __threadfence();
    mine = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!mine) return;
  double p = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += AB) p += __ldcg(partials + b);
  __syncthreads();
  p = block_sum(p, sh);
  if (threadIdx.x == 0) {
    const double nrm = sqrt(p);
    est[0] = nrm > 0.0 ? 1.0 / nrm : 1.0;
    est[1] = 1.1 * nrm;
    cheb_coefficients(est[1], ratio, coef);
  }
}

// The whole estimate of a small level in one kernel of one cluster: the 15
// products are a serial chain of small sweeps.
template <class T>
__global__ void __launch_bounds__(CLUSTER_THREADS, 1)
    k_power_cluster(RowMat<T> m, int nnz, const T* dinv, double* est, double* v, double* w, double* partials, double ratio,
                 double* coef) {
  __shared__ double sh[32];
  __shared__ double nrm_sh;
  const unsigned stride = gridDim.x * blockDim.x;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < (unsigned)m.n; i += stride) v[i] = power_start((int)i);
  cluster_barrier();
  const int lpr = cluster_lanes(m.n, nnz);
  double inv = 1.0, nrm = 0.0;
  for (int it = 0; it < POWER_STEPS; ++it) {
    const double* vin = (it & 1) ? w : v;
    double* wout = (it & 1) ? v : w;
    double q;
    switch (lpr) {
      case 1: q = ph_power<true, 1, T>(m, dinv, vin, inv, wout); break;
      case 4: q = ph_power<true, 4, T>(m, dinv, vin, inv, wout); break;
      default: q = ph_power<true, 16, T>(m, dinv, vin, inv, wout);
    }
    const double s = block_sum(q, sh);
    // two sets of partials in turn: a block may still be reading the last step's
    if (threadIdx.x == 0) partials[(it & 1) * CLUSTER_BLOCKS + blockIdx.x] = s;
    cluster_barrier();
    if (threadIdx.x < 32) {
      const double p = threadIdx.x < gridDim.x ? partials[(it & 1) * CLUSTER_BLOCKS + threadIdx.x] : 0.0;
      const double t = sqrt(group_sum<32>(p));
      if (threadIdx.x == 0) nrm_sh = t;
    }
    __syncthreads();
    nrm = nrm_sh;
    inv = nrm > 0.0 ? 1.0 / nrm : 1.0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    est[0] = inv;
    est[1] = 1.1 * nrm;
    cheb_coefficients(est[1], ratio, coef);
  }
}

// a kernel over rows, by the lanes of a row
#define OA_LPR_LAUNCH(lpr, kernel, T, rows, st, ...)                                         \
  do {                                                                                        \
    if ((lpr) == 1)                                                                           \
      kernel<T, 1><<<grid_for(rows, 1), AB, 0, st>>>(__VA_ARGS__);                            \
    else if ((lpr) == 4)                                                                      \
      kernel<T, 4><<<grid_for(rows, 4), AB, 0, st>>>(__VA_ARGS__);                            \
    else if ((lpr) == 8)                                                                      \
      kernel<T, 8><<<grid_for(rows, 8), AB, 0, st>>>(__VA_ARGS__);                            \
    else                                                                                      \
      kernel<T, 32><<<grid_for(rows, 32), AB, 0, st>>>(__VA_ARGS__);                          \
    count_launches(1);                                                                        \
  } while (0)

// the same for kernels over the finest level's matrix, which may be in
// fixed-width storage
#define OA_MAT_LAUNCH(format, kernel, T, rows, st, ...)                                      \
  do {                                                                                        \
    const int f_ = (format);                                                                  \
    if (f_ < ELL) {                                                                           \
      OA_LPR_LAUNCH(f_, kernel, T, rows, st, __VA_ARGS__);                                    \
    } else {                                                                                  \
      if (f_ == ELL + 7)                                                                      \
        kernel<T, ELL + 7><<<grid_for(rows, 1), AB, 0, st>>>(__VA_ARGS__);                    \
      else if (f_ == ELL + 15)                                                                \
        kernel<T, ELL + 15><<<grid_for(rows, 1), AB, 0, st>>>(__VA_ARGS__);                   \
      else if (f_ == ELL_STREAM + 7)                                                          \
        kernel<T, ELL_STREAM + 7><<<grid_for(rows, 1), AB, 0, st>>>(__VA_ARGS__);             \
      else                                                                                    \
        kernel<T, ELL_STREAM + 15><<<grid_for(rows, 1), AB, 0, st>>>(__VA_ARGS__);            \
      count_launches(1);                                                                      \
    }                                                                                         \
  } while (0)

// ---------------------------------------------------------------------------
template <class T>
static RowMat<T> level_matrix(const AmgLevel<T>& v) {
  return {v.n, v.rp, v.cols, v.A, ell_mat(v.ell, v.ell_val)};
}
template <class T>
static int level_format(const AmgLevel<T>& v) {
  return v.ell_val ? ell_format(v.ell.w, v.ell.slots, sizeof(T)) : v.lpr_a;
}

template <class T>
int Amg<T>::setup(int n, const int* h_rp, const int* h_cols, const int* h_diag, int* d_rp, int* d_cols, int* d_diag) {
  release();
  // tuning knobs: prolongation type, Jacobi damping, coarse-correction scaling
  if (const char* e = std::getenv("OA_AMG_SMOOTHED")) smoothed = std::atoi(e) != 0;
  omega = smoothed ? 0.8 : 0.7;
  alpha = smoothed ? 1.0 : 1.8;
  if (const char* e = std::getenv("OA_AMG_OMEGA")) omega = std::atof(e);
  if (const char* e = std::getenv("OA_AMG_ALPHA")) alpha = std::atof(e);
  if (const char* e = std::getenv("OA_AMG_OMEGA_P")) omega_p = std::atof(e);
  if (const char* e = std::getenv("OA_AMG_CHEB_DEGREE")) cheb_degree = std::atoi(e);
  if (const char* e = std::getenv("OA_AMG_CHEB_ROWS")) cheb_rows = std::atoi(e);
  if (const char* e = std::getenv("OA_AMG_CHEB_RATIO")) cheb_ratio = std::max(1.5, std::atof(e));
  if (cheb_degree < 2 || !smoothed) cheb_degree = 0;
  if (cheb_degree > MAX_CHEB) return fail(OA_ERR_ARG, "AMG: Chebyshev degree above the supported maximum");
  std::vector<int> rp(h_rp, h_rp + n + 1), cols(h_cols, h_cols + h_rp[n]), dg(h_diag, h_diag + n);
  int cur = n;
  for (int lev = 0;; ++lev) {
    // the level joins L before anything is allocated for it, so an error
    // return leaves every allocation where release() finds it
    L.emplace_back();
    AmgLevel<T>& lv = L.back();
    lv.n = cur;
    lv.nnz = rp[cur];
    if (lev == 0) {
      lv.rp = d_rp;
      lv.cols = d_cols;
      lv.diag = d_diag;
    } else {
      int s;
      if ((s = upload(&lv.rp, rp)) || (s = upload(&lv.cols, cols)) || (s = upload(&lv.diag, dg))) return s;
      if ((s = dalloc(&lv.A, (size_t)lv.nnz))) return s;
      lv.own_A = true;
    }
    int s;
    if ((s = dalloc(&lv.dinv, cur)) || (s = dalloc(&lv.r, cur)) || (s = dalloc(&lv.t, cur))) return s;
    if (lev > 0 && ((s = dalloc(&lv.x, cur)) || (s = dalloc(&lv.b, cur)))) return s;
    lv.lpr_a = lanes_for(double(lv.nnz) / std::max(1, cur), cur);
    const bool last = cur <= COARSE_MAX || lev >= 14;
    if (last) break;
    // not on the finest level: its matrix is always the caller's current one,
    // while the spectral estimate (like Dinv) is refreshed only with the
    // hierarchy; a coarse level's matrix, Dinv and estimate come from the same
    // numeric phase
    if (cheb_degree >= 2 && lev > 0 && cur <= cheb_rows) {
      lv.cheb = true;
      if ((s = dalloc(&lv.cr, cur)) || (s = dalloc(&lv.cd0, cur)) || (s = dalloc(&lv.cd1, cur)) ||
          (s = dalloc(&lv.est, 2)) || (s = dalloc(&lv.coef, 1 + 2 * MAX_CHEB)) || (s = dalloc(&lv.pw_v, cur)) ||
          (s = dalloc(&lv.pw_w, cur)) || (s = dalloc(&lv.pw_part, std::max<size_t>(2 * CLUSTER_BLOCKS, grid_for(cur, lv.lpr_a)))) ||
          (s = dalloc(&lv.pw_ticket, 1)))
        return s;
      if (cudaMemset(lv.pw_ticket, 0, sizeof(unsigned)) != cudaSuccess)
        return fail(OA_ERR_CUDA, "AMG: memset failed");
    }
    int nc = 0;
    std::vector<int> crp, ccols, cdg;
    if (smoothed) {
      sa::Level H;
      if (!sa::build(cur, rp, cols, H))
        return fail(OA_ERR_SOLVER, "AMG: smoothed-aggregation term lists exceed 32-bit offsets");
      nc = H.nc;
      if (nc >= cur) return fail(OA_ERR_SOLVER, "AMG: aggregation made no progress");
      lv.nnz_t = H.trp[cur];
      lv.nnz_p = H.prp[cur];
      lv.lpr_p = lanes_for(double(lv.nnz_p) / cur, cur);
      lv.lpr_pt = lanes_for(double(lv.nnz_p) / H.nc, H.nc);
      lv.lpr_t = lanes_for(double(H.tta.size()) / std::max(1, lv.nnz_t), lv.nnz_t);
      lv.lpr_c = lanes_for(double(H.ctp.size()) / std::max(1, H.crp[H.nc]), H.crp[H.nc]);
      if ((s = upload(&lv.p_rp, H.prp)) || (s = upload(&lv.p_cols, H.pcols)) || (s = upload(&lv.p_diag, H.pdiag)) ||
          (s = upload(&lv.pg_ptr, H.pgptr)) || (s = upload(&lv.pg_list, H.pglist)) ||
          (s = upload(&lv.pt_rp, H.ptrp)) || (s = upload(&lv.pt_rows, H.ptrows)) || (s = upload(&lv.pt_src, H.ptsrc)) ||
          (s = upload(&lv.tt_ptr, H.ttptr)) || (s = upload(&lv.tt_a, H.tta)) || (s = upload(&lv.tt_p, H.ttp)) ||
          (s = upload(&lv.ct_ptr, H.ctptr)) || (s = upload(&lv.ct_p, H.ctp)) || (s = upload(&lv.ct_t, H.ctt)) ||
          (s = dalloc(&lv.pv, H.pcols.size())) || (s = dalloc(&lv.ptv, H.pcols.size())) ||
          (s = dalloc(&lv.tv, (size_t)lv.nnz_t)))
        return s;
      crp.swap(H.crp);
      ccols.swap(H.ccols);
      cdg.swap(H.cdg);
    } else {
      std::vector<int> agg;
      nc = sa::aggregate(cur, rp, cols, agg);
      if (nc >= cur) return fail(OA_ERR_SOLVER, "AMG: aggregation made no progress");
      // members of each aggregate, in row order
      std::vector<int> mptr(nc + 1, 0), mlist(cur);
      for (int i = 0; i < cur; ++i) mptr[agg[i] + 1]++;
      for (int c = 0; c < nc; ++c) mptr[c + 1] += mptr[c];
      {
        std::vector<int> pos(mptr.begin(), mptr.end() - 1);
        for (int i = 0; i < cur; ++i) mlist[pos[agg[i]]++] = i;
      }
      // coarse graph (sorted columns) and the gather list of each coarse entry
      crp.assign(nc + 1, 0);
      cdg.assign(nc, 0);
      std::vector<int> tmp;
      for (int c = 0; c < nc; ++c) {
        tmp.clear();
        for (int m = mptr[c]; m < mptr[c + 1]; ++m) {
          const int i = mlist[m];
          for (int k = rp[i]; k < rp[i + 1]; ++k) tmp.push_back(agg[cols[k]]);
        }
        std::sort(tmp.begin(), tmp.end());
        tmp.erase(std::unique(tmp.begin(), tmp.end()), tmp.end());
        for (size_t q = 0; q < tmp.size(); ++q)
          if (tmp[q] == c) cdg[c] = (int)q;
        ccols.insert(ccols.end(), tmp.begin(), tmp.end());
        crp[c + 1] = (int)ccols.size();
      }
      const int cnnz = crp[nc];
      std::vector<int> gcnt(cnnz + 1, 0), target(rp[cur]);
      for (int c = 0; c < nc; ++c)
        for (int m = mptr[c]; m < mptr[c + 1]; ++m) {
          const int i = mlist[m];
          for (int k = rp[i]; k < rp[i + 1]; ++k) {
            const int cj = agg[cols[k]];
            const int pos =
                (int)(std::lower_bound(ccols.begin() + crp[c], ccols.begin() + crp[c + 1], cj) - ccols.begin());
            target[k] = pos;
            gcnt[pos + 1]++;
          }
        }
      for (int q = 0; q < cnnz; ++q) gcnt[q + 1] += gcnt[q];
      std::vector<int> glist(rp[cur]);
      {
        std::vector<int> pos(gcnt.begin(), gcnt.end() - 1);
        for (int c = 0; c < nc; ++c)
          for (int m = mptr[c]; m < mptr[c + 1]; ++m) {
            const int i = mlist[m];
            for (int k = rp[i]; k < rp[i + 1]; ++k) glist[pos[target[k]]++] = k;
          }
      }
      if ((s = upload(&lv.agg, agg)) || (s = upload(&lv.mptr, mptr)) || (s = upload(&lv.mlist, mlist)) ||
          (s = upload(&lv.gptr, gcnt)) || (s = upload(&lv.glist, glist)))
        return s;
    }
    rp.swap(crp);
    cols.swap(ccols);
    dg.swap(cdg);
    cur = nc;
  }
  coarse_n = L.back().n;
  if (cudaMalloc(&dense_inv, sizeof(double) * 2 * (size_t)coarse_n * coarse_n) != cudaSuccess)
    return fail(OA_ERR_CUDA, "AMG: dense coarse allocation failed");
  power_cluster = cluster_fits(k_power_cluster<T>);
  // the dense operator's level and the workspace its columns are formed in
  tail = (int)L.size() - 1;
  // (the finest matrix is always the current one, and an FP32 cycle rounds its
  // vectors after every phase, which the operator would not)
  while (smoothed && sizeof(T) == 8 && tail > 1 && L[tail - 1].n <= DENSE_ROWS) --tail;
  const int last = (int)L.size() - 1;
  if (tail < last) {
    const size_t nt = L[tail].n;
    size_t rows = 0;
    for (size_t l = tail; l < L.size(); ++l) rows += L[l].n;
    // operator, then workspace; without room for them the cycle runs through these levels
    dense_op = static_cast<double*>(
        spare_alloc(sizeof(double) * (nt * nt + 6 * rows * std::min<size_t>(nt, DENSE_COLS)), n));
    if (dense_op) dense_work = dense_op + nt * nt;
    else tail = last;
  }
  ready = true;
  return OA_OK;
}

template <class T>
int Amg<T>::numeric(const T* A_fine, cudaStream_t st) {
  if (!ready) return fail(OA_ERR_NOT_READY, "AMG: numeric before setup");
  L[0].A = const_cast<T*>(A_fine);
  for (size_t l = 0; l < L.size(); ++l) {
    AmgLevel<T>& v = L[l];
    k_dinv<T><<<(v.n + AB - 1) / AB, AB, 0, st>>>(v.n, v.rp, v.diag, v.A, v.dinv);
    count_launches(1);
    if (v.cheb && power_cluster && (size_t)v.nnz * (sizeof(T) + sizeof(int)) <= POWER_CLUSTER_BYTES) {
      if (int s = launch_cluster(k_power_cluster<T>, st, level_matrix(v), v.nnz, (const T*)v.dinv, v.est, v.pw_v, v.pw_w,
                                 v.pw_part, cheb_ratio, v.coef))
        return s;
    } else if (v.cheb) {
      k_power_init<<<(v.n + AB - 1) / AB, AB, 0, st>>>(v.n, v.pw_v, v.est);
      count_launches(1);
      for (int it = 0; it < POWER_STEPS; ++it) {
        const double* vin = (it & 1) ? v.pw_w : v.pw_v;
        double* wout = (it & 1) ? v.pw_v : v.pw_w;
        OA_LPR_LAUNCH(v.lpr_a, k_power_step, T, v.n, st, level_matrix(v), v.dinv, vin, v.est, wout, v.pw_part,
                      v.pw_ticket, cheb_ratio, v.coef);
      }
    }
    if (l + 1 < L.size()) {
      AmgLevel<T>& c = L[l + 1];
      if (smoothed) {
        OA_LPR_LAUNCH(v.lpr_p, k_sa_prolongator, T, v.n, st, v.n, v.p_rp, v.p_diag, v.pg_ptr, v.pg_list, v.A,
                      v.dinv, omega_p, v.pv);
        k_gather<T><<<(v.nnz_p + AB - 1) / AB, AB, 0, st>>>(v.nnz_p, v.pt_src, v.pv, v.ptv);
        count_launches(1);
        OA_LPR_LAUNCH(v.lpr_t, k_pair_sum, T, v.nnz_t, st, v.nnz_t, v.tt_ptr, v.tt_a, v.tt_p, v.A, v.pv, v.tv);
        OA_LPR_LAUNCH(v.lpr_c, k_pair_sum, T, c.nnz, st, c.nnz, v.ct_ptr, v.ct_p, v.ct_t, v.pv, v.tv, c.A);
      } else {
        k_galerkin<T><<<(c.nnz + AB - 1) / AB, AB, 0, st>>>(c.nnz, v.gptr, v.glist, v.A, c.A);
        count_launches(1);
      }
    }
  }
  const AmgLevel<T>& cl = L.back();
  k_dense_fill<T><<<cl.n, 128, 0, st>>>(cl.n, cl.rp, cl.cols, cl.A, dense_inv);
  if (cl.n <= 128) {
    k_invert<1><<<1, 1024, 0, st>>>(cl.n, dense_inv);
  } else if (cl.n <= 256) {
    cudaLaunchConfig_t c = {};
    c.gridDim = 4;
    c.blockDim = 1024;
    c.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 4;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = 1;
    OA_CUDA(cudaLaunchKernelEx(&c, k_invert<4>, cl.n, dense_inv));
  } else {
    k_gauss_jordan<<<1, 1024, 0, st>>>(cl.n, dense_inv);
  }
  count_launches(2);
  OA_CUDA(cudaGetLastError());
  return dense_operator(st);
}

// ---------------------------------------------------------------------------
// The V-cycle from a small level down as one dense operator.
//
// From a zero iterate the cycle is linear in its right-hand side, and its
// matrices only change with the numeric phase. At 1,000 rows its eight
// or more phases are nothing but latency (launch, flag, row pointer -> column ->
// vector; 2.7 to 3.3 us each in the iteration graph), so the numeric phase forms
// the n x n operator and a cycle applies it in one kernel whose loads do not
// depend on one another. The columns come from the same
// phases applied to blocks of unit vectors, in FP64 throughout, and stay FP64.
// Between two numeric phases there are up to 8 to 16 solves of 12 to 25 cycles,
// but a run that starts refreshes on its first few. At 830 rows (a 128 x 48 x 48
// channel) the operator costs 0.4 ms and saves about 30 us a cycle; at 1,400
// rows it took 0.65 ms, as much as the 20 cycles of one solve save. FP64 cycles
// only: the FP32 one rounds every phase's vectors, and a cycle without those
// roundings leaves the pressure of a solve stopped at 1e-8 up to 1e-4 away on
// stretched channels (both within the solve's tolerance). (Also tried: the
// cycle of these levels in one cluster of 16 blocks, with the matrices in L2 or
// resident in shared memory and the vectors exchanged through distributed
// shared memory. A phase then takes 3,000 to 7,000 cycles: no gain.)
enum ColumnOp { CO_JACOBI, CO_CHEB_FIRST, CO_CHEB_NEXT, CO_RESID, CO_SUM, CO_PROLONG, CO_POST, CO_CHEB_START };

struct ColumnArgs {
  int op, C, step;
  double w;           // Jacobi or coarse-correction weight
  const double* X;    // gathered columns [.][C]
  const double* b;    // right-hand side columns
  double *x, *r, *o;  // iterate, Chebyshev residual, output columns
  const double* coef;
};

// s = sum_k A_ik g(X_k.) for every column, then the phase's row update; threads
// along the columns, one row per block row. (32 columns of 8 to 32 consecutive
// rows per block, for more reuse in L1, took 33 instead of 27 us at 1,400 rows.)

template <class T>
__global__ void __launch_bounds__(128) k_columns(RowMat<T> m, const T* __restrict__ dinv, ColumnArgs a) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (c >= a.C) return;
  const bool from_b = a.op == CO_JACOBI || a.op == CO_CHEB_FIRST;
  double s = 0.0;
  const int e = __ldg(m.rp + i + 1);
#pragma unroll 8
  for (int k = __ldg(m.rp + i); k < e; ++k) {
    const int j = __ldg(m.cols + k);
    const double xj = a.X[(size_t)j * a.C + c];
    s += double(__ldg(m.A + k)) * (from_b ? double(__ldg(dinv + j)) * xj : xj);
  }
  const size_t t = (size_t)i * a.C + c;
  const double di = dinv ? double(__ldg(dinv + i)) : 0.0;
  switch (a.op) {
    case CO_JACOBI:
      a.x[t] = a.w * di * a.b[t];
      a.o[t] = a.b[t] - a.w * s;
      break;
    case CO_CHEB_FIRST: {
      const double db = di * a.b[t], r1 = db - di * s * a.coef[0], d0 = db * a.coef[0];
      const double dn = a.coef[1] * d0 + a.coef[2] * r1;
      a.r[t] = r1;
      a.o[t] = dn;
      a.x[t] = d0 + dn;
      break;
    }
    case CO_CHEB_NEXT: {
      const double r = a.r[t] - di * s;
      const double dn = a.coef[2 * a.step - 1] * a.X[t] + a.coef[2 * a.step] * r;
      a.r[t] = r;
      a.o[t] = dn;
      a.x[t] += dn;
      break;
    }
    case CO_RESID: a.o[t] = a.b[t] - s; break;
    case CO_SUM: a.o[t] = s; break;
    case CO_PROLONG: a.x[t] += a.w * s; break;
    case CO_POST: a.o[t] = a.x[t] + a.w * di * (a.b[t] - s); break;
    case CO_CHEB_START: {
      const double r0 = di * (a.b[t] - s), d = r0 * a.coef[0];
      a.r[t] = r0;
      a.o[t] = d;
      a.x[t] += d;
    }
  }
}

// columns c0 .. c0 + C of the identity
__global__ void k_unit_columns(int n, int C, int c0, double* b) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n * C) b[t] = t / C == c0 + t % C ? 1.0 : 0.0;
}

// columns of the coarsest level's solution from its inverse (M: [A | A^-1])
__global__ void __launch_bounds__(128) k_inverse_columns(int n, int C, const double* __restrict__ M,
                                                         const double* __restrict__ b, double* __restrict__ x) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (c >= C) return;
  double s = 0.0;
#pragma unroll 4
  for (int j = 0; j < n; ++j) s += __ldg(M + (size_t)i * 2 * n + n + j) * b[(size_t)j * C + c];
  x[(size_t)i * C + c] = s;
}

// columns c0 .. c0 + C into the row-major operator
__global__ void k_store_columns(int n, int C, int c0, const double* __restrict__ x, double* __restrict__ M) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n * C) M[(size_t)(t / C) * n + c0 + t % C] = x[t];
}

template <class T>
int Amg<T>::dense_operator(cudaStream_t st) {
  const int nl = (int)L.size(), n = L[tail].n;
  if (tail == nl - 1) return OA_OK;  // the coarsest level's inverse itself
  const int cols = std::min(n, DENSE_COLS);
  struct Cols {
    double *b, *x, *r, *d0, *d1, *t;
  };
  std::vector<Cols> W(nl);
  double* at = dense_work;
  for (int l = tail; l < nl; ++l) {
    const size_t k = (size_t)L[l].n * cols;
    W[l] = {at, at + k, at + 2 * k, at + 3 * k, at + 4 * k, at + 5 * k};
    at += 6 * k;
  }
  for (int c0 = 0; c0 < n; c0 += cols) {
    const int C = std::min(cols, n - c0);
    auto phase = [&](const RowMat<T>& m, const T* dinv, ColumnArgs a) {
      a.C = C;
      k_columns<T><<<dim3((C + 127) / 128, m.n), 128, 0, st>>>(m, dinv, a);
      count_launches(1);
    };
    k_unit_columns<<<(n * C + AB - 1) / AB, AB, 0, st>>>(n, C, c0, W[tail].b);
    for (int l = tail; l < nl - 1; ++l) {
      const AmgLevel<T>& v = L[l];
      const Cols& w = W[l];
      const RowMat<T> A = level_matrix(v);
      if (v.cheb) {
        phase(A, v.dinv, {CO_CHEB_FIRST, 0, 0, 0.0, w.b, w.b, w.x, w.r, w.d1, v.coef});
        for (int k = 2; k < cheb_degree; ++k)
          phase(A, v.dinv, {CO_CHEB_NEXT, 0, k, 0.0, (k & 1) ? w.d0 : w.d1, w.b, w.x, w.r, (k & 1) ? w.d1 : w.d0, v.coef});
        phase(A, v.dinv, {CO_RESID, 0, 0, 0.0, w.x, w.b, nullptr, nullptr, w.t, nullptr});
      } else {
        phase(A, v.dinv, {CO_JACOBI, 0, 0, omega, w.b, w.b, w.x, nullptr, w.t, nullptr});
      }
      const RowMat<T> pt = {L[l + 1].n, v.pt_rp, v.pt_rows, v.ptv, nullptr, nullptr};
      phase(pt, nullptr, {CO_SUM, 0, 0, 0.0, w.t, nullptr, nullptr, nullptr, W[l + 1].b, nullptr});
    }
    const AmgLevel<T>& cl = L.back();
    k_inverse_columns<<<dim3((C + 127) / 128, cl.n), 128, 0, st>>>(cl.n, C, dense_inv, W.back().b, W.back().x);
    const double* xc = W.back().x;
    for (int l = nl - 2; l >= tail; --l) {
      const AmgLevel<T>& v = L[l];
      const Cols& w = W[l];
      const RowMat<T> A = level_matrix(v), p = {v.n, v.p_rp, v.p_cols, v.pv, nullptr, nullptr};
      phase(p, nullptr, {CO_PROLONG, 0, 0, alpha, xc, nullptr, w.x, nullptr, nullptr, nullptr});
      if (v.cheb) {
        // the iterate is gathered and updated in the same phase: from a copy
        OA_CUDA(cudaMemcpyAsync(w.t, w.x, sizeof(double) * v.n * C, cudaMemcpyDeviceToDevice, st));
        phase(A, v.dinv, {CO_CHEB_START, 0, 0, 0.0, w.t, w.b, w.x, w.r, w.d0, v.coef});
        for (int k = 1; k < cheb_degree; ++k)
          phase(A, v.dinv, {CO_CHEB_NEXT, 0, k, 0.0, (k & 1) ? w.d0 : w.d1, w.b, w.x, w.r, (k & 1) ? w.d1 : w.d0, v.coef});
        xc = w.x;
      } else {
        phase(A, v.dinv, {CO_POST, 0, 0, omega, w.x, w.b, w.x, nullptr, w.t, nullptr});
        xc = w.t;
      }
    }
    k_store_columns<<<(n * C + AB - 1) / AB, AB, 0, st>>>(n, C, c0, xc, dense_op);
    count_launches(3);
  }
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}

template <class T>
int Amg<T>::apply(const T* v, T* z, const int* done, cudaStream_t st) {
  const int nl = (int)L.size();
  // downward pass above the dense operator: smooth + residual (row parallel), restriction
  for (int l = 0; l < tail; ++l) {
    AmgLevel<T>& lv = L[l];
    AmgLevel<T>& c = L[l + 1];
    const T* b = l == 0 ? v : lv.b;
    const RowMat<T> m = level_matrix(lv);
    if (lv.cheb) {
      OA_LPR_LAUNCH(lv.lpr_a, k_cheb_first, T, lv.n, st, m, lv.dinv, b, lv.coef, lv.cr, lv.cd1, lv.t, done);
      for (int k = 2; k < cheb_degree; ++k) {
        const T* din = (k & 1) ? lv.cd0 : lv.cd1;
        T* dout = (k & 1) ? lv.cd1 : lv.cd0;
        OA_LPR_LAUNCH(lv.lpr_a, k_cheb_next, T, lv.n, st, m, lv.dinv, din, lv.coef, k, lv.cr, dout, lv.t, done);
      }
      OA_LPR_LAUNCH(lv.lpr_a, k_resid, T, lv.n, st, m, b, lv.t, lv.r, done);
    } else {
      OA_MAT_LAUNCH(level_format(lv), k_smooth_resid, T, lv.n, st, m, lv.dinv, b, lv.t, lv.r, omega, done);
    }
    if (smoothed) {
      const RowMat<T> pt = {c.n, lv.pt_rp, lv.pt_rows, lv.ptv, nullptr, nullptr};
      OA_LPR_LAUNCH(lv.lpr_pt, k_restrict, T, c.n, st, pt, lv.r, c.b, done);
    } else {
      k_restrict_pc<T><<<(c.n + AB - 1) / AB, AB, 0, st>>>(c.n, lv.mptr, lv.mlist, lv.r, c.b, done);
      count_launches(1);
    }
  }
  {
    AmgLevel<T>& lv = L[tail];
    const double* M = dense_op ? dense_op : dense_inv + lv.n;
    k_dense_apply<T><<<grid_for(lv.n, 32), AB, 0, st>>>(lv.n, M, dense_op ? lv.n : 2 * lv.n, tail == 0 ? v : lv.b,
                                                        tail == 0 ? z : lv.x, done);
    count_launches(1);
  }
  // upward pass above the dense operator: prolongation + post-smooth (one fused kernel
  // for the piecewise-constant prolongation, two for the smoothed one)
  for (int l = tail - 1; l >= 0; --l) {
    AmgLevel<T>& lv = L[l];
    const T* b = l == 0 ? v : lv.b;
    T* x = l == 0 ? z : lv.x;
    const T* xc = L[l + 1].x;
    const RowMat<T> m = level_matrix(lv);
    if (!smoothed) {
      k_up<T><<<(lv.n + AB - 1) / AB, AB, 0, st>>>(m, lv.dinv, lv.agg, b, lv.t, xc, x, omega, alpha, done);
      count_launches(1);
      continue;
    }
    const RowMat<T> p = {lv.n, lv.p_rp, lv.p_cols, lv.pv, nullptr, nullptr};
    OA_LPR_LAUNCH(lv.lpr_p, k_prolong_add, T, lv.n, st, p, xc, lv.t, alpha, done);
    if (lv.cheb) {
      OA_LPR_LAUNCH(lv.lpr_a, k_cheb_start, T, lv.n, st, m, lv.dinv, b, lv.t, lv.coef, lv.cr, lv.cd0, x, done);
      for (int k = 1; k < cheb_degree; ++k) {
        const T* din = (k & 1) ? lv.cd0 : lv.cd1;
        T* dout = (k & 1) ? lv.cd1 : lv.cd0;
        OA_LPR_LAUNCH(lv.lpr_a, k_cheb_next, T, lv.n, st, m, lv.dinv, din, lv.coef, k, lv.cr, dout, x, done);
      }
    } else {
      OA_MAT_LAUNCH(level_format(lv), k_post_smooth, T, lv.n, st, m, lv.dinv, b, lv.t, x, omega, done);
    }
  }
  OA_CUDA(cudaGetLastError());
  return OA_OK;
}

template <class T>
int Amg<T>::set_smoothing(int degree, double prolongation_damping) {
  if (degree < 2 || degree > MAX_CHEB || !(prolongation_damping > 0.0 && prolongation_damping < 1.5))
    return fail(OA_ERR_ARG, "AMG: Chebyshev degree 2..6 and prolongation damping in (0, 1.5)");
  omega_p = prolongation_damping;
  if (!smoothed) return OA_OK;
  if (dense_op && degree != cheb_degree) operator_stale = true;
  cheb_degree = degree;
  return OA_OK;
}

template struct Amg<double>;
template struct Amg<float>;

}  // namespace oa
