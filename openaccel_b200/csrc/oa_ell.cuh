// Fixed-width row storage of a scalar CSR matrix (internal).
//
// Rows come in groups of 32; entry q of row i sits at 32 (W (i / 32) + q) + i % 32.
// A warp whose lanes take one row each then reads every slot as one contiguous
// line of values and one of columns (in CSR the same loads are strided by the
// row length), needs no row pointer in its chain of dependent loads, and has
// all W slots in flight at once. W is a compile-time constant, for the two row
// lengths of the stencils this library assembles: 7 (a node of a hex block and
// its edge neighbours) and 15 (a node of a block split into Kuhn tets). Other
// graphs keep CSR, and so does one that the padding would more than double.
// Measured product, matrix in DRAM: 97^3 rows FP64 14.8 us (CSR 22.8), 129^3 rows
// FP32 20.7 us (CSR 32.8), that is 6.2 and 6.6 TB/s; a run-time width lost most
// of it (20.7 and 28.9 us). Entries past a row's end have value 0 and the row's
// first column (0 in an empty row).
#pragma once
#include <cuda_runtime.h>

namespace oa {

// Formats of a row product: lanes per row of a CSR matrix (1, 4, 8, 32), or ELL +
// width, or, for a matrix that does not fit L2 beside the vectors, ELL_STREAM +
// width (loads that do not displace the vectors; with everything in L2 they
// cost 7 %).
constexpr int ELL = 100, ELL_STREAM = 200;
constexpr long long ELL_STREAM_BYTES = 32 << 20;

constexpr int lanes_of(int format) { return format >= ELL ? 1 : format; }

struct EllGraph {
  int w = 0;  // 0: the graph has none
  const int* cols = nullptr;
  long long slots = 0;
};
inline int ell_format(int w, long long slots, size_t value_bytes) {
  return w ? (slots * (long long)(value_bytes + sizeof(int)) > ELL_STREAM_BYTES ? ELL_STREAM : ELL) + w : 1;
}

template <bool STREAM, class X>
__device__ __forceinline__ X ell_load(const X* p) {
  return STREAM ? __ldcs(p) : __ldg(p);
}

// sum of value * get(column) over row i, in slot order
template <int FORMAT, class T, class G>
__device__ __forceinline__ double ell_row(const int* __restrict__ cols, const T* __restrict__ val, int i, G get) {
  constexpr int W = FORMAT % 100;
  constexpr bool STREAM = FORMAT >= ELL_STREAM;
  const size_t at = (size_t)(i >> 5) * (32 * W) + (i & 31);
  int j[W];
  T v[W];
#pragma unroll
  for (int q = 0; q < W; ++q) {
    j[q] = ell_load<STREAM>(cols + at + 32 * q);
    v[q] = ell_load<STREAM>(val + at + 32 * q);
  }
  double s = 0.0;
#pragma unroll
  for (int q = 0; q < W; ++q) s += double(v[q]) * get(j[q]);
  return s;
}

// Width and device columns of a graph (w 0 where it keeps CSR); the caller frees
// the columns.
int ell_graph(int n, const int* h_rp, const int* rp, const int* cols, EllGraph* out, cudaStream_t st);
// values of a CSR matrix into the fixed-width storage (padding zero)
template <class T>
int ell_values(int n, const int* rp, const T* csr, int w, T* out, cudaStream_t st);

}  // namespace oa
