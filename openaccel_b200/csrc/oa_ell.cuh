// Fixed-width row storage of a scalar CSR matrix (internal).
//
// Rows come in groups of 32; slot q of row i sits at 32 (W (i / 32) + q) + i % 32.
// A warp whose lanes take one row each then reads every slot as one contiguous
// line of values (in CSR the same loads are strided by the row length), needs no
// row pointer in its chain of dependent loads, and has all W slots in flight at
// once. W is a compile-time constant, for the two row lengths of the stencils
// this library assembles: 7 (a node of a hex block and its edge neighbours) and
// 15 (a node of a block split into Kuhn tets, or of hex blocks around an axis). A
// graph takes 7 where no row is longer, 15 where none is longer than that, and
// keeps CSR otherwise, where the slots are more than 2 nnz + 4096 and where device
// memory is short.
//
// In a block's numbering the 32 rows of a group have their columns at the same
// few distances, so a group keeps the distances once where W of them hold all its
// rows' columns, and a row the set of slots it has (2 bytes): the product is
// bound by DRAM, and columns of 4 bytes per entry are half of an FP32 matrix.
// Groups with more distances (ends of blocks, unordered meshes) read columns.
//
// Measured product, matrix in DRAM: 97^3 rows FP64 CSR 22.8 us, with columns 14.8;
// 129^3 rows FP32 32.8 and 20.7; a run-time width lost most of it (20.7 and 28.9
// us). On 129^3 rows FP32 with columns and with distances: smoothing step with
// residual 24.7 and 22.8 us, smoothing step 23.8 and 20.9, product in GCR 26.6
// and 24.7. Absent slots have value 0 and a column that the row reads anyway: the
// row itself by distances, the row's first one by columns.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace oa {

// Formats of a row product: lanes per row of a CSR matrix (1, 4, 8, 32), or ELL +
// width, or, for a matrix that does not fit L2 beside the vectors, ELL_STREAM +
// width (loads that do not displace the vectors; with everything in L2 they
// cost 7 %).
constexpr int ELL = 100, ELL_STREAM = 200;
constexpr long long ELL_STREAM_BYTES = 32 << 20;

// Width that keeps distances; with 15 of them the products ran out of registers
// (conduction on 65^3 nodes, mixed: 2.47 ms with columns, 2.90 with distances).
constexpr int ELL_DISTANCES = 7;

constexpr int lanes_of(int format) { return format >= ELL ? 1 : format; }

struct EllGraph {
  int w = 0;  // 0: the graph has none
  int* cols = nullptr;  // [n/32][W][32], and after it in the same allocation:
  const int* delta = nullptr;       // [n/32][W + 1] distances; 1 last where the rows read columns
  const uint16_t* mask = nullptr;   // [n] slots of each row
  long long slots = 0;
};
template <class T>
struct EllMat {
  const int *cols, *delta;
  const uint16_t* mask;
  const T* val;
};
template <class T>
inline EllMat<T> ell_mat(const EllGraph& g, const T* val) {
  return {g.cols, g.delta, g.mask, val};
}
inline int ell_format(int w, long long slots, size_t value_bytes) {
  return w ? (slots * (long long)value_bytes > ELL_STREAM_BYTES ? ELL_STREAM : ELL) + w : 1;
}

template <bool STREAM, class X>
__device__ __forceinline__ X ell_load(const X* p) {
  return STREAM ? __ldcs(p) : __ldg(p);
}

// sum of value * get(column) over row i, in slot order
template <int FORMAT, class T, class G>
__device__ __forceinline__ double ell_row(const EllMat<T>& m, int i, G get) {
  constexpr int W = FORMAT % 100;
  constexpr bool STREAM = FORMAT >= ELL_STREAM;
  const size_t at = (size_t)(i >> 5) * (32 * W) + (i & 31);
  T v[W];
  int j[W + 1];
#pragma unroll
  for (int q = 0; q < W; ++q) v[q] = ell_load<STREAM>(m.val + at + 32 * q);
  if constexpr (W == ELL_DISTANCES) {
    const unsigned mask = __ldg(m.mask + i);
    const int4* d = reinterpret_cast<const int4*>(m.delta + (size_t)(i >> 5) * (W + 1));
#pragma unroll
    for (int q = 0; q < W + 1; q += 4) {
      const int4 t = __ldg(d + q / 4);
      j[q] = t.x;
      j[q + 1] = t.y;
      j[q + 2] = t.z;
      j[q + 3] = t.w;
    }
    if (j[W]) {
#pragma unroll
      for (int q = 0; q < W; ++q) j[q] = ell_load<STREAM>(m.cols + at + 32 * q);
    } else {
#pragma unroll
      for (int q = 0; q < W; ++q) j[q] = mask >> q & 1 ? i + j[q] : i;
    }
  } else {
#pragma unroll
    for (int q = 0; q < W; ++q) j[q] = ell_load<STREAM>(m.cols + at + 32 * q);
  }
  double s = 0.0;
#pragma unroll
  for (int q = 0; q < W; ++q) s += double(v[q]) * get(j[q]);
  return s;
}

// Width and device graph (w 0 where it keeps CSR); the caller frees cols.
int ell_graph(int n, const int* h_rp, const int* rp, const int* cols, EllGraph* out, cudaStream_t st);
// values of a CSR matrix into the fixed-width storage (absent slots zero)
template <class T>
int ell_values(int n, const int* rp, const T* csr, const EllGraph& g, T* out, cudaStream_t st);

}  // namespace oa
