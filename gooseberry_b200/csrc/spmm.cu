// spmm.cu -- C = A B for several right-hand sides in one launch (the
// reference's __sparse_mult_dense_block with bncols > 1, src/blas.c:67-92).
//
// B is column-major (B[j * ncols + c], the reference's layout), C row-major
// (C[i * k + j]).  One thread per row (grid-stride): the row's first
// kSpmmStage (or, when every row fits, 5 or 7) indices and values are loaded
// once into registers, then for each group of up to four columns all of the
// row's gathers from those columns of B are issued before any is used, and the
// group's entries of C are written, where they fill a 32-byte sector, in one
// store.  Each element is summed k ascending with unfused multiply and add,
// exactly like the reference's inner loop, so C is bit-identical to
// blas_spmult's.  Against one SpMV per column, A's indices and values leave
// memory once instead of k times and the product is one launch.  Matrices with
// rows too long for one thread keep the per-column SpMV.
#include <algorithm>

#include "gb_internal.h"
#include "spmv_tiles.cuh"

namespace gb {
namespace {

constexpr int kSpmmBlock = 256;
constexpr int kSpmmStage = 8;  // a row's entries held in registers (longer rows: tail loop)

// N values to consecutive addresses p, p + 1, ...; `wide`: p is aligned to
// all of them
template <typename T, int N>
__device__ __forceinline__ void store_run(T * p, const T (&v)[N], bool wide) {
  if constexpr (N == 4 && sizeof(T) == 8) {
    if (wide) {
      asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]),
                   "d"(v[2]), "d"(v[3])
                   : "memory");
      return;
    }
  } else if constexpr (N == 4 && sizeof(T) == 4) {
    if (wide) {
      *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
      return;
    }
  } else if constexpr (N == 2 && sizeof(T) == 8) {
    if (wide) {
      *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
      return;
    }
  }
#pragma unroll
  for (int q = 0; q < N; ++q) p[q] = v[q];
}

template <typename T, int STAGE, int COLS, int MINB>
__global__ void __launch_bounds__(kSpmmBlock, MINB) spmm_rows_kernel(
    uint32_t nrows, uint32_t ncols, uint32_t k, const uint32_t * __restrict__ rowptr,
    const uint32_t * __restrict__ rowind, const T * __restrict__ val, const T * __restrict__ b,
    T * __restrict__ c, bool wide) {
  const uint32_t cmax = ncols - 1;
  for (uint32_t i = blockIdx.x * kSpmmBlock + threadIdx.x; i < nrows;
       i += gridDim.x * kSpmmBlock) {
    const uint32_t rb = __ldg(rowptr + i), re = __ldg(rowptr + i + 1);
    uint32_t col[STAGE];
    T w[STAGE];
#pragma unroll
    for (int s = 0; s < STAGE; ++s)
      if (rb + s < re) {
        col[s] = min(__ldg(rowind + rb + s), cmax);
        w[s] = __ldg(val + rb + s);
      }
    T * crow = c + static_cast<size_t>(i) * k;
    uint32_t j = 0;
    if constexpr (COLS > 1) for (; j + COLS <= k; j += COLS) {
      const T * bj = b + static_cast<size_t>(j) * ncols;
      T x[COLS][STAGE];
#pragma unroll
      for (int q = 0; q < COLS; ++q)
#pragma unroll
        for (int s = 0; s < STAGE; ++s)
          if (rb + s < re) x[q][s] = __ldg(bj + q * static_cast<size_t>(ncols) + col[s]);
      T acc[COLS];
#pragma unroll
      for (int q = 0; q < COLS; ++q) {
        acc[q] = T(0);
#pragma unroll
        for (int s = 0; s < STAGE; ++s)
          if (rb + s < re) acc[q] = add_rn(acc[q], mul_rn(w[s], x[q][s]));
      }
      for (uint32_t t = rb + STAGE; t < re; ++t) {  // long-row tail
        const uint32_t ct = min(__ldg(rowind + t), cmax);
        const T wt = __ldg(val + t);
#pragma unroll
        for (int q = 0; q < COLS; ++q)
          acc[q] = add_rn(acc[q], mul_rn(wt, __ldg(bj + static_cast<size_t>(q) * ncols + ct)));
      }
      store_run<T, COLS>(crow + j, acc, wide);
    }
    for (; j < k; ++j) {
      const T * bj = b + static_cast<size_t>(j) * ncols;
      T x[STAGE];
#pragma unroll
      for (int s = 0; s < STAGE; ++s)
        if (rb + s < re) x[s] = __ldg(bj + col[s]);
      T acc = T(0);
#pragma unroll
      for (int s = 0; s < STAGE; ++s)
        if (rb + s < re) acc = add_rn(acc, mul_rn(w[s], x[s]));
      for (uint32_t t = rb + STAGE; t < re; ++t)  // long-row tail
        acc = add_rn(acc, mul_rn(__ldg(val + t), __ldg(bj + min(__ldg(rowind + t), cmax))));
      crow[j] = acc;
    }
  }
}

}  // namespace

// Longest row the fused kernel takes: a thread walks its rows alone.
constexpr uint32_t kSpmmMaxRow = 256;

template <typename T>
int launch_spmm_fused(const gb_csr & a, uint32_t k, const T * vals, const T * b, T * c,
    cudaStream_t stream, bool * done) {
  *done = false;
  if (a.plan.max_row > kSpmmMaxRow || k < 2) return GOOSEBERRY_SUCCESS;
  *done = true;
  if (a.nrows == 0) return GOOSEBERRY_SUCCESS;
  int sms = 148;
  GB_TRY(sm_count_of_current_device(&sms));
  const uint32_t grid = std::max<uint32_t>(1, std::min<uint32_t>(
      (a.nrows + kSpmmBlock - 1) / kSpmmBlock, static_cast<uint32_t>(sms) * 8));
  // Columns at a time (us, one column or a pair at a time -> four): 1024^2
  // Laplacian, k = 8 62 -> 54; 700^2, k = 16 69 -> 47; 100^3, k = 8 84 -> 66, k =
  // 16 176 -> 111.  With fewer than four columns a pair (5 entries: k = 2 27 us,
  // where the four-column form takes 39), or one (7 entries: k = 3 29 us, 40).
  // Two CTAs an SM, so that the 20 or 28 gathers in flight have registers:
  // at three the compiler spills (95 us for the first).
  uint32_t cols = 1;
  auto kern = spmm_rows_kernel<T, kSpmmStage, 1, 4>;
  if (a.plan.max_row <= 5) {
    cols = k >= 4 ? 4 : 2;
    kern = k >= 4 ? spmm_rows_kernel<T, 5, 4, 2> : spmm_rows_kernel<T, 5, 2, 3>;
  } else if (a.plan.max_row <= 7 && k >= 4) {
    cols = 4;
    kern = spmm_rows_kernel<T, 7, 4, 2>;
  }
  const bool wide = k % cols == 0 && reinterpret_cast<uintptr_t>(c) % (cols * sizeof(T)) == 0;
  kern<<<grid, kSpmmBlock, 0, stream>>>(a.nrows, std::max<uint32_t>(a.ncols, 1), k, a.rowptr,
      a.rowind, vals, b, c, wide);
  GB_CUDA_TRY(cudaGetLastError());
  return GOOSEBERRY_SUCCESS;
}

template int launch_spmm_fused<double>(const gb_csr &, uint32_t, const double *, const double *,
    double *, cudaStream_t, bool *);
template int launch_spmm_fused<float>(const gb_csr &, uint32_t, const float *, const float *,
    float *, cudaStream_t, bool *);

}  // namespace gb
