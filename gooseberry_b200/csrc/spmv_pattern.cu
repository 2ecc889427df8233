// spmv_pattern.cu -- y = A x for pattern matrices (stencils): rows of at most
// 7 entries that form at most 256 distinct lists of column offsets from the
// diagonal.
//
// The row schedule streams a banded matrix larger than L2 at the copy rate, so
// what is left is its bytes: 12 an entry and 4 a row.  Two forms read fewer:
//   classes   at most 256 distinct rows, offsets AND values (constant
//             coefficients): one byte a row, the rows in shared memory
//   patterns  one byte a row for the columns, values from the CSR array
//             (through rowptr)
// On the 4096^2 Laplacian a pass moves 285 MB instead of 1.34 GB.  Rows are
// summed in CSR order with unfused multiply and add, as the row schedule does,
// so the result has its bits (and blas_spmult's, src/blas.c:82-91).  The
// autotuner builds the form and takes it when it times faster.
//
// A thread takes one row at a time, its next row's byte (and rowptr) loaded
// ahead; the offsets (and values) of a row's class stay in registers from one
// row to the next, reloaded when the class changes (on a grid, at its edges).
// Measured (us, row schedule -> here): 4000^2 grid, FP64 193 -> 72 (classes),
// 153 (patterns: 0.97 of the copy rate on its bytes); FP32 147 -> 48, 105;
// 200^3 FP64 135 -> 50, 100; FP32 100 -> 36, 66; 1000^2 FP64 11 -> 9.  Two and
// four rows at a time, without the next row's byte: 120-217 where one takes 86.
#include <algorithm>
#include <type_traits>

#include "cg_resident.h"
#include "gb_internal.h"
#include "spmv_tiles.cuh"

namespace gb {
namespace {

constexpr int kPatBlock = 256;

template <typename T, int STAGE, bool CLASS>
struct PatRow {
  int code = -1, len = 0;
  int off[STAGE];
  T val[CLASS ? STAGE : 1];
  __device__ __forceinline__ void load(int c, const unsigned char * table) {
    if (c == code) return;
    code = c;
    const int32_t * o = CLASS ? reinterpret_cast<const ResRowClass *>(table)[c].off
                              : reinterpret_cast<const int32_t *>(table) + c * kPatMax;
#pragma unroll
    for (int j = 0; j < STAGE; ++j) off[j] = o[j];
    len = o[kPatMax - 1];
    if constexpr (CLASS) {
#pragma unroll
      for (int j = 0; j < STAGE; ++j)
        val[j] = static_cast<T>(reinterpret_cast<const ResRowClass *>(table)[c].val[j]);
    }
  }
};

// CTAs per SM: as many as the registers hold without spills (one more of each:
// FP64 5 entries 72 -> 107 us at 6, FP32 7 entries 66 -> 91 us at 8).
template <typename T, int STAGE>
struct PatMinBlocks {
  static constexpr int value = sizeof(T) == 8 ? (STAGE == 5 ? 4 : 3) : (STAGE == 5 ? 8 : 6);
};

template <typename T, int STAGE, bool CLASS>
__global__ void __launch_bounds__(kPatBlock, PatMinBlocks<T, STAGE>::value)
spmv_pattern_kernel(uint32_t n, const uint8_t * __restrict__ codes,
    const void * __restrict__ table_g, uint32_t table_words,
    const uint32_t * __restrict__ rowptr, const T * __restrict__ val,
    const T * __restrict__ x, T * __restrict__ y, uint32_t stride) {
  extern __shared__ __align__(16) unsigned char table[];
  for (uint32_t i = threadIdx.x; i < table_words; i += kPatBlock)
    reinterpret_cast<uint32_t *>(table)[i] = static_cast<const uint32_t *>(table_g)[i];
  __syncthreads();
  const uint32_t step = gridDim.x * kPatBlock;
  uint32_t i = blockIdx.x * kPatBlock + threadIdx.x;
  if (i >= n) return;
  PatRow<T, STAGE, CLASS> w;
  int c = __ldg(codes + i);
  uint32_t b = CLASS ? 0u : __ldg(rowptr + i);
  for (; i < n; i += step) {
    w.load(c, table);
    T xv[STAGE], v[CLASS ? 1 : STAGE];
#pragma unroll
    for (int j = 0; j < STAGE; ++j)
      if (j < w.len) {
        xv[j] = __ldg(x + (i + static_cast<uint32_t>(w.off[j])));
        if constexpr (!CLASS) v[j] = __ldg(val + b + j);
      }
    const uint32_t nx = i + step;
    if (nx < n) {
      c = __ldg(codes + nx);
      if constexpr (!CLASS) b = __ldg(rowptr + nx);
    }
    T sum = T(0);
#pragma unroll
    for (int j = 0; j < STAGE; ++j)
      if (j < w.len) sum = add_rn(sum, mul_rn(CLASS ? w.val[CLASS ? j : 0] : v[CLASS ? 0 : j], xv[j]));
    y[static_cast<size_t>(i) * stride] = sum;
  }
}

template <typename T, int STAGE, bool CLASS>
int launch_t(const gb_csr & a, const SpmvPattern & p, const T * val, const T * x, T * y,
    uint32_t stride, cudaStream_t s) {
  auto kern = spmv_pattern_kernel<T, STAGE, CLASS>;
  const size_t bytes = CLASS ? p.cls.count * sizeof(ResRowClass) : p.pat.npat * kPatMax * 4;
  int occ = 0;
  GB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kPatBlock, bytes));
  const unsigned grid = static_cast<unsigned>(std::max<size_t>(1, std::min<size_t>(
      (a.nrows + kPatBlock - 1) / kPatBlock,
      static_cast<size_t>(a.sm_count) * std::max(occ, 1))));
  const void * table = CLASS ? static_cast<const void *>(p.cls.rows)
                             : static_cast<const void *>(p.pat.off);
  kern<<<grid, kPatBlock, bytes, s>>>(a.nrows, CLASS ? p.cls.code8 : p.pat.code8, table,
      static_cast<uint32_t>(bytes / 4), a.rowptr, val, x, y, stride);
  GB_CUDA_TRY(cudaGetLastError());
  return GOOSEBERRY_SUCCESS;
}

template <typename T>
int launch(const gb_csr & a, const SpmvPattern & p, const T * val, const T * x, T * y,
    uint32_t stride, cudaStream_t s) {
  const bool s5 = a.plan.max_row <= 5;
  if (p.cls.code8)
    return s5 ? launch_t<T, 5, true>(a, p, val, x, y, stride, s)
              : launch_t<T, 7, true>(a, p, val, x, y, stride, s);
  return s5 ? launch_t<T, 5, false>(a, p, val, x, y, stride, s)
            : launch_t<T, 7, false>(a, p, val, x, y, stride, s);
}

}  // namespace

int launch_spmv_pattern(const gb_csr & a, const SpmvPattern & p, const double * x, double * y,
    uint32_t stride, cudaStream_t s) {
  return launch(a, p, a.val64, x, y, stride, s);
}
int launch_spmv_pattern(const gb_csr & a, const SpmvPattern & p, const float * x, float * y,
    uint32_t stride, cudaStream_t s) {
  return launch(a, p, a.val32, x, y, stride, s);
}

int build_spmv_pattern(const gb_csr & a, bool f32, SpmvPattern ** out, cudaStream_t s) {
  *out = nullptr;
  if (a.nrows == 0 || a.nnz == 0 || a.plan.max_row > 7) return GOOSEBERRY_SUCCESS;
  SpmvPattern * p = new SpmvPattern();
  int rc = f32 ? build_row_classes(a, a.val32, &p->cls, s) : build_row_classes(a, a.val64, &p->cls, s);
  if (rc == GOOSEBERRY_SUCCESS && !p->cls.code8) rc = build_row_patterns(a, &p->pat, s);
  if (rc != GOOSEBERRY_SUCCESS || (!p->cls.code8 && !p->pat.code8)) {
    free_spmv_pattern(p);
    return rc;
  }
  *out = p;
  return GOOSEBERRY_SUCCESS;
}

void free_spmv_pattern(SpmvPattern * p) {
  if (!p) return;
  free_row_classes(p->cls);
  free_row_patterns(p->pat);
  delete p;
}

}  // namespace gb
