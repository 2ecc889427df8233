// cg_resident.h -- interface of the on-chip CG solver (cg_resident.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "gb_internal.h"

namespace gb {

// A whole matrix row shared by many rows: column offsets from the diagonal
// (the eighth slot is the length) and values.
struct ResRowClass {
  int32_t off[8];
  double val[8];
};

// The distinct rows of a matrix (rows of at most 7 entries), at most 256.
struct RowClasses {
  uint8_t * code8 = nullptr;     // [nrows]
  ResRowClass * rows = nullptr;  // [count]
  uint32_t count = 0;
};
// Leaves `out` empty past 256 classes, or for longer rows.
int build_row_classes(const gb_csr & a, const double * val, RowClasses * out, cudaStream_t s);
int build_row_classes(const gb_csr & a, const float * val, RowClasses * out, cudaStream_t s);
void free_row_classes(RowClasses & c);

// A pattern matrix for plain SpMV (spmv_pattern.cu): its classes, or else its
// column patterns.
struct SpmvPattern {
  RowPatterns pat;
  RowClasses cls;
};
// *out stays null when the matrix has neither.
int build_spmv_pattern(const gb_csr & a, bool f32, SpmvPattern ** out, cudaStream_t s);
void free_spmv_pattern(SpmvPattern * p);
int launch_spmv_pattern(const gb_csr & a, const SpmvPattern & p, const double * x, double * y,
    uint32_t stride, cudaStream_t s);
int launch_spmv_pattern(const gb_csr & a, const SpmvPattern & p, const float * x, float * y,
    uint32_t stride, cudaStream_t s);

// What the solve kernel reports, in pinned host memory.
struct ResResult {
  int status;
  int aborted;  // some CTA gave up waiting
  unsigned long long iter;
  double rr, bnorm;
  unsigned epoch;  // all-reduces so far
  unsigned long long ns_a, ns_b;  // time in the two phases (a timed solve)
};

struct ResOutcome {
  ResResult result{};
  bool cancelled_waiting = false;  // cancelled before it got its SMs
};

// The matrix as the FP64 solver has laid it out (cg.cu).
struct ResidentIn {
  const RowPatterns * pat = nullptr;
  int stage = 0;               // 5 or 7 entries a row at most
  bool plain = false;          // read the CSR arrays
  const uint2 * ell8 = nullptr;
  const double * table = nullptr;
  uint32_t ntable = 0;
  const void * ellv = nullptr;
  int ellv_width = 0;
  bool ellv_f32 = false;
};

struct ResidentCg;
// Whether a matrix of this many rows can be solved on the chip at all.
bool resident_size_ok(const gb_csr & a);
// *out stays null when the system does not fit the chip; the solution is
// left in `x` (device, n doubles).
int resident_create(const gb_csr & a, const ResidentIn & in, double * x, ResidentCg ** out);
void resident_destroy(ResidentCg * s);
// Runs a solve to its end.  `result.aborted` asks the caller to run the solve
// another way.
int resident_solve(ResidentCg * s, const double * b, double tol, int tol_relative,
    unsigned long long niter, double * dhist, unsigned long long hist_len,
    const int * cancel_h, const int * cancel_d, bool timed, cudaStream_t stream,
    ResOutcome * res);

// SMs of a device shared by the grids whose CTAs wait for one another; false
// if `cancel` (host, may be null) was set before the SMs were free.
bool resident_acquire(int device, unsigned ctas, unsigned capacity, const int * cancel);
void resident_release(int device, unsigned ctas, unsigned capacity);

}  // namespace gb
