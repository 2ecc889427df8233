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
  unsigned long long ran;  // iterations of this launch
  double rr, bnorm;
  double pap, beta;  // of the last iteration, for a solve that goes on
  unsigned epoch;  // all-reduces so far
  unsigned long long ns_a, ns_b;  // time in the two phases (a timed solve)
  unsigned long long t0, t1;      // begin and end
  int done;                       // written last (with ResArgs::arrived)
};

// `status` of a launch that ended before its solve (ResArgs::more).
constexpr int kResPaused = 100;

// ---- the solve kernel's arguments ------------------------------------------------
// What has a place in shared memory besides p, Ap, the tables and the row bytes.
struct ResPlaces {
  int x, halo;  // x (else in L2); the neighbours' r as fetched (else not fetched ahead)
};

struct ResArgs {
  uint32_t n, rows, halo, ctas;
  int tol_relative;
  ResPlaces at;
  const uint8_t * row_code;       // class or pattern of each row
  const ResRowClass * classes;    // RES_CLASS
  const int32_t * pat_off;        // the other pattern sources
  uint32_t ncode;                 // classes or patterns
  const void * vals;              // rows of values or codes
  int val_width;                  // elements per row of `vals`
  const double * table;           // RES_CODES
  uint32_t ntable;
  const uint32_t * rowptr;        // RES_CSR
  const uint32_t * rowind;
  const double * val64;
  const double * b;
  double * x;
  ulonglong2 * r_edge;            // [n] tagged r; only rows near a block edge are used
  unsigned long long * words;     // [2][16]: the fixed-point sums (3 of 16 used)
  ulonglong2 * box;               // [2][ctas] tagged partials
  int * abort_flag;
  const int * cancel;
  ResResult * out;                // host-mapped
  double * hist;
  unsigned long long hist_len, niter;
  uint32_t epoch0;
  double tol;
  int timed;                      // report the phases' times
  // With `more` the launch's niter is not the solve's: it leaves r and p in r_save
  // and p_save [n].  One that goes on takes them, x and the scalars below.
  double * r_save;
  double * p_save;
  int more, resume;
  unsigned long long it0;
  double rr0, pap0, beta0, bnorm0;
  unsigned long long wait_ns;     // a wait that lasts longer is given up
  unsigned long long late_ns;     // for tests: CTA 0 is that late after iteration 64
  unsigned * arrived;             // may be null; 0 before: count the CTAs out, so that the last
                                  // one reports `done` and no event has to follow the launch
};

// One solve's grid and kernel, from its size alone: matrix values in shared
// memory, read from the CSR arrays (args.vals stays null).  fn is null when the
// system does not fit.  `want`: rows a CTA should own.
struct ResShape {
  ResArgs args{};
  const void * fn = nullptr;
  size_t smem = 0;
  int threads = 0;
  int fault = GB_CHIP_FAULT_NONE;  // for tests
};
// A launch's time: how often what waits for SMs (other solves, other streams'
// kernels) gets its turn.  A launch more costs 22 us at 400^2, 31 us at 1024^2.
constexpr double kResSliceNs = 1e7;
// The niter of a solve's next launch, of about `ns`, after `last` (null: the
// first); with p_save null there is only one.
void resident_slice(ResArgs * g, unsigned long long niter, int fault, double ns,
    const ResResult * last);
// Sets the limit of a solve's waits (0: the usual one) and, for tests, a fault.
void resident_set_waits(ResArgs * g, int fault, unsigned limit_ms);
int resident_shape(uint32_t n, uint32_t half, int max_row, uint32_t npat, int sms, uint32_t want,
    ResShape * out);
// Load every kernel that resident_shape may choose.  A kernel is otherwise
// loaded at its first use, and what is launched after a load waits until the
// kernels that run have ended: a request behind a long solve would wait for it.
int resident_preload();
// Enqueue a solve.  The caller holds the grid's SMs (resident_try_acquire) until
// it has ended, and has cleared words, box, abort flag and r_edge.
int resident_launch(const ResShape & sh, ResArgs args, cudaStream_t stream, bool * refused);
constexpr int kResMaxCtas = 160;  // tagged partials polled, 5 a lane

// r = b - A x and r.r into *rr (may be host-mapped), with `grid` partials and a
// ticket that is 0 before and after; x += d (cg.cu).
int launch_true_residual(uint32_t n, const uint32_t * rowptr, const uint32_t * rowind,
    const double * val, const double * b, const double * x, double * r, double * partial,
    unsigned grid, double * rr, unsigned * ticket, cudaStream_t stream);
int launch_add_to(size_t n, const double * d, double * x, unsigned grid, cudaStream_t stream);
int preload_true_residual();  // loads the two kernels above

struct ResOutcome {
  ResResult result{};
  unsigned launches = 0;
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

// For tests of the give-up path: what the following solves do (GB_CHIP_FAULT_*)
// and the limit of their waits in ms (0: the usual one); false if the solve has
// one CTA, which waits for nobody.
bool resident_set_fault(ResidentCg * s, int fault, unsigned limit_ms);

// SMs of a device shared by the grids whose CTAs wait for one another.  Each
// returns an id to release them by, or 0.  Waits for them at the head of the
// queue for limit_ns at most, and not once `cancel` (host, may be null) is set.
unsigned long long resident_acquire(int device, unsigned ctas, unsigned capacity,
    const int * cancel, unsigned long long limit_ns, bool * cancelled);
// Without waiting: 0 if the SMs are not free, or others wait for some.  They are
// free again when `done` (host, zero now) is set, or when they are released.
unsigned long long resident_try_acquire(int device, unsigned ctas, unsigned capacity,
    const int * done);
void resident_release(int device, unsigned long long id);

}  // namespace gb
