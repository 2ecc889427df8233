// cg_resident.cu -- conjugate gradient with the Krylov vectors on the chip.
//
// The graph-replayed solver (cg.cu) streams r, p, Ap and x through L2 twice
// per iteration (about 90 bytes a row) and pays two dependent launches.  A
// system whose vectors fit the SMs' shared memory and registers needs
// neither: here cooperative launches of many iterations run the solve, one CTA
// per SM, each CTA owning a contiguous block of rows for its whole life.
//
//   shared memory  p over the CTA's rows and H rows on either side (H = the
//                  matrix's half bandwidth), Ap, x, the row patterns, and the
//                  matrix values when they fit
//   registers      r of the rows a thread owns
//   L2             the r values within H rows of a block edge, which the
//                  neighbours read, and the messages of the all-reduces
//
// Per iteration:
//   A  p = r + beta p on the own rows; the halo's p is updated the same way
//      from the neighbours' r (the same fma on the same operands, so every
//      copy of a p value has the same bits); Ap from shared memory; p.Ap.
//   -- all-reduce: every CTA gets p.Ap, alpha
//   B  r -= alpha Ap, r.r; the block's edge r values go to L2
//   -- all-reduce: r.r, beta, the stop test; meanwhile the warps that would
//      wait for it do x += alpha p and fetch the neighbours' r
//
// The all-reduce is one hop, and exact: a CTA turns its partial sum into a
// 131-bit fixed-point number, scaled by the previous iteration's sum, and adds
// it with three 64-bit reductions to three words in L2, each of which also
// counts its arrivals in its top byte; three lanes of every CTA poll the words
// until all CTAs are in.  Integer addition is associative, so the sum does not
// depend on the order of arrival: every CTA holds the same bits, and so does
// every run.  Measured among 148 CTAs of 512 threads, with the sum within the
// CTA: 2,060 clocks, against 4,570 for an arrival counter and an array of
// partials, 6,700 for a mailbox per CTA that all others write, and 11,240 for
// one array of tagged partials that all poll (two CTAs: 1,830, the store and
// the poll that any exchange through L2 pays).  The words run on for ever (a
// reader keeps the value it saw last), so nothing has to be cleared.  Sums of
// unknown scale (the first ones, and any that left the range of the fixed
// point) go through the tagged array instead.
//
// An r value for a neighbour is two 64-bit words of half a double and a tag
// each, so a word that has arrived carries its own proof: no fence and no flag
// behind it.  An r value of one iteration is read before the reader adds its
// p.Ap of the next, and overwritten only after that all-reduce.
//
// Measured per iteration (us, B200), graph path -> here: 1024^2 Laplacian 20.9
// -> 8.6; variable coefficients 1024^2 23.9 -> 11.7, 400^2 9.0 -> 4.1, 96^2 7.0
// -> 3.3, 64^3 12.5 -> 8.1.  What an iteration of the 1024^2 Laplacian (7,086
// rows a CTA) spends, in clocks of 16,500: row sums 5,200 (shared-memory
// loads: 15 wavefronts a 32-row sum, floor 3,400), p updates 1,500, the
// exchanges 2,600 and 5,900 (the second as long as the x update and the
// neighbours' r take behind it), r 570, two divisions 600.  Small systems wait
// for the two exchanges, which cost what L2 does: 2,100 clocks each.
//
// A launch runs for as many iterations as take about kResSliceNs, writes r and p
// beside x and ends, so that other streams' kernels, which find no room on SMs
// held so, get their turn; the next launch goes on with the same bits.  (A clock
// read by the CTAs and a request to pause sent with the sums cost 2-5% of every
// iteration; the count costs nothing, as the limit is checked anyway.)
//
// A wait that lasts longer than a limit raises the abort flag; every CTA
// leaves, and the host runs the solve on the graph path instead.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "cg_common.cuh"
#include "cg_resident.h"
#include "gb_internal.h"
#include "spmv_tiles.cuh"

namespace gb {
namespace {

// Threads and rows a thread: 512 threads (128 registers) up to 8 rows each,
// 384 (168 registers) up to 19 past that: r takes two registers a row, and at
// 512 threads the 14-row form issued its shared-memory loads one at a time
// (every phase 2-3 times slower) or spilled.
constexpr int kResThreads = 512, kResRows = 8;
constexpr int kResThreadsWide = 384, kResRowsWide = 19;
// Up to here one CTA, which needs no exchange (variable coefficients, 1,600
// rows: 2.68 us an iteration, 3.36 over four CTAs; 2,304 rows: 3.41 and 3.39).
constexpr uint32_t kResOneCta = 2048;
constexpr unsigned long long kResWaitNs = 2000000000ull;

// How a CTA finds its matrix rows.
enum ResSource {
  RES_CLASS = 0,   // a byte per row naming one of <= 256 whole rows (offsets and values)
  RES_SMEM_F64 = 1,  // pattern byte; doubles in shared memory, slot-major
  RES_SMEM_F32 = 2,  // pattern byte; exact floats in shared memory, slot-major
  RES_GLOBAL_F64 = 3,  // pattern byte; rows of 6 or 8 doubles in global memory
  RES_GLOBAL_F32 = 4,  // pattern byte; rows of 8 exact floats in global memory
  RES_CODES = 5,   // pattern byte; rows of 8 value codes in global memory
  RES_CSR = 6      // the plain CSR arrays
};

// Shared-memory regions, the same on host and device.
struct ResLayout {
  size_t p, ap, x, halo, vals, table, codes, total;
  __host__ __device__ ResLayout(uint32_t rows, uint32_t half, int threads, ResPlaces at,
      size_t val_bytes_row, size_t table_bytes) {
    const size_t r = rows, h = half;
    size_t o = 0;
    p = o;
    o += 8 * (r + 2 * h);
    ap = o;
    o += 8 * ((r + threads - 1) / threads * threads);  // read unguarded
    x = o;
    if (at.x) o += 8 * r;
    halo = o;
    if (at.halo) o += 16 * h;
    o = (o + 15) / 16 * 16;
    vals = o;
    o += val_bytes_row * r;
    o = (o + 15) / 16 * 16;
    table = o;
    o += (table_bytes + 15) / 16 * 16;
    codes = o;
    total = (o + r + 15) / 16 * 16;
  }
};

__host__ __device__ constexpr size_t res_val_bytes(int src, int stage) {
  return src == RES_SMEM_F64 ? 8 * stage : src == RES_SMEM_F32 ? 4 * stage : 0;
}

__host__ __device__ inline size_t res_table_bytes(int src, uint32_t ncode, uint32_t ntable) {
  return src == RES_CLASS ? ncode * sizeof(ResRowClass)
         : src == RES_CSR ? 0
                          : ncode * kPatMax * 4 + (src == RES_CODES ? ntable * 8 : 0);
}

__device__ __forceinline__ unsigned long long res_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// A double with a tag, as two words that are each whole on arrival.
__device__ __forceinline__ void tagged_store(ulonglong2 * p, double v, uint32_t tag) {
  const unsigned long long b = __double_as_longlong(v), t = static_cast<unsigned long long>(tag)
                                                            << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p),
               "l"(t | (b & 0xffffffffull)), "l"(t | (b >> 32))
               : "memory");
}
__device__ __forceinline__ ulonglong2 tagged_load(const ulonglong2 * p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
               : "=l"(v.x), "=l"(v.y)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ bool tag_is(const ulonglong2 & m, uint32_t tag) {
  return static_cast<uint32_t>(m.x >> 32) == tag && static_cast<uint32_t>(m.y >> 32) == tag;
}
__device__ __forceinline__ double tagged_value(const ulonglong2 & m) {
  return __longlong_as_double(static_cast<long long>((m.x & 0xffffffffull) | (m.y << 32)));
}

// Every 256 polls: has some CTA given up, or is it time to?
__device__ __forceinline__ bool res_give_up(const ResArgs & a, unsigned polls,
    unsigned long long * t0) {
  if (polls & 255u) return false;
  if (*reinterpret_cast<volatile int *>(a.abort_flag)) return true;
  const unsigned long long now = res_ns();
  if (*t0 == 0) *t0 = now;
  if (now - *t0 <= a.wait_ns) return false;
  atomicExch(a.abort_flag, 1);
  return true;
}

// A test's late CTA.
__device__ __forceinline__ void res_be_late(unsigned long long ns) {
  const unsigned long long end = res_ns() + ns;
#pragma unroll 1
  for (unsigned k = 0; k < (1u << 24) && res_ns() < end; ++k) __nanosleep(2000);
}

__device__ __forceinline__ double warp_allsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

struct ResShared {
  double red[32];
  double total;
  int bad;         // a wait in this CTA was given up
  int cancel;      // the host asked to stop (CTA 0's view, as of this all-reduce)
  int cancel_req;  // CTA 0: what it will send
  double bnorm, tol, rr_far;
};

// The exchange state of a CTA (warp 0's copy is used): counts of the sums so
// far, which pick the buffers, and the words as last seen (lanes 0-2).
struct ResSums {
  uint32_t tagged, fixed;
  unsigned long long seen0, seen1;
};

// Every CTA's `v` by tagged messages, added in CTA order: lane l adds those of
// CTAs l, l + 32, ..., then the warp tree.  All lanes of warp 0 call it.
__device__ __forceinline__ double res_sum_tagged(const ResArgs & a, ResShared & sh, ResSums & st,
    uint32_t epoch, double v, int * cancel) {
  const int lane = threadIdx.x & 31;
  ulonglong2 * const box = a.box + (st.tagged++ & 1) * a.ctas;
  const uint32_t tag = epoch << 1;
  if (lane == 0) tagged_store(box + blockIdx.x, v, tag | static_cast<uint32_t>(*cancel));
  constexpr unsigned long long kNoCancel = ~(1ull << 32);
  unsigned long long t0 = 0;
  unsigned polls = 0;
  double acc = 0.0;
  for (uint32_t c = lane; c < a.ctas; c += 32) {
    ulonglong2 m = tagged_load(box + c);
    while (!tag_is(make_ulonglong2(m.x & kNoCancel, m.y & kNoCancel), tag)) {
      if (res_give_up(a, ++polls, &t0)) {
        sh.bad = 1;
        break;
      }
      m = tagged_load(box + c);
    }
    acc += tagged_value(m);
    if (c == 0) *cancel = static_cast<int>((m.x >> 32) & 1u);
  }
  *cancel = __shfl_sync(0xffffffffu, *cancel, 0);
  return warp_allsum(acc);
}

// The same by fixed-point words.  A CTA's number is |v| / 2^(E - 131) cut into
// 46, 46 and 39 bits (lanes 0, 1, 2), each with v's sign and a bias that makes
// it positive, E = the exponent of `prev` + 40; field sums of 160 CTAs stay
// below 2^55, 2^55 and 2^48 of the 56 bits a word has beside its count.  Above
// them: a cancel request (CTA 0's, bit 55 of word 1) and the number of CTAs
// whose v did not fit (bits 48.. of word 2).  Returns false if some v did not
// fit or the sum is so much smaller than `prev` that the cut-off bits
// (2^(E - 131) a CTA) would show in its 53.
template <class S>
__device__ __forceinline__ bool res_sum_fixed(const ResArgs & a, ResShared & sh, ResSums & st,
    double v, double prev, int * cancel, double * total, S && sent) {
  const int lane = threadIdx.x & 31;
  const int e = ((__double2hiint(prev) >> 20) & 0x7ff) - 1023 + 40;
  const bool odd = st.fixed++ & 1;
  const unsigned long long seen = odd ? st.seen1 : st.seen0;
  unsigned long long * const w = a.words + (odd ? 16 : 0) + lane;
  if (lane < 3) {
    const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(v));
    const int ex = static_cast<int>(bits >> 52) & 0x7ff;
    // |v| = m 2^(ex - 1075); subnormals (0 among them) count as 0
    const unsigned long long m = ex ? (bits & ((1ull << 52) - 1)) | 1ull << 52 : 0ull;
    const bool fits = ex - 1023 < e;
    const int width = lane == 2 ? 39 : 46, pos = lane == 0 ? 85 : lane == 1 ? 39 : 0;
    const int up = ex - 1075 - (e - 131) - pos;  // shift of m to the field's lowest bit
    const unsigned long long t = up >= 0 ? (up < 64 ? m << up : 0ull) : (up > -64 ? m >> -up : 0ull);
    const long long c = static_cast<long long>(t & ((1ull << width) - 1));
    unsigned long long q = (1ull << width) + static_cast<unsigned long long>(
        static_cast<long long>(bits) < 0 ? -c : c);
    if (!fits) q = (1ull << width) + (lane == 2 ? 1ull << 48 : 0ull);
    if (lane == 1 && *cancel && blockIdx.x == 0) q |= 1ull << 55;
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(w), "l"(q + (1ull << 56))
                 : "memory");
  }
  sent();
  // One poll in flight: more of them queue at the words' L2 slice and delay
  // the arrivals (three, 250 clocks apart: 2,490 -> 3,490 clocks a sum).
  unsigned long long cur = 0, t0 = 0;
  for (unsigned polls = 1;; ++polls) {
    if (lane < 3) asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(cur) : "l"(w) : "memory");
    const bool all = lane >= 3 || static_cast<uint32_t>((cur - seen) >> 56) == a.ctas;
    if (__all_sync(0xffffffffu, all)) break;
    if (__any_sync(0xffffffffu, res_give_up(a, polls, &t0))) {
      sh.bad = 1;
      break;
    }
  }
  if (odd) st.seen1 = cur;
  else st.seen0 = cur;
  cur = (cur - seen) & ((1ull << 56) - 1);
  const unsigned long long w0 = __shfl_sync(0xffffffffu, cur, 0);
  const unsigned long long w1 = __shfl_sync(0xffffffffu, cur, 1);
  const unsigned long long w2 = __shfl_sync(0xffffffffu, cur, 2);
  *cancel = static_cast<int>(w1 >> 55);
  const bool unfit = (w2 >> 48) != 0;
  const long long n = a.ctas;
  long long lo = static_cast<long long>(w2 & ((1ull << 48) - 1)) - (n << 39);
  long long mid = static_cast<long long>(w1 & ((1ull << 55) - 1)) - (n << 46) + (lo >> 39);
  const long long hi = static_cast<long long>(w0) - (n << 46) + (mid >> 46);
  lo &= (1ll << 39) - 1;
  mid &= (1ll << 46) - 1;
  const double s = __ll2double_rn(hi) +
                   (__ll2double_rn(mid) + __ll2double_rn(lo) * 0x1p-39) * 0x1p-46;
  *total = s * __hiloint2double((e - 46 + 1023) << 20, 0);
  return !unfit && s >= 0x1p-23;
}

// Sum of every CTA's `local` (over its threads), the same bits in every CTA.
// `prev`: a sum of about this size, the same in every CTA (0: unknown).  Warps
// 1.. run `hidden` while warp 0 exchanges the sums, and warp 0 runs `sent` between
// its send and its wait.  Returns false when a wait was given up, in every thread
// of the CTA alike: sh.bad is written between the two barriers here, and elsewhere
// only behind a barrier that follows.
template <int T, class F, class S>
__device__ __forceinline__ bool res_allreduce(const ResArgs & a, ResShared & sh, ResSums & st,
    uint32_t & epoch, double local, double prev, F && hidden, S && sent, double * total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  local = warp_allsum(local);
  if (lane == 0) sh.red[warp] = local;
  __syncthreads();
  if (warp == 0) {
    const double v = warp_allsum(lane < T / 32 ? sh.red[lane] : 0.0);
    double sum = v;
    int cancel = sh.cancel_req;
    if (a.ctas > 1) {
      // (the bounds keep the fixed point's unit and the sum normal)
      const bool known = prev > 0x1p-960 && prev < INFINITY;
      const int asked = cancel;
      if (!known) sent();
      if (!known || !res_sum_fixed(a, sh, st, v, prev, &cancel, &sum, sent)) {
        cancel = asked;
        sum = res_sum_tagged(a, sh, st, epoch, v, &cancel);
      }
    }
    if (lane == 0) {
      sh.total = sum;
      sh.cancel = cancel;
    }
  } else {
    hidden();
  }
  __syncthreads();
  *total = sh.total;
  return sh.bad == 0;
}

// One thread's cached view of a row pattern (and, for RES_CLASS, its values):
// neighbouring rows mostly share it, so it is reloaded only when the code
// changes.  `at` are byte offsets, so that a row's loads are one address
// register each plus a constant.
template <int SRC, int STAGE>
struct ResRow {
  int code = -1, len = 0;
  int at[STAGE];
  double val[SRC == RES_CLASS ? STAGE : 1];
};

template <int SRC, int STAGE>
__device__ __forceinline__ void res_row_load(ResRow<SRC, STAGE> & w, int code,
    const unsigned char * table) {
  w.code = code;
  if constexpr (SRC == RES_CLASS) {
    const ResRowClass * c = reinterpret_cast<const ResRowClass *>(table) + code;
#pragma unroll
    for (int j = 0; j < STAGE; ++j) {
      w.at[j] = 8 * c->off[j];
      w.val[j] = c->val[j];
    }
    w.len = c->off[kPatMax - 1];
  } else {
    const int32_t * c = reinterpret_cast<const int32_t *>(table) + code * kPatMax;
#pragma unroll
    for (int j = 0; j < STAGE; ++j) w.at[j] = 8 * c[j];
    w.len = c[kPatMax - 1];
  }
}

// (A v)[i] for local row i of the pattern in `w`; v(o) is the vector at byte
// offset o from row i.  Products summed in CSR order with unfused multiply and
// add, as the reference does.  Shorter rows are padded with zero values at the
// row's own column (which leaves every finite sum as it is), so that rows of
// different patterns run the same code.  `vals`: the row's first value in
// shared memory (slot-major).
template <int SRC, int STAGE, class V>
__device__ __forceinline__ double res_row_sum(const ResArgs & a, const ResRow<SRC, STAGE> & w,
    uint32_t row, const unsigned char * table, const unsigned char * vals, V && v) {
  double sum = 0.0;
  if constexpr (SRC == RES_CSR) {
    const uint32_t e = __ldg(a.rowptr + row + 1);
    for (uint32_t k = __ldg(a.rowptr + row); k < e; ++k)
      sum = add_rn(sum, mul_rn(__ldg(a.val64 + k),
          v(8 * static_cast<int>(__ldg(a.rowind + k) - row))));
  } else if constexpr (SRC == RES_CLASS) {
#pragma unroll
    for (int j = 0; j < STAGE; ++j)
      sum = add_rn(sum, mul_rn(w.val[j], v(w.at[j])));
  } else if constexpr (SRC == RES_SMEM_F64) {
#pragma unroll
    for (int j = 0; j < STAGE; ++j)
      sum = add_rn(sum, mul_rn(*reinterpret_cast<const double *>(vals + 8 * j * a.rows), v(w.at[j])));
  } else if constexpr (SRC == RES_SMEM_F32) {
#pragma unroll
    for (int j = 0; j < STAGE; ++j)
      sum = add_rn(sum, mul_rn(static_cast<double>(
                              *reinterpret_cast<const float *>(vals + 4 * j * a.rows)), v(w.at[j])));
  } else if constexpr (SRC == RES_CODES) {
    const uint2 c = __ldg(reinterpret_cast<const uint2 *>(a.vals) + row);
    const double * t = reinterpret_cast<const double *>(table + a.ncode * kPatMax * 4);
#pragma unroll
    for (int j = 0; j < STAGE; ++j)
      if (j < w.len)
        sum = add_rn(sum, mul_rn(t[((j < 4 ? c.x : c.y) >> (8 * (j & 3))) & 0xffu],
            v(w.at[j])));
  } else if constexpr (SRC == RES_GLOBAL_F64) {
    constexpr int W = STAGE <= 5 ? 6 : 8;  // the solver's row width (cg.cu)
    const double2 * s = reinterpret_cast<const double2 *>(a.vals) +
                        static_cast<size_t>(W / 2) * row;
    double2 q[(STAGE + 1) / 2];
#pragma unroll
    for (int j = 0; j < (STAGE + 1) / 2; ++j) q[j] = __ldg(s + j);
#pragma unroll
    for (int j = 0; j < STAGE; ++j)
      sum = add_rn(sum, mul_rn((j & 1) ? q[j / 2].y : q[j / 2].x, v(w.at[j])));
  } else {
    const float4 * s = reinterpret_cast<const float4 *>(a.vals) + static_cast<size_t>(2) * row;
    const float4 q0 = __ldg(s), q1 = __ldg(s + 1);
    const float f[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
    for (int j = 0; j < STAGE; ++j)
      sum = add_rn(sum, mul_rn(static_cast<double>(f[j]), v(w.at[j])));
  }
  return sum;
}

// x += alpha p over rows first, first + step, ...
__device__ __forceinline__ void res_x_update(double * x, const double * p, double alpha,
    uint32_t first, uint32_t n, uint32_t step) {
  constexpr uint32_t U = 5;
  for (uint32_t i0 = first; i0 < n; i0 += U * step) {
    double xv[U], pv[U];
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t i = i0 + u * step;
      xv[u] = i < n ? x[i] : 0.0;
      pv[u] = i < n ? p[i] : 0.0;
    }
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t i = i0 + u * step;
      if (i < n) x[i] = fma(alpha, pv[u], xv[u]);
    }
  }
}

template <int SRC, int STAGE, int K, int T>
__global__ void __launch_bounds__(T, 1) cg_resident_kernel(const ResArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ ResShared sh;
  const ResLayout L(a.rows, a.halo, T, a.at, res_val_bytes(SRC, STAGE),
      res_table_bytes(SRC, a.ncode, a.ntable));
  double * const pw = reinterpret_cast<double *>(smem + L.p);
  const unsigned char * const table = smem + L.table;
  uint8_t * const codes = smem + L.codes;
  uint32_t lo = blockIdx.x * a.rows;
  uint32_t nloc = min(a.rows, a.n - lo);
  uint32_t H = a.halo;
  uint32_t tid = threadIdx.x;
  double * const po = pw + a.halo;  // p of the own rows
  double * const aps = reinterpret_cast<double *>(smem + L.ap);
  double * const xs = reinterpret_cast<double *>(smem + L.x);  // with a.at.x
  double * const rh = reinterpret_cast<double *>(smem + L.halo);
  // Bounds and indexes of the unrolled row loops are cheap to form again;
  // hoisted out of the solve's loop they would take the registers that hold r.
  const auto reform = [&] { asm volatile("" : "+r"(lo), "+r"(nloc), "+r"(H), "+r"(tid)); };

  // ---- the CTA's matrix rows; x = 0, r = b, p = 0, or where the last launch ended ----
  if constexpr (SRC != RES_CSR) {
    unsigned char * const t = smem + L.table;
    const uint32_t tw = static_cast<uint32_t>(
        (SRC == RES_CLASS ? a.ncode * sizeof(ResRowClass) : a.ncode * kPatMax * 4) / 4);
    const uint32_t * src = SRC == RES_CLASS ? reinterpret_cast<const uint32_t *>(a.classes)
                                            : reinterpret_cast<const uint32_t *>(a.pat_off);
    for (uint32_t i = tid; i < tw; i += T) reinterpret_cast<uint32_t *>(t)[i] = src[i];
    if constexpr (SRC == RES_CODES)
      for (uint32_t i = tid; i < a.ntable; i += T)
        reinterpret_cast<double *>(t + a.ncode * kPatMax * 4)[i] = a.table[i];
    for (uint32_t i = tid; i < nloc; i += T) codes[i] = a.row_code[lo + i];
    if constexpr (SRC == RES_SMEM_F64 || SRC == RES_SMEM_F32) {
      using V = typename std::conditional<SRC == RES_SMEM_F64, double, float>::type;
      V * s = reinterpret_cast<V *>(smem + L.vals);
      if (a.vals) {  // rows of val_width values
        const V * g = reinterpret_cast<const V *>(a.vals) + static_cast<size_t>(a.val_width) * lo;
        const uint32_t m = nloc * a.val_width;
        for (uint32_t i = tid; i < m; i += T) {
          const uint32_t row = i / a.val_width, j = i - row * a.val_width;
          if (j < STAGE) s[j * a.rows + row] = g[i];
        }
      } else {  // the CSR array
        for (uint32_t i = tid; i < nloc; i += T) {
          const uint32_t b = a.rowptr[lo + i], e = a.rowptr[lo + i + 1];
#pragma unroll
          for (int j = 0; j < STAGE; ++j)
            s[j * a.rows + i] = b + j < e ? static_cast<V>(a.val64[b + j]) : V(0);
        }
      }
    }
  }
  if (blockIdx.x == 0 && tid == 0) a.out->t0 = res_ns();
  if (tid == 0) {
    sh.bad = 0;
    sh.cancel = 0;
    sh.cancel_req = blockIdx.x == 0 ? (*reinterpret_cast<const volatile int *>(a.cancel) != 0) : 0;
  }
  uint32_t epoch = a.epoch0 + 1;  // numbers the published r values
  ResSums sums{0, 0, 0, 0};
  if (tid < 3 && a.ctas > 1) {  // before this CTA's first message: nobody adds until all have sent
    sums.seen0 = *reinterpret_cast<volatile unsigned long long *>(a.words + tid);
    sums.seen1 = *reinterpret_cast<volatile unsigned long long *>(a.words + 16 + tid);
  }
  double r[K];
  double acc = 0.0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const uint32_t i = k * T + tid;
    r[k] = 0.0;
    if (k * T < nloc) aps[i] = 0.0;  // rows past the block's end keep r = Ap = 0
    if (i < nloc) {
      r[k] = a.resume ? a.r_save[lo + i] : a.b[lo + i];
      if (a.at.x) xs[i] = a.resume ? a.x[lo + i] : 0.0;
      else if (!a.resume) a.x[lo + i] = 0.0;
      acc = fma(r[k], r[k], acc);
    }
  }
  for (uint32_t i = tid; i < nloc + 2 * H; i += T) {
    const uint32_t g = lo - H + i;  // wraps to >= n outside the matrix
    pw[i] = a.resume && g < a.n ? a.p_save[g] : 0.0;
  }

  // ---- the neighbours' r ----
  // Halo entry j: the H rows below the block, then the H rows above it.  With
  // room for them in shared memory warps 1.. fetch them while warp 0 waits for
  // the sum; else all warps fetch them after it.  put(j, r of entry j) is
  // called for every entry that lies in the matrix.
  constexpr uint32_t kHidden = T - 32;
  const uint32_t nh = a.ctas > 1 ? 2 * H : 0;
  const auto halo_win = [&](uint32_t j) -> uint32_t { return j < H ? j : nloc + j; };
  const auto halo_fetch = [&](uint32_t first, uint32_t step, auto && put) {
    constexpr int U = 5;  // loads in flight per thread
    for (uint32_t j0 = first; j0 < nh; j0 += U * step) {
      ulonglong2 m[U];
      const auto row_of = [&](uint32_t j) -> uint32_t {  // wraps to >= n outside the matrix
        return j < H ? lo - H + j : lo + nloc + (j - H);
      };
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t j = j0 + u * step, g = row_of(j);
        if (j < nh && g < a.n) m[u] = tagged_load(a.r_edge + g);
      }
      unsigned long long t0 = 0;
      unsigned polls = 0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t j = j0 + u * step, g = row_of(j);
        if (j < nh && g < a.n) {
          while (!tag_is(m[u], epoch)) {
            if (res_give_up(a, ++polls, &t0)) {
              sh.bad = 1;
              break;
            }
            m[u] = tagged_load(a.r_edge + g);
          }
          put(j, tagged_value(m[u]));
        }
      }
    }
  };
  // the own r values that neighbours read
  const auto publish = [&] {
    if (nh == 0) return;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const uint32_t i0 = k * T, i = i0 + tid;
      if ((i0 < H || i0 + T + H > nloc) && i < nloc && (i < H || i + H >= nloc))
        tagged_store(a.r_edge + lo + i, r[k], epoch);
    }
  };
  const auto prefetch_halo = [&] {
    if (a.at.halo) halo_fetch(tid - 32, kHidden, [&](uint32_t j, double v) { rh[j] = v; });
  };
  if (a.at.halo)  // entries outside the matrix stay 0
    for (uint32_t j = tid; j < nh; j += T) rh[j] = 0.0;

  double rr = 0.0, beta = 0.0, pap = 0.0;
  bool ok = res_allreduce<T>(a, sh, sums, epoch, acc, 0.0, [&] {
    publish();
    prefetch_halo();
  }, publish, &rr);
  if (a.resume) {
    rr = a.rr0;
    pap = a.pap0;
    beta = a.beta0;
  }
  if (tid == 0) {
    sh.bnorm = a.resume ? a.bnorm0 : sqrt(rr);
    const double tol = a.tol_relative ? a.tol * sh.bnorm : a.tol;
    sh.tol = tol;
    // r.r above this means ||r|| > tol without taking the root (infinite where
    // the square of tol is not accurate: then the root decides every time)
    sh.rr_far = tol > 1e-140 ? tol * tol * (1.0 + 1e-14) : INFINITY;
  }
  __syncthreads();
  unsigned long long it = a.resume ? a.it0 : 0;
  unsigned long long t_a = 0, t_b = 0;  // ns in A and B (a.timed)
  int status = GB_CG_MAXITER;
  bool running = ok;
  if (rr == 0.0) {
    status = GB_CG_CONVERGED;
    running = false;
  } else if (!(rr == rr) || isinf(rr)) {
    status = GB_CG_NONFINITE;
    running = false;
  }
  while (running) {
    // ---- A ----
    if (a.timed && tid == 0) t_a -= res_ns();
    reform();
    if (a.at.halo) {
      for (uint32_t j = tid; j < nh; j += T) {
        const uint32_t win = halo_win(j);
        pw[win] = fma(beta, pw[win], rh[j]);
      }
    } else {
      __syncthreads();  // all have read sh.bad
      halo_fetch(tid, T, [&](uint32_t j, double v) {
        const uint32_t win = halo_win(j);
        pw[win] = fma(beta, pw[win], v);
      });
    }
    {
      constexpr int U = K < 7 ? K : 7;  // loads in flight
#pragma unroll
      for (int k0 = 0; k0 < K; k0 += U) {
        double t[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const uint32_t i = (k0 + u) * T + tid;
          t[u] = k0 + u < K && i < nloc ? po[i] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const uint32_t i = (k0 + u) * T + tid;
          if (k0 + u < K && i < nloc) po[i] = fma(beta, t[u], r[k0 + u < K ? k0 + u : 0]);
        }
      }
    }
    __syncthreads();
    reform();
    acc = 0.0;
    {
      // R rows at a time, each with its own cached pattern, so that their
      // loads and sums interleave
      constexpr int R = K <= 1 ? 1 : 2;
      ResRow<SRC, STAGE> w[R];
      constexpr uint32_t kVal = SRC == RES_SMEM_F32 ? 4 : 8;
      const auto row = [&](const ResRow<SRC, STAGE> & wr, uint32_t i) {
        const char * const pi = reinterpret_cast<const char *>(po + i);
        return res_row_sum<SRC, STAGE>(a, wr, lo + i, table, smem + L.vals + kVal * i,
            [&](int o) { return *reinterpret_cast<const double *>(pi + o); });
      };
      const auto want = [&](ResRow<SRC, STAGE> & wr, int c) {
        if (SRC != RES_CSR && c != wr.code) res_row_load<SRC, STAGE>(wr, c, table);
      };
#pragma unroll 1
      for (uint32_t i = tid; i < nloc; i += R * T) {
        if (i + (R - 1) * T < nloc) {
          int c[R];
          double v[R], pv[R];
#pragma unroll
          for (int u = 0; u < R; ++u) c[u] = SRC == RES_CSR ? 0 : codes[i + u * T];
#pragma unroll
          for (int u = 0; u < R; ++u) want(w[u], c[u]);
#pragma unroll
          for (int u = 0; u < R; ++u) pv[u] = po[i + u * T];
#pragma unroll
          for (int u = 0; u < R; ++u) v[u] = row(w[u], i + u * T);
#pragma unroll
          for (int u = 0; u < R; ++u) {
            aps[i + u * T] = v[u];
            acc = fma(pv[u], v[u], acc);
          }
        } else {
#pragma unroll 1
          for (uint32_t q = i; q < nloc; q += T) {
            want(w[0], SRC == RES_CSR ? 0 : codes[q]);
            const double v = row(w[0], q);
            aps[q] = v;
            acc = fma(po[q], v, acc);
          }
        }
      }
    }
    if (!res_allreduce<T>(a, sh, sums, ++epoch, acc, pap, [] {}, [] {}, &pap)) {
      ok = false;
      break;
    }
    if (sh.cancel) {  // before x moves, so x matches `it`
      status = GB_CG_CANCELLED;
      break;
    }
    if (!(pap > 0.0)) {
      status = (pap == pap && rr == rr) ? GB_CG_BREAKDOWN : GB_CG_NONFINITE;
      break;
    }
    if (a.timed && tid == 0) {
      const unsigned long long t = res_ns();
      t_a += t;
      t_b -= t;
    }
    const double alpha = rr / pap;
    // ---- B ----
    reform();
    ++epoch;
    acc = 0.0;
    {
      double acc2 = 0.0;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const double v = k * T < nloc ? aps[k * T + tid] : 0.0;
        r[k] = fma(-alpha, v, r[k]);
        if (k & 1) acc2 = fma(r[k], r[k], acc2);
        else acc = fma(r[k], r[k], acc);
      }
      acc += acc2;
    }
    double rr_new;
    if (!res_allreduce<T>(a, sh, sums, epoch, acc, rr, [&] {
          publish();
          if (a.at.x) res_x_update(xs, po, alpha, tid - 32, nloc, kHidden);
          else res_x_update(a.x + lo, po, alpha, tid - 32, nloc, kHidden);
          prefetch_halo();
          // the host's flag costs a trip over PCIe, so it is read now and then
          if (blockIdx.x == 0 && tid == T - 1 && (it & 63) == 0) {
            if (it && a.late_ns) res_be_late(a.late_ns);
            sh.cancel_req = *reinterpret_cast<const volatile int *>(a.cancel) != 0;
          }
        }, publish, &rr_new)) {
      ok = false;
      break;
    }
    ++it;
    if (a.timed && tid == 0) t_b += res_ns();
    if (!(rr_new > sh.rr_far && rr_new < INFINITY) || (a.niter && it >= a.niter)) {
      const double rnorm = sqrt(rr_new);
      running = false;
      if (!(rnorm == rnorm) || isinf(rnorm)) status = GB_CG_NONFINITE;
      else if (rnorm <= sh.tol) status = GB_CG_CONVERGED;
      else if (a.niter && it >= a.niter) status = GB_CG_MAXITER;
      else running = true;
      if (!running && blockIdx.x == 0 && tid == 0) {
        // here, not behind the loop: alive there, they cost 1-3% of every iteration
        a.out->pap = pap;
        a.out->beta = rr_new / rr;
      }
    }
    if (a.hist && blockIdx.x == 0 && tid == T - 1 && it <= a.hist_len)
      a.hist[it - 1] = sqrt(rr_new);
    beta = rr_new / rr;
    rr = rr_new;
  }
  __syncthreads();
  const bool more = a.more && status == GB_CG_MAXITER;
  if (ok && more) {
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (k * T + tid < nloc) a.r_save[lo + k * T + tid] = r[k];
    for (uint32_t i = tid; i < nloc; i += T) a.p_save[lo + i] = po[i];
  }
  if (ok && a.at.x)
    for (uint32_t i = tid; i < nloc; i += T) a.x[lo + i] = xs[i];
  if (blockIdx.x == 0 && tid == 0) {
    a.out->status = more ? kResPaused : status;
    a.out->iter = it;
    a.out->rr = rr;
    a.out->bnorm = sh.bnorm;
    a.out->ran = it - (a.resume ? a.it0 : 0);
    a.out->t1 = res_ns();
    a.out->epoch = epoch;
    a.out->ns_a = t_a;
    a.out->ns_b = t_b;
  }
  // any CTA that gave up marks the solve
  if ((!ok || sh.bad) && tid == 0) a.out->aborted = 1;
  if (a.arrived) {  // every CTA's part of x and of the result, then `done`
    __threadfence_system();
    __syncthreads();
    if (tid == 0 && atomicAdd(a.arrived, 1u) + 1 == gridDim.x) {
      a.out->t1 = res_ns();
      __threadfence_system();
      *reinterpret_cast<volatile int *>(&a.out->done) = 1;
    }
  }
}

using ResKernel = void (*)(ResArgs);

// The form for `k` rows a thread at `threads` threads.
template <int SRC, int STAGE>
ResKernel res_kernel_k(int threads, int k) {
  if (threads == kResThreadsWide)
    return cg_resident_kernel<SRC, STAGE, kResRowsWide, kResThreadsWide>;
  return k <= 1 ? cg_resident_kernel<SRC, STAGE, 1, kResThreads>
         : k <= 4 ? cg_resident_kernel<SRC, STAGE, 4, kResThreads>
                  : cg_resident_kernel<SRC, STAGE, kResRows, kResThreads>;
}

template <int STAGE>
ResKernel res_kernel_s(int src, int threads, int k) {
  switch (src) {
    case RES_CLASS: return res_kernel_k<RES_CLASS, STAGE>(threads, k);
    case RES_SMEM_F64: return res_kernel_k<RES_SMEM_F64, STAGE>(threads, k);
    case RES_SMEM_F32: return res_kernel_k<RES_SMEM_F32, STAGE>(threads, k);
    case RES_GLOBAL_F64: return res_kernel_k<RES_GLOBAL_F64, STAGE>(threads, k);
    case RES_GLOBAL_F32: return res_kernel_k<RES_GLOBAL_F32, STAGE>(threads, k);
    case RES_CODES: return res_kernel_k<RES_CODES, STAGE>(threads, k);
    default: return res_kernel_k<RES_CSR, STAGE>(threads, k);
  }
}

// ---- co-residency of several solves -------------------------------------------
//
// A resident grid's CTAs wait for one another, so all of them must get an SM.
// Solves of one process on one device share its SMs through this count: a
// solve holds as many units as it has CTAs and waits while they are not free.
// A holder that nobody waits for on the host (the solve server's) names the
// word in which its kernel reports its end: whoever needs SMs takes those of
// ended holders back, so nobody depends on the holder's owner to look.
struct ResGate {
  struct Held {
    unsigned long long id;
    unsigned units;
    const int * done;  // may be null
  };
  struct Device {
    unsigned used = 0;
    std::vector<Held> held;
    unsigned long long next = 0, serving = 0;  // first come, first served
  };
  std::mutex mu;
  std::condition_variable cv;
  std::map<int, Device> devices;
  unsigned long long last_id = 0;
};
ResGate & gate() {
  static ResGate g;
  return g;
}

// Drop holders that `gone` names.  The gate is locked.
template <class F>
void gate_drop(ResGate & g, ResGate::Device & d, F && gone) {
  for (size_t k = 0; k < d.held.size();)
    if (gone(d.held[k])) {
      d.used -= d.held[k].units;
      d.held.erase(d.held.begin() + k);
      g.cv.notify_all();
    } else {
      ++k;
    }
}

// A holder's id if its units are free now, else 0.  The gate is locked.
unsigned long long gate_take(ResGate & g, ResGate::Device & d, unsigned units, unsigned capacity,
    const int * done) {
  gate_drop(g, d, [](const ResGate::Held & h) {
    return h.done && __atomic_load_n(h.done, __ATOMIC_ACQUIRE);
  });
  units = std::min(units, capacity);
  if (d.used + units > capacity) return 0;
  d.held.push_back({++g.last_id, units, done});
  d.used += units;
  return g.last_id;
}

}  // namespace

unsigned long long resident_acquire(int device, unsigned ctas, unsigned capacity,
    const int * cancel, unsigned long long limit_ns, bool * cancelled) {
  ResGate & g = gate();
  std::unique_lock<std::mutex> lk(g.mu);
  ResGate::Device & d = g.devices[device];
  const unsigned long long mine = d.next++;
  *cancelled = false;
  std::chrono::steady_clock::time_point since{};
  unsigned long long id = 0;
  for (;;) {
    if (d.serving == mine) {
      if ((id = gate_take(g, d, ctas, capacity, nullptr)) != 0) break;
      // a wait that is given up still takes its turn, so that the queue moves on
      if (cancel && __atomic_load_n(cancel, __ATOMIC_ACQUIRE)) {
        *cancelled = true;
        break;
      }
      const auto now = std::chrono::steady_clock::now();
      if (since.time_since_epoch().count() == 0) since = now;
      if (static_cast<unsigned long long>(
              std::chrono::duration_cast<std::chrono::nanoseconds>(now - since).count()) >
          limit_ns)
        break;
    }
    g.cv.wait_for(lk, std::chrono::microseconds(200));  // an ended kernel notifies nobody
  }
  ++d.serving;
  g.cv.notify_all();
  return id;
}

unsigned long long resident_try_acquire(int device, unsigned ctas, unsigned capacity,
    const int * done) {
  ResGate & g = gate();
  std::lock_guard<std::mutex> lk(g.mu);
  ResGate::Device & d = g.devices[device];
  return d.next != d.serving ? 0 : gate_take(g, d, ctas, capacity, done);
}

void resident_release(int device, unsigned long long id) {
  ResGate & g = gate();
  std::lock_guard<std::mutex> lk(g.mu);
  gate_drop(g, g.devices[device], [&](const ResGate::Held & h) { return h.id == id; });
}

struct ResidentCg {
  const gb_csr * a = nullptr;
  ResArgs args{};
  ResKernel fn = nullptr;
  size_t smem = 0;
  int threads = 0;
  unsigned capacity = 0;     // SMs
  ulonglong2 * r_edge = nullptr;
  unsigned long long * words = nullptr;  // [32]
  ulonglong2 * box = nullptr;
  size_t box_bytes = 0;      // the tagged partials and, behind them, the abort flag
  double * save = nullptr;   // [2][n] r and p of a solve between two launches
  ResResult * out_h = nullptr;
  ResResult * out_d = nullptr;
  RowClasses classes;
  uint32_t epoch = 0;        // all-reduces so far; 0: tags have to be cleared
  int fault = GB_CHIP_FAULT_NONE;  // for tests
};

// The grid of a solve (a test's missing CTA is the last one: the others wait for
// its part of the sums and for its edge values).
static unsigned resident_grid(const ResArgs & g, int fault) {
  return g.ctas - (fault == GB_CHIP_FAULT_MISSING && g.ctas > 1 ? 1u : 0u);
}

void resident_destroy(ResidentCg * s) {
  if (!s) return;
  dev_free(s->r_edge);
  dev_free(s->words);
  dev_free(s->box);
  dev_free(s->save);
  pinned_slot_free(s->out_h);
  free_row_classes(s->classes);
  delete s;
}

int resident_shape(uint32_t n, uint32_t half, int max_row, uint32_t npat, int sms, uint32_t want,
    ResShape * out) {
  *out = ResShape{};
  int dev = 0, max_smem = 0;
  GB_CUDA_TRY(cudaGetDevice(&dev));
  GB_CUDA_TRY(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  if (n == 0 || max_row < 1 || max_row > 7 || npat == 0 || npat > 256) return GOOSEBERRY_SUCCESS;
  const uint32_t cap = static_cast<uint32_t>(std::min(sms, kResMaxCtas));
  const int stage = max_row <= 5 ? 5 : 7;
  const size_t room = static_cast<size_t>(max_smem) - 1024;
  for (uint32_t rows = want; rows >= 512; rows /= 2) {
    const uint32_t parts = (n + rows - 1) / rows;  // equal parts of at most `rows`
    const uint32_t r = ((n + parts - 1) / parts + 1) / 2 * 2, ctas = (n + r - 1) / r;
    if (ctas > cap || r > kResThreads * kResRows) break;
    const uint32_t halo = ctas > 1 ? std::min(half, n) : 0;
    const auto need = [&](ResPlaces at) {
      return ResLayout(r, halo, kResThreads, at, res_val_bytes(RES_SMEM_F64, stage),
          res_table_bytes(RES_SMEM_F64, npat, 0)).total;
    };
    if (need(ResPlaces{1, 0}) > room) continue;
    out->args.n = n;
    out->args.rows = r;
    out->args.halo = halo;
    out->args.ctas = ctas;
    out->args.ncode = npat;
    resident_set_waits(&out->args, GB_CHIP_FAULT_NONE, 0);
    out->args.at = ResPlaces{1, ctas > 1 && need(ResPlaces{1, 1}) <= room ? 1 : 0};
    out->smem = need(out->args.at);
    out->threads = kResThreads;
    const int k = static_cast<int>((r + kResThreads - 1) / kResThreads);
    const ResKernel fn = stage == 5 ? res_kernel_s<5>(RES_SMEM_F64, kResThreads, k)
                                    : res_kernel_s<7>(RES_SMEM_F64, kResThreads, k);
    out->fn = reinterpret_cast<const void *>(fn);
    GB_TRY(raise_smem_limit(out->fn, out->smem));
    return GOOSEBERRY_SUCCESS;
  }
  return GOOSEBERRY_SUCCESS;
}

int resident_preload() {
  cudaFuncAttributes at;
  for (int k : {1, 4, kResRows}) {
    GB_CUDA_TRY(cudaFuncGetAttributes(&at,
        reinterpret_cast<const void *>(res_kernel_s<5>(RES_SMEM_F64, kResThreads, k))));
    GB_CUDA_TRY(cudaFuncGetAttributes(&at,
        reinterpret_cast<const void *>(res_kernel_s<7>(RES_SMEM_F64, kResThreads, k))));
  }
  return GOOSEBERRY_SUCCESS;
}

// A cooperative launch that the driver turns down (the SMs that this process may
// use do not hold the grid) leaves the device as it was.
static cudaError_t resident_start(const void * fn, int threads, size_t smem, ResArgs * args,
    int fault, cudaStream_t stream, bool * refused) {
  void * kargs[] = {args};
  cudaError_t e = fault == GB_CHIP_FAULT_REFUSED
      ? cudaErrorCooperativeLaunchTooLarge
      : cudaLaunchCooperativeKernel(fn, dim3(resident_grid(*args, fault)), dim3(threads), kargs,
            smem, stream);
  *refused = e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources ||
             e == cudaErrorNotSupported || e == cudaErrorNotPermitted;
  if (*refused) {
    cudaGetLastError();
    e = cudaSuccess;
  }
  return e;
}

int resident_launch(const ResShape & sh, ResArgs args, cudaStream_t stream, bool * refused) {
  GB_CUDA_TRY(resident_start(sh.fn, sh.threads, sh.smem, &args, sh.fault, stream, refused));
  return GOOSEBERRY_SUCCESS;
}

bool resident_size_ok(const gb_csr & a) {
  return a.nrows > 0 && a.nrows <= static_cast<size_t>(std::min(a.sm_count, kResMaxCtas)) *
                                       kResThreadsWide * kResRowsWide;
}

int resident_create(const gb_csr & a, const ResidentIn & in, double * x, ResidentCg ** out) {
  *out = nullptr;
  if (!in.pat || !in.pat->code8 || a.nrows == 0 || !a.val64 || in.stage == 6)
    return GOOSEBERRY_SUCCESS;
  int dev = 0, coop = 0, max_smem = 0;
  GB_CUDA_TRY(cudaGetDevice(&dev));
  GB_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  GB_CUDA_TRY(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const unsigned sms = std::min<unsigned>(a.sm_count, kResMaxCtas);
  if (!coop || sms == 0) return GOOSEBERRY_SUCCESS;
  const uint32_t n = a.nrows;
  // Rows a CTA owns: all of a small system, else one per thread at least
  // (fewer CTAs make cheaper sums), else an even split over all SMs.
  uint32_t rows = std::max<uint32_t>((n + sms - 1) / sms, kResThreads);
  if (n <= kResOneCta) rows = n;
  rows = std::min((rows + 1) / 2 * 2, (n + 1) / 2 * 2);  // even: keeps the regions aligned
  if (rows > kResThreadsWide * kResRowsWide) return GOOSEBERRY_SUCCESS;
  const int threads = rows <= kResThreads * kResRows ? kResThreads : kResThreadsWide;
  const unsigned ctas = (n + rows - 1) / rows;
  // half bandwidth from the pattern table
  std::vector<int32_t> off(static_cast<size_t>(in.pat->npat) * kPatMax);
  GB_CUDA_TRY(cudaMemcpy(off.data(), in.pat->off, off.size() * 4, cudaMemcpyDeviceToHost));
  long long half = 0;
  for (size_t p = 0; p < in.pat->npat; ++p)
    for (int j = 0; j < off[p * kPatMax + kPatMax - 1]; ++j)
      half = std::max<long long>(half, std::llabs(static_cast<long long>(off[p * kPatMax + j])));
  const uint32_t halo = ctas > 1 ? static_cast<uint32_t>(std::min<long long>(half, n)) : 0;
  // The vectors have to fit whatever the matrix source (the rule may not
  // depend on it: a plain-entries solver gives the same iterates): p with its
  // halo and the largest table.  The 1 KiB is static shared memory.
  const size_t room = static_cast<size_t>(max_smem) - 1024;
  const int stage = in.stage;
  if (ResLayout(rows, halo, threads, ResPlaces{}, 0, 256 * sizeof(ResRowClass)).total > room)
    return GOOSEBERRY_SUCCESS;

  ResidentCg * s = new ResidentCg();
  int rc = GOOSEBERRY_SUCCESS;
  const auto fail = [&](int code) {
    resident_destroy(s);
    return code;
  };
  s->a = &a;
  s->capacity = sms;
  s->threads = threads;
  ResArgs & g = s->args;
  g.n = n;
  g.rows = rows;
  g.halo = halo;
  g.ctas = ctas;
  g.rowptr = a.rowptr;
  g.rowind = a.rowind;
  g.val64 = a.val64;
  g.row_code = in.pat->code8;
  g.pat_off = in.pat->off;
  g.ncode = in.pat->npat;
  g.x = x;
  resident_set_waits(&g, GB_CHIP_FAULT_NONE, 0);
  const int k = static_cast<int>((rows + threads - 1) / threads);
  int src = RES_CSR;
  if (!in.plain) {
    if (in.ell8) {
      if ((rc = build_row_classes(a, a.val64, &s->classes, nullptr)) != GOOSEBERRY_SUCCESS)
        return fail(rc);
      if (s->classes.code8) {
        src = RES_CLASS;
        g.row_code = s->classes.code8;
        g.classes = s->classes.rows;
        g.ncode = s->classes.count;
      } else {
        src = RES_CODES;
        g.vals = in.ell8;
        g.table = in.table;
        g.ntable = in.ntable;
      }
    } else if (in.ellv) {
      g.vals = in.ellv;
      g.val_width = in.ellv_width;
      const int sm_src = in.ellv_f32 ? RES_SMEM_F32 : RES_SMEM_F64;
      src = ResLayout(rows, halo, threads, ResPlaces{}, res_val_bytes(sm_src, stage),
                res_table_bytes(sm_src, g.ncode, 0)).total <= room
                ? sm_src
                : (in.ellv_f32 ? RES_GLOBAL_F32 : RES_GLOBAL_F64);
    }
  }
  const auto fits = [&](ResPlaces at) {
    const size_t need = ResLayout(rows, halo, threads, at, res_val_bytes(src, stage),
        res_table_bytes(src, g.ncode, g.ntable)).total;
    if (need > room) return false;
    g.at = at;
    s->smem = need;
    return true;
  };
  // x, then the neighbours' r as far as there is room
  fits(ResPlaces{0, 0});
  fits(ResPlaces{1, 0});
  if (ctas > 1) fits(ResPlaces{g.at.x, 1});
  s->fn = stage == 5 ? res_kernel_s<5>(src, threads, k) : res_kernel_s<7>(src, threads, k);
  if ((rc = raise_smem_limit(reinterpret_cast<const void *>(s->fn), s->smem)) !=
      GOOSEBERRY_SUCCESS)
    return fail(rc);
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, s->fn, threads, s->smem) !=
          cudaSuccess ||
      occ < 1)
    return fail(GOOSEBERRY_SUCCESS);
  s->box_bytes = 2 * static_cast<size_t>(ctas) * sizeof(ulonglong2);
  if ((rc = dev_alloc(&s->r_edge, static_cast<size_t>(n) * sizeof(ulonglong2))) !=
          GOOSEBERRY_SUCCESS ||
      (rc = dev_alloc(&s->words, 32 * sizeof(unsigned long long))) != GOOSEBERRY_SUCCESS ||
      (rc = dev_alloc(&s->box, s->box_bytes + 16)) != GOOSEBERRY_SUCCESS ||
      (rc = pinned_slot_alloc(sizeof(ResResult), reinterpret_cast<void **>(&s->out_h),
           reinterpret_cast<void **>(&s->out_d))) != GOOSEBERRY_SUCCESS)
    return fail(rc);
  g.r_edge = s->r_edge;
  g.words = s->words;
  g.box = s->box;
  g.abort_flag = reinterpret_cast<int *>(reinterpret_cast<char *>(s->box) + s->box_bytes);
  g.out = s->out_d;
  if (dev_alloc(&s->save, 2 * static_cast<size_t>(n) * sizeof(double)) == GOOSEBERRY_SUCCESS) {
    g.r_save = s->save;
    g.p_save = s->save + n;
  } else {
    cudaGetLastError();  // no memory to pause with: one launch
    s->save = nullptr;
  }
  *out = s;
  return GOOSEBERRY_SUCCESS;
}

void resident_slice(ResArgs * g, unsigned long long niter, int fault, double ns,
    const ResResult * last) {
  g->niter = niter;
  g->more = 0;
  if (!g->p_save) return;  // no memory to go on from: one launch
  // The first launch's iterations by the rows of a CTA, estimated long (3 us and
  // 0.8 to 1.6 ns a row, see above); the others' as long as the last one's.
  double n = ns / (4000.0 + 1.6 * g->rows);
  if (last)
    n = static_cast<double>(last->ran) * ns /
        std::max<double>(1.0, static_cast<double>(last->t1 - last->t0));
  const unsigned long long from = last ? last->iter : 0;
  const unsigned long long upto = from + (fault == GB_CHIP_FAULT_SHORT
      ? 64 : static_cast<unsigned long long>(std::max(n, 64.0)));
  if (!niter || upto < niter) {
    g->niter = upto;
    g->more = 1;
  }
  if (!last) return;
  g->resume = 1;
  g->it0 = last->iter;
  g->rr0 = last->rr;
  g->pap0 = last->pap;
  g->beta0 = last->beta;
  g->bnorm0 = last->bnorm;
}

void resident_set_waits(ResArgs * g, int fault, unsigned limit_ms) {
  g->wait_ns = limit_ms ? limit_ms * 1000000ull : kResWaitNs;
  g->late_ns = fault == GB_CHIP_FAULT_LATE ? 2 * g->wait_ns : 0;
}

bool resident_set_fault(ResidentCg * s, int fault, unsigned limit_ms) {
  if (fault != GB_CHIP_FAULT_NONE && s->args.ctas < 2) return false;
  s->fault = fault;
  resident_set_waits(&s->args, fault, limit_ms);
  return true;
}

int resident_solve(ResidentCg * s, const double * b, double tol, int tol_relative,
    unsigned long long niter, double * dhist, unsigned long long hist_len,
    const int * cancel_h, const int * cancel_d, bool timed, cudaStream_t stream,
    ResOutcome * res) {
  ResArgs g = s->args;
  g.timed = timed ? 1 : 0;
  g.b = b;
  g.tol = tol;
  g.tol_relative = tol_relative;
  g.niter = niter;
  g.hist = dhist;
  g.hist_len = hist_len;
  g.cancel = cancel_d;
  *res = ResOutcome{};
  do {
    if (!timed) resident_slice(&g, niter, s->fault, kResSliceNs,
                    res->launches ? &res->result : nullptr);
    // Tags of one launch must not meet those that earlier ones left in memory:
    // the count goes on from launch to launch, and starts over, with cleared
    // memory, before it could wrap (a tag is the count's low 31 bits).
    if (s->epoch == 0 || s->epoch > (1u << 29)) {
      GB_CUDA_TRY(cudaMemsetAsync(s->words, 0, 32 * sizeof(unsigned long long), stream));
      GB_CUDA_TRY(cudaMemsetAsync(s->box, 0, s->box_bytes + 16, stream));
      GB_CUDA_TRY(cudaMemsetAsync(s->r_edge, 0, static_cast<size_t>(g.n) * sizeof(ulonglong2),
          stream));
      s->epoch = 2;
    }
    g.epoch0 = s->epoch;
    unsigned long long held = 0;
    bool cancelled = false;
    if (g.ctas > 1 && !(held = resident_acquire(s->a->device, g.ctas, s->capacity, cancel_h,
                            g.wait_ns, &cancelled))) {
      if (!cancelled) res->result.aborted = 1;
      else if (g.resume) res->result.status = GB_CG_CANCELLED;  // x is that of the last launch
      else res->cancelled_waiting = true;
      return GOOSEBERRY_SUCCESS;
    }
    std::memset(s->out_h, 0, sizeof(ResResult));
    bool refused = false;
    cudaError_t e = resident_start(reinterpret_cast<const void *>(s->fn), s->threads, s->smem, &g,
        s->fault, stream, &refused);
    const cudaError_t e2 = cudaStreamSynchronize(stream);
    resident_release(s->a->device, held);
    if (e == cudaSuccess) e = e2;
    if (e != cudaSuccess) {
      s->epoch = 0;
      set_error("CG solve failed: %s", cudaGetErrorString(e));
      return GOOSEBERRY_ERROR_UNKNOWN;
    }
    if (refused) s->out_h->aborted = 1;  // nothing ran
    res->result = *s->out_h;
    ++res->launches;
    // an abandoned solve leaves the CTAs at different counts
    s->epoch = s->out_h->aborted ? 0 : s->out_h->epoch;
  } while (!res->result.aborted && res->result.status == kResPaused);
  return GOOSEBERRY_SUCCESS;
}

}  // namespace gb
