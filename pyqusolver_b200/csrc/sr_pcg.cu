// The whole SR solve as one persistent kernel: the force F, then every CG iteration, in one
// cooperative launch of at most one CTA per SM.
//
// A CTA owns R samples for the whole solve.  Their T = tanh(theta) stays in shared memory (float32),
// their spins stay in tensor memory as the A operands of both contractions (exact in BF16), and the
// CTA's slice of x, r and p stays in registers, so that an iteration moves only
//   z = Sigma V + v_b     A = [sigma_s | 1] from TMEM, B = V (BF16 hi/lo) streamed from L2
//   w_s = sum_m t_sm z_sm + sigma_s . v_a              (float32 epilogue), mean over the grid
//   Sigma^T Q, Q_sm = conj(t_sm) u_s                   A = Sigma^T from TMEM, B = Q built in shared
//                                                      memory from the resident T (BF16 hi/lo)
//   one partial P-vector per CTA, summed in float64 by the CTAs that own the entries.
// What bounds an iteration: the latency of its chain of steps and, from about 60 sites x 190 units on, the
// L2 traffic: V is read by every CTA and every CTA writes a whole partial (heis10x10: 26 + 24 + 24 MB).
// Clocks per iteration on CTA 0 (about 1.9 GHz), of the sections in order, for 16 sites x 16 units, 1,024 samples (32 CTAs)
// and for 63 x 189 complex, 5,000 samples (105 CTAs): direction exchange 2,600 / 4,300; first contraction with sigma . v_a
// 2,400 / 4,900; its epilogue 600 / 2,900; u 400 / 800; Q 1,200 / 4,000; g_a and the rest of the second contraction
// 1,200 / 1,700; partials out 600 / 6,700; their barrier 2,900 / 3,000; their sum 3,000 / 7,200; the dot products
// 3,100 / 8,500; vectors and the next operand 800 / 1,300.  The exchanges include the wait for the last CTA.
// Measured per CG iteration (250 against 50 iterations of a solve) against the chain of kernels (sr.cu, sr_tc.cu): 16 sites x 16
// units, 1,024 samples 17.9 -> 9.8 us; 63 x 126, 1,000 samples 24.5 -> 12.6; 6x6 x 144 complex, 8,192 samples
// 28.2 -> 17.7; 63 x 189 complex, 5,000 samples 30.7 -> 23.3; 10x10 x 200 complex, 16,384 samples 41.7 -> 33.6 us.
// The last one is the largest that fits: it takes all 512 TMEM columns (NZ + Kz / 2 + R / 2) and 232,344 bytes of
// shared memory.  Beyond it the chain runs: 208 units 42.4 us, 240 units 64, 18,944 samples 59, 11x11 x 242 units 91.
//
// Two exchanges of the textbook iteration are not needed:
//  * the mean of w = O p: O-bar . p is known before w is (O-bar once per solve, then the recurrences of r and
//    p), so u is centred by it, and what it leaves of the mean, summed from the w themselves, is taken
//    out of S p in float64;
//  * |r_k+1|^2 for beta: |r_k|^2 - 2 alpha r.Ap + alpha^2 |Ap|^2 with |r_k|^2 summed from the vector itself in
//    the same exchange, so nothing is carried over; where it would lose digits (a drop below 1e-6 in
//    one step) the vector is summed in one more exchange.
//
// Warps 0-15 compute; warp 16 carries the direction exchange and issues the bulk copies of V, warp 17 the
// MMAs.  Every wait is bounded: a wait that runs out sets *status or *err, every CTA leaves after the
// partials of a pass (or the sums after them) at the latest, and the host reports QES_ERR_TIMEOUT.  The warps meet
// at kBarAll before every iteration, which is where warps 16 and 17 learn of the end: a CTA that fails in pass -2
// therefore still builds pass -1's operand, which warp 17 waits for.  A compute warp arrives for an operand stage again
// only after warp 17 has met its last arrival: warp 17 waits for nothing but copies that are under way (kBarGo comes
// first) and gives up on all of an iteration's before a compute warp gives up on their products.
#include "common.cuh"
#include "sr_pcg.h"
#include "umma.cuh"

#include <algorithm>
#include <cmath>
#include <cuda_bf16.h>

namespace {

constexpr int kCompute = 512;                    // threads of the compute warps
constexpr int kThreadsP = kCompute + 64;         // + bulk-copy warp and MMA warp
constexpr uint32_t kWaitP = 1u << 22;            // try_wait polls of the compute warps before giving up
constexpr uint32_t kWaitOp = kWaitP >> 4;        // of warps 16 and 17, once per k-step: up to 8 in a row are over first
constexpr uint32_t kPollLimit = 1u << 22;        // slot polls before giving up
constexpr size_t kSmemMax = 227 * 1024;
constexpr unsigned long long kEmptySlot = ~0ull;  // a NaN pattern that no sum produces
constexpr int kBarLeft = 11, kBarGo = 12, kBarCompute = 13, kBarAll = 14;           // named barriers (1 .. S: operand stages)
constexpr int kMaxStages = 8;
constexpr int kVals = 6;                         // values of one grid-wide sum
constexpr int kDirect = 32;                      // CTAs that exchange without collectors; collectors and their senders
enum { X_DOTS = 0, X_RR = 1 };                   // sums
enum { X_PART = 0, X_DIR = 1 };                  // barriers

template <class T> struct PV;
template <> struct PV<float> { using type = double; };
template <> struct PV<float2> { using type = double2; };

__device__ __forceinline__ void bar_sync(int id, int n) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int n) {
  __syncwarp();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

__device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
  const float2 hf = __bfloat1622float2(h);
  const __nv_bfloat162 l = __floats2bfloat162_rn(x0 - hf.x, x1 - hf.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// TMEM stores of 8 columns per lane, and the MMA with A in TMEM
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void mma_bf16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 8 columns of one or two accumulator halves behind one wait
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
  uint32_t r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int q = 0; q < 8; ++q) v[q] = __uint_as_float(r[q]);
}
__device__ __forceinline__ void tmem_ld8x2(uint32_t ta, uint32_t tb, float (&v0)[8], float (&v1)[8]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(ta), "r"(tb)
      : "memory");
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    v0[q] = __uint_as_float(r[q]);
    v1[q] = __uint_as_float(r[8 + q]);
  }
}

// element (sample s, unit m) of the resident T: rows of Mh elements whose units are permuted by an xor
// with the row, so that both a column of 32 rows (O v epilogue) and a row of 32 units (Q) are read
// without bank conflicts
template <class T>
__device__ __forceinline__ int t_xor(int s, int Mh) {
  if constexpr (sizeof(T) == 8) return (Mh & 8) ? ((s >> 1) & 7) : (s & 15);
  else return (Mh & 16) ? ((s >> 1) & 15) : (s & 31);
}
template <class T>
__device__ __forceinline__ int t_index(int s, int m, int Mh) { return s * Mh + (m ^ t_xor<T>(s, Mh)); }

// Grid-wide sums go through mailboxes in two levels: a CTA pushes its values to its collector (one of
// nc), a collector adds its senders' values and pushes the subtotal into the box of every CTA, and each
// CTA adds the nc subtotals.  No line is polled by more than one SM: measured per exchange of one value
// on 148 CTAs, 3.5 us with one shared box that all CTAs poll and 1.8 us with every CTA pushing to
// every other; on up to kDirect CTAs the latter takes 0.55 us, one L2 store and load, and is used.
// Words hold a sentinel until they are written and are reset by their reader.
struct Exchange {
  double* box1;              // [type][parity][value][sender]: level 1, read by the sender's collector
  double* box2;              // [receiver][type][parity][value][kDirect]: subtotals
  unsigned int* count;       // barrier counters, one line each
  int G, nc, cta;
  uint32_t polls;            // of a wait before it gives up
  bool mute;                 // test hook: this CTA's value of the next sum is never sent
  int* err;
  int* s_fail;               // shared: written and read by the compute warps inside an exchange only
  const int* s_bad;          // shared: an operand wait gave up (any warp, any time)
  double* s_red;             // shared: [kVals][16] warp sums, [kVals] results
  __device__ __forceinline__ double* slot1(int type, int par, int val, int sender) const {
    return box1 + ((size_t)((type * 2 + par) * kVals + val)) * G + sender;
  }
  __device__ __forceinline__ double* slot2(int receiver, int type, int par, int val) const {
    return box2 + (((size_t)receiver * 2 + type) * 2 + par) * (kVals * kDirect) + val * kDirect;
  }
};

__device__ __forceinline__ void slot_put(double* p, double v) {
  unsigned long long u = (unsigned long long)__double_as_longlong(v);
  if (u == kEmptySlot) u = 0x7ff8000000000000ull;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(u) : "memory");
}
__device__ __forceinline__ void slot_clear(double* p) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(kEmptySlot) : "memory");
}
__device__ __forceinline__ bool slot_wait(const double* p, uint32_t polls, int* err, double& v) {
  for (uint32_t it = 0; it < polls; ++it) {
    unsigned long long u;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(u) : "l"(p) : "memory");
    if (u != kEmptySlot) {
      v = __longlong_as_double((long long)u);
      return true;
    }
    if ((it & 1023u) == 1023u && *(volatile int*)err != 0) break;
  }
  atomicCAS(err, 0, 1);
  return false;
}

// Warp sums of up to 8 values at once by halving: in each step a lane hands the half of its values that it
// does not keep to its partner, 9 exchanged doubles instead of 5 per value.  Lane l returns the sum of
// value (l >> 2) & 7.
template <int NV>
__device__ __forceinline__ double warp_sum_split(const double (&v)[NV], int lane) {
  double a[4], b[2], c;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const double lo = q < NV ? v[q < NV ? q : 0] : 0.0, hi = q + 4 < NV ? v[q + 4 < NV ? q + 4 : 0] : 0.0;
    const bool up = (lane & 16) != 0;
    a[q] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, 16);
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const bool up = (lane & 8) != 0;
    b[q] = (up ? a[q + 2] : a[q]) + __shfl_xor_sync(0xffffffffu, up ? a[q] : a[q + 2], 8);
  }
  {
    const bool up = (lane & 4) != 0;
    c = (up ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, up ? b[0] : b[1], 4);
  }
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  return c;
}

// grid-wide sums of NV values (each thread of the first n_warps compute warps passes its addends): all CTAs
// return the same sums, added in the same order.  No memory ordering beyond the values themselves.
template <int NV>
__device__ __forceinline__ bool exchange_sum(const Exchange& X, int type, int par, int n_warps, double (&v)[NV]) {
  static_assert(NV <= kVals, "");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp < n_warps) {
    const double t = warp_sum_split<NV>(v, lane);
    const int q = (lane >> 2) & 7;
    if ((lane & 3) == 0 && q < NV) X.s_red[16 * q + warp] = t;
  }
  bar_sync(kBarCompute, kCompute);
  if (tid == 0 && *(const volatile int*)X.s_bad != 0) *X.s_fail = 1;
  if (warp < NV) {                                          // warp q carries value q
    double t = warp_sum(lane < n_warps ? X.s_red[16 * warp + lane] : 0.0);
    bool good = true;
    const bool direct = X.G <= kDirect;
    if (!direct) {
      if (lane == 0 && !X.mute) slot_put(X.slot1(type, par, warp, X.cta), t);
      if (X.cta < X.nc) {                                   // senders cta, cta + nc, ...
        const int sender = X.cta + lane * X.nc;
        t = 0.0;
        if (sender < X.G) good = slot_wait(X.slot1(type, par, warp, sender), X.polls, X.err, t);
        t = warp_sum(t);
      }
    }
    if (direct ? !X.mute : X.cta < X.nc)
      for (int r = lane; r < X.G; r += 32) slot_put(X.slot2(r, type, par, warp) + X.cta, t);
    t = 0.0;
    if (lane < X.nc) good = slot_wait(X.slot2(X.cta, type, par, warp) + lane, X.polls, X.err, t) && good;
    t = warp_sum(t);
    if (!good) *X.s_fail = 1;
    if (lane == 0) X.s_red[16 * kVals + warp] = t;
  }
  bar_sync(kBarCompute, kCompute);
#pragma unroll
  for (int q = 0; q < NV; ++q) v[q] = X.s_red[16 * kVals + q];
  return *(volatile int*)X.s_fail == 0;
}
// this CTA's words of one finished exchange (read; nobody writes them before the next X_DIR)
__device__ __forceinline__ void exchange_reset(const Exchange& X, int type, int par) {
  const int tid = threadIdx.x;
  if (tid < kVals * kDirect) slot_clear(X.slot2(X.cta, type, par, 0) + tid);
  if (X.G > kDirect && X.cta < X.nc)
    for (int q = tid; q < kVals * 32; q += kCompute) {
      const int sender = X.cta + (q & 31) * X.nc;
      if (sender < X.G) slot_clear(X.slot1(type, par, q >> 5, sender));
    }
}

// Grid-wide barrier, one thread of each CTA after its CTA has synchronised: everything that the CTAs wrote
// to global memory before it is visible after it.  One counter that every CTA polls: 1.2 us on 148 CTAs,
// against 1.7 us with a separate release flag.
__device__ __forceinline__ bool grid_arrive_wait(unsigned int* c, unsigned int target, uint32_t polls, int* err) {
  unsigned int v;
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(c) : "memory");
  for (uint32_t it = 1;; ++it) {
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(c) : "memory");
    if ((int)(v - target) >= 0) return true;
    if (it >= polls || ((it & 1023u) == 0 && *(volatile int*)err != 0)) {
      atomicCAS(err, 0, 1);
      return false;
    }
  }
}
// extra: arrivals that never come (test hook)
__device__ __forceinline__ bool exchange_barrier(const Exchange& X, int which, unsigned int round, unsigned int extra) {
  bar_sync(kBarCompute, kCompute);
  if (threadIdx.x == 0) {
    if (*(const volatile int*)X.s_bad != 0) *X.s_fail = 1;
    if (!grid_arrive_wait(X.count + 32 * which, round * (unsigned int)X.G + extra, X.polls, X.err)) *X.s_fail = 1;
  }
  bar_sync(kBarCompute, kCompute);
  return *(volatile int*)X.s_fail == 0;
}

}  // namespace

template <class T>
__global__ void __launch_bounds__(kThreadsP, 1)
cg_persist_kernel(PcgDims d, int64_t n_samples, const uint32_t* __restrict__ bits, const T* __restrict__ tt,
                  const float2* __restrict__ eloc, const float* __restrict__ wts, double shift, double rtol,
                  double atol, int maxiter, double prefactor, double* __restrict__ x_nat, double* __restrict__ b_nat,
                  double* __restrict__ x_out, double* __restrict__ scal, float4* __restrict__ partial,
                  uint8_t* __restrict__ vz, float* __restrict__ va, double2* __restrict__ wres,
                  double* __restrict__ slots, unsigned int* __restrict__ counters,
                  int* __restrict__ status, int* __restrict__ err, PcgWaitTest hook) {
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr bool CPLX = ScalarTraits<T>::is_complex;
  constexpr int H = CPLX ? 2 : 1;
  const int ns = d.ns, nh = d.nh, Mh = d.Mh, NZ = d.NZ, Kz = d.Kz, R = d.R, S = d.S, G = d.G;
  const int nks = Kz / 16, nqs = R / 16, nw = n_words(ns);
  const uint32_t stage_bytes = (uint32_t)NZ * 64u;           // one k-step of a hi/lo operand pair
  const size_t t_bytes = ((size_t)R * Mh * sizeof(T) + 127) & ~(size_t)127;
  size_t region = (size_t)S * stage_bytes;
  if (region < 16384 + 128) region = 16384 + 128;
  T* sT = reinterpret_cast<T*>(smem);
  uint8_t* sB = smem + t_bytes;
  T* s_u = reinterpret_cast<T*>(sB + region);                // [R]
  double* s_red = reinterpret_cast<double*>(s_u + R);        // [17 kVals + 10]
  uint64_t* full = reinterpret_cast<uint64_t*>(s_red + 17 * kVals + 10);  // [S]
  uint64_t* empty = full + S;
  uint64_t* done = empty + S;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1);
  int* s_fail = reinterpret_cast<int*>(tslot + 1);
  int* s_stop = s_fail + 1;
  int* s_bad = s_fail + 2;
  float2* s_part = reinterpret_cast<float2*>(sB);            // [4][128], between the two contractions
  double* s_acc = reinterpret_cast<double*>(sB);             // [groups][vpc][4], reduction

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = blockIdx.x;
  const int64_t s0 = (int64_t)cta * R;
  if (tid == 0) {
    for (int q = 0; q < S; ++q) {
      umma::mbar_init(&full[q], 1);
      umma::mbar_init(&empty[q], 1);
    }
    umma::mbar_init(done, 1);
    umma::fence_mbar_init();
    *s_fail = 0;
    *s_stop = 0;
    *s_bad = 0;
  }
  if (warp == 17) {
    umma::tmem_alloc(tslot, d.tmem_cols);
    umma::tmem_relinquish();
  }
  // resident T (zero beyond the samples and the hidden units)
  for (int e = tid; e < R * Mh; e += kThreadsP) {
    const int s = e / Mh, m = e - s * Mh;
    sT[t_index<T>(s, m, Mh)] = (s0 + s < n_samples && m < nh) ? tt[(s0 + s) * nh + m] : ScalarTraits<T>::zero();
  }
  // the direction operand's padding (K rows past the ones column, units past nh) stays zero
  for (int64_t e = (int64_t)cta * kThreadsP + tid; e < (int64_t)nks * NZ * 4; e += (int64_t)G * kThreadsP)
    reinterpret_cast<uint4*>(vz)[e] = make_uint4(0u, 0u, 0u, 0u);
  asm volatile("fence.proxy.async;" ::: "memory");
  auto gave_up = [&]() {                                     // a bounded operand wait ran out
    atomicCAS(status, 0, QES_ERR_TIMEOUT);
    atomicCAS(err, 0, 1);
    *(volatile int*)s_bad = 1;
  };
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tbase = *tslot;
  const uint32_t col_as = tbase + NZ, col_at = col_as + Kz / 2;      // spins: samples x sites, sites x samples

  if (warp < 16) {
    // ------------------------------------------------------------------ compute warps
    const int quarter = warp & 3, cg = warp >> 2;
    const int row = 32 * quarter + lane;                     // sample (O v) or site (O^H u) of this lane
    const uint32_t lane_off = (uint32_t)(32 * quarter) << 16;
    const int64_t s = s0 + row;
    const bool sval = row < R && s < n_samples;
    // spins into TMEM: 16 K entries (8 columns) per store
    for (int blk = cg; blk < nks; blk += 4) {
      const uint32_t w = (sval && (blk >> 1) < nw) ? bits[s * nw + (blk >> 1)] >> (16 * (blk & 1)) : 0u;
      uint32_t r[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        uint32_t v = 0;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int k = 16 * blk + 2 * q + e;
          uint32_t x = 0;
          if (sval) x = k < ns ? (((w >> (2 * q + e)) & 1u) ? 0x3F80u : 0xBF80u) : (k == ns ? 0x3F80u : 0u);
          v |= x << (16 * e);
        }
        r[q] = v;
      }
      tmem_st8(col_as + lane_off + 8 * blk, r);
    }
    for (int blk = cg; blk < nqs; blk += 4) {
      uint32_t r[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        uint32_t v = 0;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int64_t sp = s0 + 16 * blk + 2 * q + e;
          uint32_t x = 0;
          if (sp < n_samples) {
            if (row < ns) x = ((bits[sp * nw + (row >> 5)] >> (row & 31)) & 1u) ? 0x3F80u : 0xBF80u;
            else if (row == 127) x = 0x3F80u;                // ones row: g_b
          }
          v |= x << (16 * e);
        }
        r[q] = v;
      }
      tmem_st8(col_at + lane_off + 8 * blk, r);
    }
    tmem_wait_st();
    umma::tc_fence_before();
    // spin word cg of the lane's sample (sigma . v_a), and the spins of site tid / 4 over the samples
    // 4 k + tid % 4 (g_a)
    const uint32_t sword = (sval && cg < nw) ? bits[s * nw + cg] : 0u;
    const int n_site = min(32, ns - 32 * cg);
    const int ga_site = tid >> 2, ga_grp = tid & 3;
    uint32_t ga_bits = 0;
    if (ga_site < ns)
      for (int k = 0; 4 * k + ga_grp < R; ++k) {
        const int64_t sp = s0 + 4 * k + ga_grp;
        if (sp < n_samples) ga_bits |= ((bits[sp * nw + (ga_site >> 5)] >> (ga_site & 31)) & 1u) << k;
      }
    const float wt = (sval && wts) ? wts[s] : 1.f;
    // owned entries of the parameter vector: 16-byte vectors [v0, v0 + nv), one scalar per thread
    const int64_t v0 = (int64_t)cta * d.vpc;
    const int nv = (int)max((int64_t)0, min((int64_t)d.vpc, d.nvec - v0));
    const int64_t n_mat = (int64_t)NZ * (ns + 1);
    const int own_warps = max(1, (4 * nv + 31) / 32);        // warps that own entries
    int64_t nat = -1;                                        // index in the natural order (in reals)
    uint32_t op_off = 0xffffffffu;                           // operand byte offset, or entry of va
    bool is_va = false;
    if (tid < 4 * nv) {
      const int64_t e = 4 * v0 + tid;
      if (e < n_mat) {
        const int cc = (int)(e / (16 * (ns + 1)));
        const int site = (int)((e >> 4) % (ns + 1)), col = cc * 16 + (int)(e & 15);
        const int h = (CPLX && col >= Mh) ? 1 : 0, m = col - h * Mh;
        if (m < nh) {
          nat = ((site < ns ? (int64_t)ns + nh + (int64_t)site * nh : (int64_t)ns) + m) * H + h;
          op_off = (uint32_t)(site >> 4) * stage_bytes + umma::kmajor_offset((uint32_t)col, (uint32_t)(site & 15), (uint32_t)NZ);
        }
      } else if (e - n_mat < (int64_t)ns * H) {
        nat = e - n_mat;
        op_off = (uint32_t)nat;
        is_va = true;
      }
    }
    const int sg = tid / d.vpc, vl = tid - sg * d.vpc;       // split group and vector of the reduction
    Exchange X{slots, slots + (size_t)2 * 2 * kVals * G, counters, G, d.nc, cta, hook.polls, false, err, s_fail, s_bad, s_red};
    const float fs = (float)(1.0 / (double)n_samples);
    const double inv_n = 1.0 / (double)n_samples;
    float4* part_mine = partial + (int64_t)cta * d.nvec;
    double xk = 0.0, rk = 0.0, pk = 0.0, rr = 0.0, thresh = 0.0, bb = 0.0;
    double ob = 0.0, ob2 = 0.0;                              // conj(O-bar): this entry's part and the other one
    double crr = 0.0, cri = 0.0, cpr = 0.0, cpi = 0.0;       // O-bar . r and O-bar . p: the expected mean of w
    int g = 0, iters = 0;                                    // operand stages used so far
    uint32_t dph = 0;
    bool ok = true, conv = false;
    // pass -2: O^H 1 (conj(O-bar)); pass -1: the force; then the iterations
    for (int it = -2;; ++it) {
      const int par = it & 1;
      X.mute = hook.which == PcgWaitTest::SUM && it == hook.pass && cta == 0;
      float2 w = make_float2(0.f, 0.f);
      if (it == -2) {
        if (warp < 4 && sval) w = make_float2(1.f, 0.f);
      } else if (it == -1) {
        if (warp < 4 && sval) w = eloc[s];
        // the energy mean is exchanged: nothing predicts it
        double m2[2] = {(double)wt * w.x, (double)wt * w.y};
        ok = exchange_sum<2>(X, X_RR, 1, 4, m2);
        cpr = m2[0] * inv_n;
        cpi = m2[1] * inv_n;
        if (cta == 0 && tid == 0) {
          scal[12] = cpr;
          scal[13] = cpi;
        }
      } else {
        // ---- w = O p: sigma . v_a while the MMAs run, then t . z
        bar_sync(kBarGo, kCompute + 64);                     // every CTA's operand entries are written
        float2 acc = make_float2(0.f, 0.f);
        if (cg < nw) {
          float vr = 0.f, vi = 0.f;
          if (lane < n_site) {
            if constexpr (CPLX) {
              const float2 q = __ldcg(reinterpret_cast<const float2*>(va) + 32 * cg + lane);
              vr = q.x;
              vi = q.y;
            } else {
              vr = __ldcg(va + 32 * cg + lane);
            }
          }
          float sre = 0.f, sim = 0.f;
#pragma unroll 8
          for (int i = 0; i < 32; ++i) {                     // lanes past the sites hold zero
            const int sgn = (int)((~sword >> i) & 1u) << 31;
            sre += __int_as_float(__float_as_int(__shfl_sync(0xffffffffu, vr, i)) ^ sgn);
            if constexpr (CPLX) sim += __int_as_float(__float_as_int(__shfl_sync(0xffffffffu, vi, i)) ^ sgn);
          }
          acc = make_float2(sre, sim);
        }
        g += nks;
        if (!umma::mbar_wait(done, dph, kWaitP)) gave_up();
        dph ^= 1u;
        umma::tc_fence_after();
        const T* trow = sT + (row < R ? row : 0) * Mh;
        const int tx = t_xor<T>(row, Mh);
        for (int c = cg; c < Mh / 8; c += 4) {
          float zr[8], zi[8];
          T t[8];
          const T* tc = trow + ((8 * c) ^ (tx & ~7));
#pragma unroll
          for (int q = 0; q < 8; ++q) t[q] = tc[q ^ (tx & 7)];
          __syncwarp();
          if constexpr (CPLX) tmem_ld8x2(tbase + lane_off + 8 * c, tbase + lane_off + Mh + 8 * c, zr, zi);
          else tmem_ld8(tbase + lane_off + 8 * c, zr);
          float ar = 0.f, ai = 0.f;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            if constexpr (CPLX) {
              ar = fmaf(t[q].x, zr[q], fmaf(-t[q].y, zi[q], ar));
              ai = fmaf(t[q].x, zi[q], fmaf(t[q].y, zr[q], ai));
            } else {
              ar = fmaf(t[q], zr[q], ar);
            }
          }
          acc.x += ar;
          acc.y += ai;
        }
        s_part[cg * 128 + row] = acc;
        umma::tc_fence_before();
        bar_sync(kBarCompute, kCompute);
        if (warp < 4 && sval) {
          w = s_part[row];
#pragma unroll
          for (int q = 1; q < 4; ++q) w = w + s_part[q * 128 + row];
        }
      }
      // ---- u = wts (w - c) / n, c the expected mean; what is left of the mean goes out with the partial
      double left[2] = {0.0, 0.0};
      if (warp < 4) {
        const float cr = (float)cpr, ci = (float)cpi;
        T u = ScalarTraits<T>::zero();
        if (sval) {
          const float f = wts ? fs * wt : fs;
          const float dx = w.x - cr, dy = w.y - ci;
          if constexpr (CPLX) u = make_float2(dx * f, dy * f);
          else u = dx * f;
          left[0] = (double)wt * dx;
          left[1] = (double)wt * dy;
        }
        if (row < R) s_u[row] = u;
      }
      bar_sync(kBarCompute, kCompute);
      // ---- Q = conj(t) u, 16 samples per operand stage: warps 0-7 build the even ones, 8-15 the odd ones;
      // an item is one unit x 8 samples
      for (int j = warp >> 3; j < nqs; j += 2) {
        const int use = g + j, st = use % S;
        if (use >= S && !umma::mbar_wait(&empty[st], ((use / S) - 1) & 1, kWaitP)) gave_up();
        uint8_t* base = sB + (size_t)st * stage_bytes;
        for (int item = tid & 255; item < 2 * Mh; item += 256) {
          const int h8 = item >= Mh ? 1 : 0, m = item - h8 * Mh;
          const int sl = 16 * j + 8 * h8;
          // rows sl .. sl + 7: x(sl + q) = x(sl) ^ f(q) with f known at compile time
          const int m0 = m ^ t_xor<T>(sl, Mh);
          const bool half = sizeof(T) == 8 ? (Mh & 8) != 0 : (Mh & 16) != 0;
          const T* tp = sT + sl * Mh;
          T t[8];
          if (half) {
#pragma unroll
            for (int q = 0; q < 8; ++q) t[q] = tp[q * Mh + (m0 ^ (q >> 1))];
          } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) t[q] = tp[q * Mh + (m0 ^ q)];
          }
          T u[8];
          if constexpr (CPLX) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float4 uu = reinterpret_cast<const float4*>(s_u + sl)[q];
              u[2 * q] = make_float2(uu.x, uu.y);
              u[2 * q + 1] = make_float2(uu.z, uu.w);
            }
          } else {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const float4 uu = reinterpret_cast<const float4*>(s_u + sl)[q];
              u[4 * q] = uu.x; u[4 * q + 1] = uu.y; u[4 * q + 2] = uu.z; u[4 * q + 3] = uu.w;
            }
          }
          uint32_t rh[4], rl[4], ih[4], il[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const T t0 = t[2 * q], t1 = t[2 * q + 1], u0 = u[2 * q], u1 = u[2 * q + 1];
            if constexpr (CPLX) {
              split2(t0.x * u0.x + t0.y * u0.y, t1.x * u1.x + t1.y * u1.y, rh[q], rl[q]);
              split2(t0.x * u0.y - t0.y * u0.x, t1.x * u1.y - t1.y * u1.x, ih[q], il[q]);
            } else {
              split2(t0 * u0, t1 * u1, rh[q], rl[q]);
            }
          }
          const uint32_t off = umma::kmajor_offset((uint32_t)m, (uint32_t)(8 * h8), (uint32_t)NZ);
          *reinterpret_cast<uint4*>(base + off) = make_uint4(rh[0], rh[1], rh[2], rh[3]);
          *reinterpret_cast<uint4*>(base + NZ * 32 + off) = make_uint4(rl[0], rl[1], rl[2], rl[3]);
          if constexpr (CPLX) {
            const uint32_t offi = umma::kmajor_offset((uint32_t)(Mh + m), (uint32_t)(8 * h8), (uint32_t)NZ);
            *reinterpret_cast<uint4*>(base + offi) = make_uint4(ih[0], ih[1], ih[2], ih[3]);
            *reinterpret_cast<uint4*>(base + NZ * 32 + offi) = make_uint4(il[0], il[1], il[2], il[3]);
          }
        }
        umma::fence_proxy_async_smem();
        bar_arrive(1 + st, 256 + 32);
      }
      g += nqs;
      // ---- g_a while the MMAs drain
      if (cta < d.n_chunks) {
        float gx = 0.f, gy = 0.f;
        if (ga_site < ns) {
#pragma unroll 4
          for (int k = 0; k < R / 4; ++k) {
            const int sgn = (int)((~ga_bits >> k) & 1u) << 31;
            const T u = s_u[4 * k + ga_grp];
            if constexpr (CPLX) {
              gx += __int_as_float(__float_as_int(u.x) ^ sgn);
              gy += __int_as_float(__float_as_int(u.y) ^ sgn);
            } else {
              gx += __int_as_float(__float_as_int(u) ^ sgn);
            }
          }
        }
        gx += __shfl_xor_sync(0xffffffffu, gx, 1);
        gx += __shfl_xor_sync(0xffffffffu, gx, 2);
        if constexpr (CPLX) {
          gy += __shfl_xor_sync(0xffffffffu, gy, 1);
          gy += __shfl_xor_sync(0xffffffffu, gy, 2);
        }
        if (ga_site < ns && ga_grp == 0) {
          float* dst = reinterpret_cast<float*>(part_mine) + n_mat + (int64_t)ga_site * H;
          dst[0] = gx;
          if constexpr (CPLX) dst[1] = gy;
        }
      }
      if (it >= 0 && warp < 4) {
        const double t = warp_sum_split<2>(left, lane);
        if (lane == 0 || lane == 4) s_red[17 * kVals + 2 + 2 * warp + (lane >> 2)] = t;
      }
      // ---- the CTA's partial P-vector: [16 columns][site][16]
      if (!umma::mbar_wait(done, dph, kWaitP)) {
        gave_up();
      }
      dph ^= 1u;
      umma::tc_fence_after();
      if (cta < d.n_chunks) {
        const int drow = row < ns ? row : (row == 127 ? ns : -1);
        for (int c = cg; c < NZ / 16; c += 4) {
          float v[16];
          __syncwarp();
          umma::tmem_ld16(tbase + lane_off + 16 * c, v);
          if (drow >= 0) {
            float4* dst = part_mine + ((int64_t)c * (ns + 1) + drow) * 4;
#pragma unroll
            for (int q = 0; q < 4; ++q) __stcg(dst + q, make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]));
          }
        }
      }
      umma::tc_fence_before();
      if (it >= 0 && warp == 3) {                            // the other three warps' sums: s_red below
        bar_sync(kBarLeft, 128);
        if (lane < 2) {
          double t = 0.0;
          for (int q = 0; q < 4; ++q) t += s_red[17 * kVals + 2 + 2 * q + lane];
          __stcg(reinterpret_cast<double*>(wres + cta) + lane, t);
        }
      } else if (it >= 0 && warp < 3) {
        bar_arrive(kBarLeft, 128);
      }
      ok = exchange_barrier(X, X_PART, (unsigned int)(it + 3),
                            hook.which == PcgWaitTest::PARTIALS && it == hook.pass ? 1u : 0u) && ok;
      if (!ok && it > -2) break;                             // from pass -2 by way of pass -1: see the header
      if (it >= 0) {                                         // the previous pass's words: read by everyone
        exchange_reset(X, X_DOTS, par ^ 1);
        exchange_reset(X, X_RR, par ^ 1);
      }
      // what the expected mean left: sum over all CTAs, the same in each (it < 0: nothing)
      double dr = 0.0, di = 0.0;
      if (it >= 0 && warp == 15) {
        double2 e[5];
        for (int q0 = 0; q0 < d.n_chunks; q0 += 160) {
#pragma unroll
          for (int b = 0; b < 5; ++b) {
            const int q = q0 + 32 * b + lane;
            e[b] = q < d.n_chunks ? __ldcg(wres + q) : make_double2(0.0, 0.0);
          }
#pragma unroll
          for (int b = 0; b < 5; ++b) {
            dr += e[b].x;
            di += e[b].y;
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          dr += __shfl_xor_sync(0xffffffffu, dr, o);
          di += __shfl_xor_sync(0xffffffffu, di, o);
        }
        if (lane == 0) {
          s_red[17 * kVals] = dr * inv_n;
          s_red[17 * kVals + 1] = di * inv_n;
        }
      }
      // ---- sum the partials of the owned entries in float64
      double y = 0.0;
      {
        double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
        if (sg < d.groups && vl < nv) {
          const float4* src = partial + v0 + vl;
          for (int z0 = sg; z0 < d.n_chunks; z0 += 12 * d.groups) {
            float4 q[12];
#pragma unroll
            for (int b = 0; b < 12; ++b) {
              const int z = z0 + b * d.groups;
              q[b] = z < d.n_chunks ? __ldcg(src + (int64_t)z * d.nvec) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int b = 0; b < 12; ++b) {
              a0 += q[b].x;
              a1 += q[b].y;
              a2 += q[b].z;
              a3 += q[b].w;
            }
          }
        }
        if (sg < d.groups) {
          double* o = s_acc + ((size_t)sg * d.vpc + vl) * 4;
          o[0] = a0;
          o[1] = a1;
          o[2] = a2;
          o[3] = a3;
        }
        bar_sync(kBarCompute, kCompute);
        if (tid < 4 * nv && nat >= 0)
          for (int q = 0; q < d.groups; ++q) y += s_acc[(size_t)q * d.vpc * 4 + tid];
        umma::fence_proxy_async_smem();                      // the scratch becomes an operand stage again
      }
      if (it == -2) {
        ob = y;
        if (nat >= 0) x_nat[nat] = y;                        // its other part may belong to another CTA
        cpr = cpi = 0.0;
        continue;
      }
      if (it == -1) {
        // y = F: threshold, start of the iteration.  x_nat: written before the X_PART barrier of this pass
        if (CPLX && nat >= 0) ob2 = (nat & 1) ? __ldcg(x_nat + nat - 1) : -__ldcg(x_nat + nat + 1);
        rk = y;
        pk = y;
        if (nat >= 0) b_nat[nat] = y;
        double v[3] = {y * y, ob * y, ob2 * y};
        ok = exchange_sum<3>(X, X_DOTS, 1, own_warps, v);
        bb = rr = v[0];
        crr = cpr = v[1];
        cri = cpi = v[2];
        const double th = fmax(rtol * sqrt(rr), atol);
        thresh = th * th;
        conv = rr <= thresh;
      } else {
        // conj(O-bar) times the left-over mean: ob2 carries the sign of the complex product
        y -= s_red[17 * kVals] * ob + (CPLX ? s_red[17 * kVals + 1] * ob2 : 0.0);
        y += shift * pk;
        // one exchange per iteration: |r_k|^2 from the vector itself, and |r_k+1|^2 from its expansion in the
        // three dot products (relative error about 1e-16 |r_k|^2 / |r_k+1|^2, as |r_k|^2 is not carried over)
        double v[6] = {pk * y, rk * y, y * y, rk * rk, ob * y, ob2 * y};
        ok = exchange_sum<6>(X, X_DOTS, par, own_warps, v);
        rr = v[3];
        const double alpha = v[0] > 0.0 ? rr / v[0] : 0.0;
        const double inv_rr = rr > 0.0 ? 1.0 / rr : 0.0;     // independent of alpha: the two divisions overlap
        double rr_new = rr - 2.0 * alpha * v[1] + alpha * alpha * v[2];
        xk += alpha * pk;
        rk += -alpha * y;
        if (!(rr_new > 1e-6 * rr)) {
          // a large drop (or a breakdown): the expansion has lost digits, so the vector is summed
          double q[1] = {rk * rk};
          ok = exchange_sum<1>(X, X_RR, par, own_warps, q) && ok;
          rr_new = q[0];
        }
        const double beta = rr_new * inv_rr;
        crr -= alpha * v[4];
        cri -= alpha * v[5];
        cpr = crr + beta * cpr;
        cpi = cri + beta * cpi;
        ++iters;
        rr = rr_new;
        conv = rr_new <= thresh;
        pk = rk + beta * pk;
      }
      if (!ok || conv || iters >= maxiter) break;
      // ---- the next direction's operand entries
      if (nat >= 0) {
        const float f = (float)pk;
        if (is_va) {
          __stcg(va + op_off, f);
        } else {
          const __nv_bfloat16 hi = __float2bfloat16_rn(f);
          const __nv_bfloat16 lo = __float2bfloat16_rn(f - __bfloat162float(hi));
          *reinterpret_cast<__nv_bfloat16*>(vz + op_off) = hi;
          *reinterpret_cast<__nv_bfloat16*>(vz + op_off + (size_t)NZ * 32) = lo;
        }
      }
      if (tid < 4 * nv) asm volatile("fence.proxy.async.global;" ::: "memory");
      bar_arrive(kBarAll, kThreadsP);                        // the bulk-copy warp carries the direction barrier
    }
    if (tid == 0) *s_stop = 1;
    asm volatile("" ::: "memory");
    bar_sync(kBarCompute, kCompute);
    bar_arrive(kBarAll, kThreadsP);
    if (nat >= 0) {
      x_nat[nat] = xk;
      x_out[nat] = prefactor * xk;
    }
    if (cta == 0 && tid == 0) {
      scal[0] = rr;
      scal[2] = rr;
      scal[3] = thresh;
      scal[4] = conv ? 1.0 : 0.0;
      scal[5] = (double)iters;
      scal[6] = bb;
    }
  } else if (warp == 16) {
    // ------------------------------------------------------------------ bulk copies of the direction operand
    int g = 2 * nqs;                                         // the two passes before the first iteration
    unsigned int round = 0;
    uint32_t last_ph = ~0u;                                  // per stage, phase of its last copy (none: passed)
    const int skip = hook.which == PcgWaitTest::COPY && cta == 0 ? g + hook.pass * (nks + nqs) : -1;   // test hook
    for (;;) {
      bar_sync(kBarAll, kThreadsP);
      if (__shfl_sync(0xffffffffu, *(volatile int*)s_stop, 0) != 0) break;
      ++round;
      const unsigned int extra = hook.which == PcgWaitTest::DIRECTION && (int)round == hook.pass + 1 ? 1u : 0u;
      if (lane == 0 && !grid_arrive_wait(counters + 32 * X_DIR, round * (unsigned int)G + extra, hook.polls, err))
        *(volatile int*)s_bad = 1;
      bar_arrive(kBarGo, kCompute + 64);
      if (lane == 0) {
        asm volatile("fence.proxy.async.global;" ::: "memory");     // other CTAs' stores before the bulk reads
        for (int c = 0; c < nks; ++c) {
          const int u = g + c, st = u % S;
          if (u >= S && !umma::mbar_wait(&empty[st], ((u / S) - 1) & 1, kWaitOp)) {
            gave_up();
            break;
          }
          if (u == skip) continue;
          umma::mbar_arrive_expect_tx(&full[st], stage_bytes);
          umma::bulk_g2s(sB + (size_t)st * stage_bytes, vz + (size_t)c * stage_bytes, stage_bytes, &full[st]);
          last_ph ^= 1u << st;
        }
      }
      g += nks + nqs;
      __syncwarp();
    }
    if (lane == 0) {                                         // no copy outlives the block, whoever gave up
#pragma unroll 1
      for (int st = 0; st < S; ++st) umma::mbar_wait(&full[st], (last_ph >> st) & 1u, kWaitOp);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ MMA issue
    const int n_parts = NZ > 256 ? 2 : 1;
    const uint32_t np0 = NZ > 256 ? 256u : (uint32_t)NZ;
    const uint32_t sb = umma::smem_u32(sB);
    uint32_t fph = 0;                                        // full[] parity per stage
    int g = 0;
    auto step = [&](int st, uint32_t a, bool first) {
      const uint32_t bh = sb + (uint32_t)st * stage_bytes;
      for (int pt = 0; pt < n_parts; ++pt) {
        const uint32_t n0 = pt ? np0 : 0u, nn = pt ? (uint32_t)NZ - np0 : np0;
        const uint32_t idesc = umma::idesc_bf16_f32(128, nn);
        const uint32_t b0 = bh + (n0 / 8u) * 128u;
        mma_bf16_ta(tbase + n0, a, umma::smem_desc(b0, (uint32_t)NZ * 16u, 128u), idesc, first ? 0u : 1u);
        mma_bf16_ta(tbase + n0, a, umma::smem_desc(b0 + (uint32_t)NZ * 32u, (uint32_t)NZ * 16u, 128u), idesc, 1u);
      }
      umma::mma_commit(&empty[st]);
    };
    for (int it = -2;; ++it) {
      if (it >= 0) {
        bar_sync(kBarAll, kThreadsP);
        if (__shfl_sync(0xffffffffu, *(volatile int*)s_stop, 0) != 0) break;
        bar_sync(kBarGo, kCompute + 64);
        if (lane == 0) {
          for (int c = 0; c < nks; ++c) {
            const int st = (g + c) % S;
            if (!umma::mbar_wait(&full[st], (fph >> st) & 1u, kWaitOp)) {
              gave_up();
            }
            fph ^= 1u << st;
            umma::tc_fence_after();
            step(st, col_as + 8 * c, c == 0);
          }
          umma::mma_commit(done);
        }
        g += nks;
        __syncwarp();
      }
      for (int j = 0; j < nqs; ++j) {
        const int st = (g + j) % S;
        bar_sync(1 + st, 256 + 32);                          // eight compute warps have built Q's stage
        if (lane == 0) {
          umma::tc_fence_after();
          step(st, col_at + 8 * j, j == 0);
          if (j == nqs - 1) umma::mma_commit(done);
        }
        __syncwarp();
      }
      g += nqs;
    }
  }
  __syncthreads();
  if (warp == 17) umma::tmem_dealloc(tbase, d.tmem_cols);
}

// ================================================================================================
// host side
// ================================================================================================
static int pcg_sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
    cudaGetLastError();
    return 148;
  }
  return n;
}

bool pcg_plan(int dtype, int ns, int nh, int64_t n, PcgDims* out) {
  if (ns > 127 || n < 1) return false;
  const bool cplx = dtype == QES_DTYPE_C64;
  const size_t ts = cplx ? 8 : 4;
  const int sms = std::min(pcg_sm_count(), 256);             // exchange_sum collects at most 256 slots
  PcgDims d{};
  d.ns = ns;
  d.nh = nh;
  d.Mh = cplx ? (nh + 7) / 8 * 8 : (nh + 15) / 16 * 16;
  d.NZ = cplx ? 2 * d.Mh : d.Mh;
  d.Kz = (ns + 1 + 15) / 16 * 16;
  if (d.NZ > 512) return false;
  int64_t R = (n + sms - 1) / sms;
  R = (R + 15) / 16 * 16;
  // small batches on at most kDirect CTAs, whose exchanges are shorter, while a CTA's own share (R x NZ operand entries)
  // is small.  us per iteration on at most kDirect / on all CTAs: 16 x 16, 1,024 samples 9.7 / 11.3; 60 x 256, 1,024
  // (R NZ = 8,192) 14.8 / 16.2; 63 x 128, 2,048 (8,192) 13.3 / 14.9; 36 x 64, 4,096 (8,192) 13.0 / 13.5; 36 x 32
  // complex, 4,096 (8,192) 13.5 / 13.3.  Above the line the two cross between 12,000 and 25,000: 63 x 240, 2,048 (15,360)
  // 15.5 / 17.8; 36 x 192, 4,096 (24,576) 15.1 / 15.2; complex 36 x 96, 2,048 (12,288) 13.6 / 14.5, 36 x 96, 4,096
  // (24,576) 15.4 / 14.9
  const int64_t Rd = ((n + kDirect - 1) / kDirect + 15) / 16 * 16;
  if (Rd <= 128 && Rd * d.NZ <= 8192 && (int64_t)d.NZ * (ns + 1) / 4 + ns <= 128 * kDirect) R = std::max(R, Rd);
  if (R > 128) return false;
  d.R = (int)R;
  d.n_chunks = (int)((n + R - 1) / R);
  d.nvec = (int64_t)d.NZ * (ns + 1) / 4 + ((int64_t)ns * (cplx ? 2 : 1) + 3) / 4;
  d.G = (int)std::max<int64_t>(d.n_chunks, (d.nvec + 127) / 128);     // one scalar per compute thread
  if (d.G > sms) return false;
  d.vpc = (int)((d.nvec + d.G - 1) / d.G);
  // split groups: each thread loads up to 12 partials in one batch, and the groups are added one by one
  d.groups = std::max(1, std::min(512 / d.vpc, (d.n_chunks + 11) / 12));
  d.nc = d.G <= kDirect ? d.G : (int)std::ceil(std::sqrt((double)d.G));       // G <= 256: at most 16 each
  const int cols = d.NZ + d.Kz / 2 + d.R / 2;
  if (cols > 512) return false;
  d.tmem_cols = 32;
  while (d.tmem_cols < cols) d.tmem_cols <<= 1;
  const size_t stage = (size_t)d.NZ * 64, t_bytes = ((size_t)R * d.Mh * ts + 127) & ~(size_t)127;
  const size_t fixed = t_bytes + R * ts + (17 * kVals + 10) * 8 + 8 * (2 * kMaxStages + 1) + 16;
  for (int S = std::min(kMaxStages, std::max(d.Kz / 16, 2)); S >= 2; --S) {
    const size_t total = fixed + std::max<size_t>((size_t)S * stage, 16384 + 128);
    if (total <= kSmemMax) {
      d.S = S;
      d.smem = (int)total;
      *out = d;
      return true;
    }
  }
  return false;
}

size_t pcg_partial_bytes(const PcgDims& d) { return (size_t)d.n_chunks * d.nvec * 16; }
size_t pcg_operand_bytes(const PcgDims& d) { return (size_t)d.Kz * d.NZ * 4 + (size_t)d.ns * 8 + 256; }
static size_t pcg_box_bytes(const PcgDims& d) {
  return (size_t)4 * kVals * d.G * (1 + kDirect) * sizeof(double);
}
// the calling thread's test hook
static thread_local PcgWaitTest t_wait_test{PcgWaitTest::NONE, 0, kPollLimit};
extern "C" int qes_sr_set_one_launch_wait_test(int which, int pass, unsigned int polls) {
  if (which < PcgWaitTest::NONE || which > PcgWaitTest::COPY || (which != PcgWaitTest::NONE && polls == 0)) {
    qes_set_last_message("qes_sr_set_one_launch_wait_test: which 0 (off), 1 (partials), 2 (sum), 3 (direction) or 4 (copy), "
                         "polls > 0");
    return QES_ERR_ARG;
  }
  t_wait_test = PcgWaitTest{which, pass, which == PcgWaitTest::NONE ? kPollLimit : std::min(polls, kPollLimit)};
  return QES_OK;
}
size_t pcg_slot_bytes(const PcgDims& d) { return pcg_box_bytes(d) + 256 + (size_t)d.G * sizeof(double2); }

template <class T>
static int pcg_solve_t(const PcgDims& d, int64_t n, const PcgArgs& a, cudaStream_t st) {
  unsigned int* counters = reinterpret_cast<unsigned int*>(reinterpret_cast<uint8_t*>(a.slots) + pcg_box_bytes(d));
  double2* wres = reinterpret_cast<double2*>(counters + 64);
  QES_CUDA_CHECK(cudaMemsetAsync(a.slots, 0xff, pcg_box_bytes(d), st));
  QES_CUDA_CHECK(cudaMemsetAsync(counters, 0, 256, st));
  QES_CUDA_CHECK(cudaMemsetAsync(a.status, 0, sizeof(int), st));
  static QesSmemAttr attr;
  QES_CUDA_CHECK(attr.set<(int)kSmemMax>(cg_persist_kernel<T>));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)d.G);
  cfg.blockDim = dim3(kThreadsP);
  cfg.dynamicSmemBytes = (size_t)d.smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  uint8_t* vz = reinterpret_cast<uint8_t*>(a.operand);
  float* va = reinterpret_cast<float*>(vz + (((size_t)d.Kz * d.NZ * 4 + 127) & ~(size_t)127));
  QES_CUDA_CHECK(cudaLaunchKernelEx(&cfg, cg_persist_kernel<T>, d, n, a.bits, (const T*)a.tt, a.eloc, a.wts, a.shift,
                                    a.rtol, a.atol, a.maxiter, a.prefactor, (double*)a.x, (double*)a.b,
                                    (double*)a.x_out, a.scal, (float4*)a.partial, vz, va, wres, a.slots, counters, a.status, a.err,
                                    t_wait_test));
  QES_LAUNCH_CHECK();
  return QES_OK;
}

int pcg_solve(int dtype, const PcgDims& d, int64_t n_samples, const PcgArgs& a, cudaStream_t st) {
  return dtype == QES_DTYPE_C64 ? pcg_solve_t<float2>(d, n_samples, a, st) : pcg_solve_t<float>(d, n_samples, a, st);
}
