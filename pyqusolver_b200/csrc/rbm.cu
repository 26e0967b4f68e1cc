// RBM kernels: initial chains, ratio tables, forward (theta / tanh / log psi),
// log-derivatives and the float64 parameter update.
#include "common.cuh"

#include <stdio.h>
#include <string.h>
#include <algorithm>
#include <atomic>

static thread_local char g_last_error[512] = "";

void qes_set_last_error(cudaError_t e, const char* what) {
  snprintf(g_last_error, sizeof(g_last_error), "%s: %s", what, cudaGetErrorString(e));
}
void qes_set_last_message(const char* msg) { snprintf(g_last_error, sizeof(g_last_error), "%s", msg); }

static std::atomic<long long> g_launches{0};
void qes_count_launches(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

static std::atomic<int> g_pdl{1};
bool qes_pdl_on() { return g_pdl.load(std::memory_order_relaxed) != 0; }
extern "C" int qes_set_pdl(int on) {
  g_pdl.store(on ? 1 : 0);
  return QES_OK;
}

extern "C" const char* qes_last_error(void) { return g_last_error; }

// ---------------------------------------------------------------- per-kernel event timing
#include <mutex>
#include <vector>
namespace {
// Event pairs are created on demand in blocks and kept for reuse; between two reads at most
// kProfMaxSlots launches are recorded (later ones are skipped, never blocked on).
constexpr int kProfBlock = 4096;
constexpr int kProfMaxSlots = 1 << 20;
std::mutex g_prof_mu;
std::atomic<int> g_prof_enabled{0};
std::vector<cudaEvent_t> g_prof_ev;   // 2 per slot
std::vector<int> g_prof_cls;
int g_prof_used = 0;
double g_prof_ms[QES_PROF_CLASSES];
long long g_prof_cnt[QES_PROF_CLASSES];

bool prof_grow() {
  const size_t have = g_prof_cls.size();
  if ((int)have >= kProfMaxSlots) return false;
  for (int q = 0; q < kProfBlock; ++q) {
    cudaEvent_t a, b;
    if (cudaEventCreate(&a) != cudaSuccess) return false;
    if (cudaEventCreate(&b) != cudaSuccess) { cudaEventDestroy(a); return false; }
    g_prof_ev.push_back(a);
    g_prof_ev.push_back(b);
    g_prof_cls.push_back(0);
  }
  return true;
}
}  // namespace

bool qes_prof_on() { return g_prof_enabled.load(std::memory_order_relaxed) != 0; }

int qes_prof_begin(int cls, cudaStream_t st) {
  if (!qes_prof_on()) return -1;
  std::lock_guard<std::mutex> lock(g_prof_mu);
  if (g_prof_used >= (int)g_prof_cls.size() && !prof_grow()) return -1;
  const int slot = g_prof_used++;
  g_prof_cls[slot] = cls;
  if (cudaEventRecord(g_prof_ev[2 * slot], st) != cudaSuccess) return -1;
  return slot;
}

void qes_prof_end(int slot, cudaStream_t st) {
  if (slot < 0) return;
  std::lock_guard<std::mutex> lock(g_prof_mu);
  cudaEventRecord(g_prof_ev[2 * slot + 1], st);
}

// folds the recorded pairs into the totals (the caller has synchronised)
static void prof_collect() {
  for (int q = 0; q < g_prof_used; ++q) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, g_prof_ev[2 * q], g_prof_ev[2 * q + 1]) == cudaSuccess) {
      g_prof_ms[g_prof_cls[q]] += ms;
      g_prof_cnt[g_prof_cls[q]] += 1;
    }
  }
  g_prof_used = 0;
}

extern "C" int qes_profile_enable(int enable) {
  std::lock_guard<std::mutex> lock(g_prof_mu);
  if (enable && g_prof_cls.empty() && !prof_grow()) {
    qes_set_last_message("qes_profile_enable: cannot create CUDA events");
    return QES_ERR_CUDA;
  }
  g_prof_enabled.store(enable ? 1 : 0);
  return QES_OK;
}

extern "C" int qes_profile_read(int reset, double* total_ms, long long* counts, int n) {
  std::lock_guard<std::mutex> lock(g_prof_mu);
  QES_CUDA_CHECK(cudaDeviceSynchronize());
  prof_collect();
  for (int k = 0; k < n && k < QES_PROF_CLASSES; ++k) {
    if (total_ms) total_ms[k] = g_prof_ms[k];
    if (counts) counts[k] = g_prof_cnt[k];
  }
  if (reset)
    for (int k = 0; k < QES_PROF_CLASSES; ++k) { g_prof_ms[k] = 0.0; g_prof_cnt[k] = 0; }
  return QES_OK;
}
extern "C" long long qes_launch_count(int reset) {
  return reset ? g_launches.exchange(0) : g_launches.load();
}
extern "C" int qes_version(void) { return 100; }

#define QES_ARG_CHECK(cond, msg) do { if (!(cond)) { qes_set_last_message(msg); return QES_ERR_ARG; } } while (0)

// ----------------------------------------------------------------------------
// initial chains
// ----------------------------------------------------------------------------
__global__ void init_chains_kernel(int kind, int n_up, uint32_t k0, uint32_t k1, int64_t chain_offset,
                                   int n_chains, int ns, uint32_t* __restrict__ out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_chains) return;
  const int nw = n_words(ns);
  uint32_t* w = out + (int64_t)c * nw;
  const uint32_t cid = (uint32_t)(chain_offset + c);
  if (kind == QES_INIT_RND) {
    for (int q = 0; q < nw; ++q) {
      Philox4 r = philox4x32_10(cid, (uint32_t)q, 0u, QES_STREAM_INIT_RND, k0, k1);
      uint32_t v = r.x;
      const int rem = ns - 32 * q;
      if (rem < 32) v &= (1u << rem) - 1u;
      w[q] = v;
    }
    return;
  }
  if (kind == QES_INIT_UP || kind == QES_INIT_DOWN) {
    for (int q = 0; q < nw; ++q) {
      uint32_t v = (kind == QES_INIT_UP) ? 0xffffffffu : 0u;
      const int rem = ns - 32 * q;
      if (rem < 32) v &= (1u << rem) - 1u;
      w[q] = v;
    }
    return;
  }
  // RND_FIXED: n_up ones at the front, then a Fisher-Yates shuffle driven by
  // counter (chain, pos, 0, 2).  Works on the packed words directly.
  for (int q = 0; q < nw; ++q) w[q] = 0u;
  for (int i = 0; i < n_up; ++i) w[i >> 5] |= 1u << (i & 31);
  for (int pos = ns - 1; pos > 0; --pos) {
    Philox4 r = philox4x32_10(cid, (uint32_t)pos, 0u, QES_STREAM_INIT_FIXED, k0, k1);
    const int j = (int)bounded_u32(r.x, (uint32_t)(pos + 1));
    const uint32_t bp = (w[pos >> 5] >> (pos & 31)) & 1u;
    const uint32_t bj = (w[j >> 5] >> (j & 31)) & 1u;
    if (bp != bj) {
      w[pos >> 5] ^= 1u << (pos & 31);
      w[j >> 5] ^= 1u << (j & 31);
    }
  }
}

extern "C" int qes_init_chains(int kind, int n_up, uint64_t seed, int64_t chain_offset, int n_chains, int ns,
                               uint32_t* bits_out, void* stream) {
  QES_ARG_CHECK(ns > 0 && n_chains >= 0 && bits_out != nullptr, "qes_init_chains: bad sizes/pointers");
  QES_ARG_CHECK(kind >= QES_INIT_RND && kind <= QES_INIT_DOWN, "qes_init_chains: unknown kind");
  QES_ARG_CHECK(kind != QES_INIT_RND_FIXED || (n_up >= 0 && n_up <= ns), "qes_init_chains: n_up out of range");
  if (n_chains == 0) return QES_OK;
  const int bs = 128;
  init_chains_kernel<<<(n_chains + bs - 1) / bs, bs, 0, (cudaStream_t)stream>>>(
      kind, n_up, (uint32_t)(seed & 0xffffffffu), (uint32_t)(seed >> 32), chain_offset, n_chains, ns, bits_out);
  QES_LAUNCH_CHECK();
  return QES_OK;
}

// ----------------------------------------------------------------------------
// ratio tables
// ----------------------------------------------------------------------------
QES_D void cosh_sinh2(float d, float& c, float& s) {
  const float e = expf(2.f * d), ei = 1.f / e;
  c = 0.5f * (e + ei);
  s = 0.5f * (e - ei);
}
QES_D void cosh_sinh2(float2 d, float2& c, float2& s) {
  // cosh(x+iy) = cosh x cos y + i sinh x sin y ; sinh(x+iy) = sinh x cos y + i cosh x sin y
  const float x = 2.f * d.x, y = 2.f * d.y;
  const float e = expf(x), ei = 1.f / e;
  const float ch = 0.5f * (e + ei), sh = 0.5f * (e - ei);
  float sn, cs;
  sincosf(y, &sn, &cs);
  c = make_float2(ch * cs, sh * sn);
  s = make_float2(sh * cs, ch * sn);
}

template <class T>
__global__ void move_tables_kernel(int nh, const T* __restrict__ a, const T* __restrict__ W, int K,
                                   const int32_t* __restrict__ mi, const int32_t* __restrict__ mj,
                                   const int32_t* __restrict__ mk, int move_major, T* __restrict__ Ct,
                                   T* __restrict__ St, T* __restrict__ A) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t total = (int64_t)K * nh;
  if (idx >= total) return;
  // layout [m][k] (local energy) or [k][m] (sampler)
  const int m = move_major ? (int)(idx % nh) : (int)(idx / K);
  const int k = move_major ? (int)(idx / nh) : (int)(idx % K);
  const int i = mi[k], j = mj[k], kind = mk[k];
  T d;
  if (kind == QES_MOVE_FLIP1) d = W[(int64_t)i * nh + m];
  else if (kind == QES_MOVE_PAIR_ANTI) d = addx(W[(int64_t)i * nh + m], scal(-1.f, W[(int64_t)j * nh + m]));
  else d = addx(W[(int64_t)i * nh + m], W[(int64_t)j * nh + m]);
  T c, s;
  cosh_sinh2(d, c, s);
  Ct[idx] = c;
  St[idx] = s;
  if (m == 0) {
    T av = a[i];
    if (kind == QES_MOVE_PAIR_ANTI) av = addx(av, scal(-1.f, a[j]));
    else if (kind == QES_MOVE_PAIR_PAR) av = addx(av, a[j]);
    A[k] = av;
  }
}

extern "C" int qes_rbm_move_tables(int dtype, int ns, int nh, const void* a, const void* W, int n_moves,
                                   const int32_t* move_i, const int32_t* move_j, const int32_t* move_kind,
                                   int move_major, void* Ct, void* St, void* A, void* stream) {
  QES_ARG_CHECK(ns > 0 && nh > 0 && n_moves >= 0, "qes_rbm_move_tables: bad sizes");
  QES_ARG_CHECK(dtype == QES_DTYPE_F32 || dtype == QES_DTYPE_C64, "qes_rbm_move_tables: bad dtype");
  if (n_moves == 0) return QES_OK;
  QES_ARG_CHECK(a && W && move_i && move_j && move_kind && Ct && St && A, "qes_rbm_move_tables: null pointer");
  const int64_t total = (int64_t)n_moves * nh;
  const int bs = 256;
  const unsigned grid = (unsigned)((total + bs - 1) / bs);
  if (dtype == QES_DTYPE_F32)
    move_tables_kernel<float><<<grid, bs, 0, (cudaStream_t)stream>>>(
        nh, (const float*)a, (const float*)W, n_moves, move_i, move_j, move_kind, move_major, (float*)Ct, (float*)St,
        (float*)A);
  else
    move_tables_kernel<float2><<<grid, bs, 0, (cudaStream_t)stream>>>(
        nh, (const float2*)a, (const float2*)W, n_moves, move_i, move_j, move_kind, move_major, (float2*)Ct,
        (float2*)St, (float2*)A);
  QES_LAUNCH_CHECK();
  return QES_OK;
}

// ----------------------------------------------------------------------------
// forward: theta, tanh(theta), log psi
// ----------------------------------------------------------------------------
// Register-tiled contraction: a block of 32 x 8 threads takes 8 RS samples and walks the hidden units 128 at a
// time, a thread accumulating RS samples x 4 units: real, units 4 lane ..; complex, lane, lane + 32, ..., since
// there tanh and log cosh, not the multiply-adds, are most of the work and a last pass of few units then skips them
// by the 32 (2,000 samples of 36 sites x 144 units: 28.5 -> 18.8 us with log psi).  Per 32 sites the block stages the
// spins as +-1 floats and the W rows in shared memory, so that a site costs a thread 2 or 3 16-byte loads for 4 RS (real) or
// 8 RS (complex) multiply-adds (one thread per unit with the signs taken from the spin words needed five
// integer and select instructions per multiply-add).  theta accumulates b, then the sites in order, each
// product exact, so its value does not depend on the tiling.  log psi (LP) does: its terms are added as 256 threads
// with units t, t + 256, ... would, then 32 at a time by butterflies, then the eight sums in order; a thread
// holds the sums of its four units of both 128-unit halves.  Bound by FP32 issue.
// W slices are copied a slice ahead (asynchronous copies into two buffers); the last one ends at a multiple of 8 sites.
// Measured (B200), the one-thread-per-unit form / this one: 16,384 samples of 20x20 x 1,600 real, tanh 2.41 / 0.62 ms,
// log psi 2.40 / 0.82 ms (0.28 ms at the FP32 rate; 0.81 / 0.83 ms with single-buffered slices), of 10x10 x 200
// complex, tanh 189 / 85 us, log psi 171 / 121 us; 20,000 samples of 100 x 64 real, 85 / 27 and 88 / 45 us.  Slower than that
// form: log psi of a handful of sites with tens of thousands of samples (50,814 of 5 x 246 real 50 / 62 us, 39,586 of 2 x 334
// 43 / 66 us), where a block's start and its sums over the units are most of its time.
constexpr int FWD_MAX_SITES = 24576;     // the entry's documented range, not a limit of the kernel
constexpr int FWD_SB = 16;               // samples per block of the batched form (RS = 2)
constexpr int FWD_TX = 32, FWD_TY = 8;
constexpr int FWD_THREADS = FWD_TX * FWD_TY;
// log psi of few sites is the latency of log cosh: two real samples per thread at three blocks per SM up to FWD_FEW sites, us
// for 20,000 samples against four samples at two blocks: 16 x 32 20 / 25, 32 x 128 24 / 29, 48 x 96 29 / 33, 64 x 128 37 / 37
constexpr int FWD_FEW = 48, FWD_MINB = 3;
constexpr int FWD_K = 32;                // sites per staged slice: one spin word
constexpr int FWD_KS = 8;                // the last slice is padded to a multiple of this
constexpr int FWD_U = 4 * FWD_TX;        // hidden units per pass

template <class T>
QES_D T fma_sign(float sg, T w, T acc);
template <>
QES_D float fma_sign<float>(float sg, float w, float acc) { return fmaf(sg, w, acc); }
template <>
QES_D float2 fma_sign<float2>(float sg, float2 w, float2 acc) {
  return make_float2(fmaf(sg, w.x, acc.x), fmaf(sg, w.y, acc.y));
}

QES_D float shfl_xor_val(float v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
QES_D float2 shfl_xor_val(float2 v, int o) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}
QES_D float shfl_val(float v, int l) { return __shfl_sync(0xffffffffu, v, l); }
QES_D float2 shfl_val(float2 v, int l) {
  return make_float2(__shfl_sync(0xffffffffu, v.x, l), __shfl_sync(0xffffffffu, v.y, l));
}

// dynamic shared memory of a block: W slices and signs, double-buffered
template <class T, int RS>
constexpr int fwd_smem() { return 2 * FWD_K * (FWD_U * (int)sizeof(T) + FWD_TY * RS * 4); }

// one block of 8 RS samples starting at row s0; VEC: W rows start on 16-byte boundaries; LP: log psi asked for; SPREAD: a lane's
// units 32 apart instead of in a row
template <class T, int RS, bool VEC, bool LP, bool SPREAD>
QES_D void rbm_forward_block(uint8_t* smem, int64_t s0, int ns, int nh, int64_t n_samples,
                             const uint32_t* __restrict__ bits, const T* __restrict__ a, const T* __restrict__ b,
                             const T* __restrict__ W, T* __restrict__ theta_out, T* __restrict__ tanh_out,
                             T* __restrict__ logpsi_out) {
  constexpr int TS = FWD_TY * RS;
  T* ws_all = reinterpret_cast<T*>(smem);                                     // [2][FWD_K][FWD_U]
  float* sg_all = reinterpret_cast<float*>(smem + 2 * FWD_K * FWD_U * sizeof(T));       // [2][FWD_K][TS]
  const int nw = n_words(ns);
  const int tid = threadIdx.x, lane = tid & 31, row = tid >> 5;
  T lsum[LP ? RS : 1][2][4];                  // of the virtual threads 128 h + (unit of c)
#pragma unroll
  for (int q = 0; q < (LP ? RS : 1); ++q)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int c = 0; c < 4; ++c) lsum[q][h][c] = ScalarTraits<T>::zero();
  // 16-byte stores where every row's groups of 4 units start on a 16-byte boundary
  const bool vec = nh % 4 == 0 && ((reinterpret_cast<uintptr_t>(theta_out) | reinterpret_cast<uintptr_t>(tanh_out)) & 15) == 0;
  // slice q = (unit pass, spin word): W by asynchronous copies, the spins of row tid % TS as +-1
  const int nsl = (ns + FWD_K - 1) / FWD_K, total = nsl * ((nh + FWD_U - 1) / FWD_U);
  constexpr int BPT = FWD_K * TS / FWD_THREADS;                               // spins per thread and slice
  const int sl = tid % TS, ib = (tid / TS) * BPT;
  auto sites = [&](int i0) { return min(FWD_K, (ns - i0 + FWD_KS - 1) / FWD_KS * FWD_KS); };   // of a slice, padded
  auto spin_word = [&](int q) {
    const int i0 = (q % nsl) * FWD_K;
    return (s0 + sl < n_samples) ? bits[(s0 + sl) * nw + (i0 >> 5)] : 0u;
  };
  auto stage = [&](int q, int buf, uint32_t word) {
    const int u0 = (q / nsl) * FWD_U, i0 = (q % nsl) * FWD_K;
    T* ws = ws_all + buf * FWD_K * FWD_U;
    constexpr int PER = VEC ? 16 / (int)sizeof(T) : 1;
#pragma unroll 4
    for (int e = tid; e < sites(i0) * FWD_U / PER; e += FWD_THREADS) {
      const int ul = (e % (FWD_U / PER)) * PER, il = e / (FWD_U / PER);
      const bool ok = i0 + il < ns && u0 + ul < nh;                           // VEC: nh is a multiple of PER
      cp_async<PER * (int)sizeof(T)>(ws + il * FWD_U + ul, ok ? W + (int64_t)(i0 + il) * nh + u0 + ul : W, ok);
    }
    cp_async_commit();
    float* sg = sg_all + buf * FWD_K * TS;
#pragma unroll
    for (int e = 0; e < BPT; ++e) {
      const int il = ib + e;
      sg[il * TS + sl] = (s0 + sl < n_samples && i0 + il < ns) ? (((word >> il) & 1u) ? 1.f : -1.f) : 0.f;
    }
  };
  uint32_t next_word = spin_word(0);
  stage(0, 0, next_word);
  if (total > 1) next_word = spin_word(1);
  int q_sl = 0;
  for (int u0 = 0; u0 < nh; u0 += FWD_U) {
    const int m0 = u0 + (SPREAD ? 1 : 4) * lane;                // unit c: m0 + c, complex m0 + 32 c
    constexpr int MC = SPREAD ? 32 : 1;
    T acc[RS][4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const T bm = (m0 + MC * c < nh) ? b[m0 + MC * c] : ScalarTraits<T>::zero();
#pragma unroll
      for (int q = 0; q < RS; ++q) acc[q][c] = bm;
    }
    for (int i0 = 0; i0 < ns; i0 += FWD_K, ++q_sl) {
      const int buf = q_sl & 1;
      cp_async_wait_all();
      __syncthreads();                                       // this slice is staged, the other buffer is consumed
      if (q_sl + 1 < total) {
        stage(q_sl + 1, buf ^ 1, next_word);
        if (q_sl + 2 < total) next_word = spin_word(q_sl + 2);
      }
      const T* ws = ws_all + buf * FWD_K * FWD_U + (SPREAD ? 1 : 4) * lane;
      const float* sg = sg_all + buf * FWD_K * TS + RS * row;
      const int nk = sites(i0);
#pragma unroll 1
      for (int ik = 0; ik < nk; ik += FWD_KS) {
#pragma unroll
      for (int il = ik; il < ik + FWD_KS; ++il) {
        T w[4];
        if constexpr (SPREAD) {
#pragma unroll
          for (int c = 0; c < 4; ++c) w[c] = ws[il * FWD_U + 32 * c];
        } else {
          const float4 w4 = *reinterpret_cast<const float4*>(ws + il * FWD_U);
          w[0] = w4.x; w[1] = w4.y; w[2] = w4.z; w[3] = w4.w;
        }
        float x[RS];
        if constexpr (RS % 4 == 0) {
#pragma unroll
          for (int q = 0; q < RS; q += 4) {
            const float4 x4 = *reinterpret_cast<const float4*>(sg + il * TS + q);
            x[q] = x4.x; x[q + 1] = x4.y; x[q + 2] = x4.z; x[q + 3] = x4.w;
          }
        } else {
#pragma unroll
          for (int q = 0; q < RS; ++q) x[q] = sg[il * TS + q];
        }
#pragma unroll
        for (int q = 0; q < RS; ++q)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[q][c] = fma_sign(x[q], w[c], acc[q][c]);
      }
      }
    }
    // Functions of all four units (theta = 0 past nh), whichever of them count: a lane's chains then overlap
#pragma unroll
    for (int q = 0; q < RS; ++q) {
      const int64_t s = s0 + RS * row + q;
      if (s < n_samples) {
        const int64_t o = s * nh + m0;
        T t[4];
        if (tanh_out) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (!SPREAD || u0 + 32 * c < nh) t[c] = tanhx(acc[q][c]);
        }
        if (SPREAD || !vec) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (m0 + MC * c < nh) {
              if (theta_out) theta_out[o + MC * c] = acc[q][c];
              if (tanh_out) tanh_out[o + MC * c] = t[c];
            }
        } else if (m0 < nh) {                                  // 16-byte vectors of 4 units
          if (theta_out) *reinterpret_cast<float4*>(theta_out + o) = *reinterpret_cast<const float4*>(acc[q]);
          if (tanh_out) *reinterpret_cast<float4*>(tanh_out + o) = *reinterpret_cast<const float4*>(t);
        }
      }
    }
    if constexpr (LP) {
      if (logpsi_out) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (!SPREAD || u0 + 32 * c < nh) {
            T l[RS];
#pragma unroll
            for (int q = 0; q < RS; ++q) {
              l[q] = log_cosh(acc[q][c]);
              if (m0 + MC * c >= nh) l[q] = ScalarTraits<T>::zero();
            }
            if ((u0 / FWD_U) & 1) {
#pragma unroll
              for (int q = 0; q < RS; ++q) lsum[q][1][c] = addx(lsum[q][1][c], l[q]);
            } else {
#pragma unroll
              for (int q = 0; q < RS; ++q) lsum[q][0][c] = addx(lsum[q][0][c], l[q]);
            }
          }
      }
    }
  }
  if constexpr (LP) {
    if (!logpsi_out) return;
    auto unit = [&](int h, int c) { return 128 * h + (SPREAD ? lane + 32 * c : 4 * lane + c); };
    T av[2][4];                                                // the visible terms of the first 256 sites
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int c = 0; c < 4; ++c) av[h][c] = unit(h, c) < ns ? a[unit(h, c)] : ScalarTraits<T>::zero();
#pragma unroll
    for (int q = 0; q < RS; ++q) {
      const int64_t s = s0 + RS * row + q;
      const uint32_t* wq = bits + (s < n_samples ? s : s0) * nw;
      T v = ScalarTraits<T>::zero();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        T x[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          x[c] = lsum[q][h][c];
          const int i0 = unit(h, c);
          if (i0 < ns) x[c] = fma_sign(sigma_of(wq, i0), av[h][c], x[c]);
          for (int i = i0 + 256; i < ns; i += 256) x[c] = fma_sign(sigma_of(wq, i), a[i], x[c]);
#pragma unroll
          for (int o = SPREAD ? 16 : 4; o > 0; o >>= 1) x[c] = addx(x[c], shfl_xor_val(x[c], o));
        }
        if constexpr (SPREAD) {                                  // the four sums of 32, in every lane
#pragma unroll
          for (int c = 0; c < 4; ++c) v = addx(v, x[c]);
        } else {                                               // threads 16, 8 and 4 apart above; 2 and 1 apart here
          const T e = addx(addx(x[0], x[2]), addx(x[1], x[3]));
#pragma unroll
          for (int g = 0; g < 4; ++g) v = addx(v, shfl_val(e, 8 * g));
        }
      }
      if (lane == 0 && s < n_samples) logpsi_out[s] = v;
    }
  }
}

template <class T, int RS, bool VEC, bool LP, bool SPREAD>
__global__ void __launch_bounds__(FWD_THREADS, LP && RS <= 2 && !ScalarTraits<T>::is_complex ? FWD_MINB : 2) rbm_forward_kernel(
    int ns, int nh, int64_t n_samples, const uint32_t* __restrict__ bits, const T* __restrict__ a,
    const T* __restrict__ b, const T* __restrict__ W, T* __restrict__ theta_out, T* __restrict__ tanh_out,
    T* __restrict__ logpsi_out) {
  extern __shared__ __align__(16) uint8_t fwd_sm[];
  rbm_forward_block<T, RS, VEC, LP, SPREAD>(fwd_sm, (int64_t)blockIdx.x * FWD_TY * RS, ns, nh, n_samples, bits, a, b, W, theta_out,
                                tanh_out, logpsi_out);
}

// Real layers of few units: a lane's units 32 apart, so that a pass of few units evaluates tanh and log cosh once or twice per
// lane and not four times, at three more loads per site: 58,532 samples of 3 x 12 tanh 29 -> 21 us, 20,000 of 100 x 30
// 37 -> 33; 128 x 64 31 -> 35, 60 x 90 23 -> 25
static bool fwd_spread(int ns, int nh) { return nh <= 64 && ns <= 96; }

template <class T, int RS, bool LP>
static int launch_forward_rs(int ns, int nh, int64_t n, const uint32_t* bits, const T* a, const T* b, const T* W,
                             T* theta_out, T* tanh_out, T* logpsi_out, cudaStream_t st) {
  const unsigned grid = (unsigned)((n + FWD_TY * RS - 1) / (FWD_TY * RS));
  const bool vec = nh % (16 / (int)sizeof(T)) == 0 && (reinterpret_cast<uintptr_t>(W) & 15) == 0;
  const bool spread = ScalarTraits<T>::is_complex || fwd_spread(ns, nh);
  constexpr bool C = ScalarTraits<T>::is_complex;
  auto kern = spread ? (vec ? rbm_forward_kernel<T, RS, true, LP, true> : rbm_forward_kernel<T, RS, false, LP, true>)
                     : (vec ? rbm_forward_kernel<T, RS, true, LP, C> : rbm_forward_kernel<T, RS, false, LP, C>);
  constexpr int smem = fwd_smem<T, RS>();
  static QesSmemAttr attr[4];
  QES_CUDA_CHECK(attr[2 * spread + vec].set<smem>(kern));
  kern<<<grid, FWD_THREADS, smem, st>>>(ns, nh, n, bits, a, b, W, theta_out, tanh_out, logpsi_out);
  QES_LAUNCH_CHECK();
  return QES_OK;
}

// samples per thread: the most that leave a block for every SM, down to one; half as many at most with log psi,
// whose eight sums per sample live in registers
template <class T>
static int launch_forward(int ns, int nh, int64_t n, const uint32_t* bits, const T* a, const T* b, const T* W,
                          T* theta_out, T* tanh_out, T* logpsi_out, cudaStream_t st) {
  constexpr int MAX = ScalarTraits<T>::is_complex ? 4 : 8;
  auto blocks = [&](int rs) { return (n + FWD_TY * rs - 1) / (FWD_TY * rs); };
#define QES_FWD(RS, LP) launch_forward_rs<T, RS, LP>(ns, nh, n, bits, a, b, W, theta_out, tanh_out, logpsi_out, st)
  if (logpsi_out) {
    if (blocks(MAX / 2) >= 148 && (MAX / 2 == 2 || ns > FWD_FEW)) return QES_FWD(MAX / 2, true);
    if constexpr (MAX / 2 > 2)
      if (blocks(2) >= 148) return QES_FWD(2, true);
    return QES_FWD(1, true);
  }
  if (blocks(MAX) >= 148) return QES_FWD(MAX, false);
  if constexpr (MAX > 4)
    if (blocks(4) >= 148) return QES_FWD(4, false);
  if (blocks(2) >= 148) return QES_FWD(2, false);
  return QES_FWD(1, false);
#undef QES_FWD
}

extern "C" int qes_rbm_forward(int dtype, int ns, int nh, int64_t n_samples, const uint32_t* bits, const void* a,
                               const void* b, const void* W, void* theta_out, void* tanh_out, void* logpsi_out,
                               void* stream) {
  QES_ARG_CHECK(ns > 0 && nh > 0 && n_samples >= 0, "qes_rbm_forward: bad sizes");
  QES_ARG_CHECK(dtype == QES_DTYPE_F32 || dtype == QES_DTYPE_C64, "qes_rbm_forward: bad dtype");
  QES_ARG_CHECK(bits && a && b && W, "qes_rbm_forward: null input");
  if (n_samples == 0) return QES_OK;
  QES_ARG_CHECK(ns <= FWD_MAX_SITES, "qes_rbm_forward: ns too large");
  if (dtype == QES_DTYPE_F32)
    return launch_forward<float>(ns, nh, n_samples, bits, (const float*)a, (const float*)b, (const float*)W,
                                 (float*)theta_out, (float*)tanh_out, (float*)logpsi_out, (cudaStream_t)stream);
  return launch_forward<float2>(ns, nh, n_samples, bits, (const float2*)a, (const float2*)b, (const float2*)W,
                                (float2*)theta_out, (float2*)tanh_out, (float2*)logpsi_out, (cudaStream_t)stream);
}

// ----------------------------------------------------------------------------
// log-derivatives O (row-major, leading dimension ldo)
// ----------------------------------------------------------------------------
// One block per sample; its warps take the a and b parts and the W rows (one row = nh consecutive elements
// sigma_i t_m) in turn, each written as 16-byte vectors between the elements before its first 16-byte boundary
// and after its last.  No division per element (the flat form divided every index by nh).  Bound by the
// stores: 4,096 rows of 20,300 complex64 elements (665 MB) 425 -> 121 us, 102 us at the measured copy rate.  Where the samples
// alone do not fill the chip, several blocks share a sample (LD_BLOCKS in all): 3 rows of 423 sites x 968 units 65 -> 14 us.
constexpr int LD_WARPS = 8;
constexpr int LD_BLOCKS = 4 * 148;
// Units up to which log_derivatives_flat_kernel runs, us of the form above / of the flat one: 100 sites x 12 real, 60,000
// rows 698 / 125, x 96, 10,208 rows 124 / 118, x 127, 7,735 rows 100 / 119; complex x 12, 38,109 rows 437 / 99, x 96, 5,104 rows
// 80 / 82, x 127, 3,867 rows 76 / 84
constexpr int LD_FLAT = 96;

// elements [0, n) of a row segment: dst[k] = f(k)
template <class T, class F>
QES_D void put_row(T* dst, int n, int lane, F f) {
  constexpr int E = 16 / (int)sizeof(T);
  const int mis = (int)((reinterpret_cast<uintptr_t>(dst) & 15) / sizeof(T));
  const int head = min(n, (E - mis) % E), nv = (n - head) / E, tail = n - head - nv * E;
  if (lane < head) dst[lane] = f(lane);
  float4* v = reinterpret_cast<float4*>(dst + head);
  for (int q = lane; q < nv; q += 32) {
    T x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) x[e] = f(head + q * E + e);
    float4 o;
    if constexpr (ScalarTraits<T>::is_complex) o = make_float4(x[0].x, x[0].y, x[1].x, x[1].y);
    else o = make_float4(x[0], x[1], x[2], x[3]);
    v[q] = o;
  }
  if (lane < tail) dst[n - tail + lane] = f(n - tail + lane);
}

template <class T>
__global__ void __launch_bounds__(32 * LD_WARPS) log_derivatives_kernel(int ns, int nh, int64_t n_samples,
                                                                       const uint32_t* __restrict__ bits,
                                                                       const T* __restrict__ tanh_theta,
                                                                       T* __restrict__ O, int64_t ldo) {
  const int64_t s = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t* w = bits + s * n_words(ns);
  T* row = O + s * ldo;
  const T* t = tanh_theta + s * nh;
  if (blockIdx.y == 0) {
    if (warp == 0) put_row(row, ns, lane, [&](int i) { return scal(sigma_of(w, i), ScalarTraits<T>::one()); });
    if (warp == 1) put_row(row + ns, nh, lane, [&](int m) { return t[m]; });
  }
  for (int64_t i = (int64_t)blockIdx.y * LD_WARPS + warp; i < ns; i += LD_WARPS * gridDim.y) {
    const float sg = sigma_of(w, (int)i);
    put_row(row + ns + nh + i * nh, nh, lane, [&](int m) { return scal(sg, t[m]); });
  }
}

// Narrow layers, whose W rows leave most of a warp without a vector: TPR threads (a warp up to P = 64 vectors, else the
// block) walk a sample's P elements as one run of 16-byte vectors, with one division per vector.  Bound by the stores from
// about 12 units on (2.5-4 TB/s).
template <class T, int TPR>
__global__ void __launch_bounds__(32 * LD_WARPS) log_derivatives_flat_kernel(int ns, int nh, int64_t n_samples,
                                                                            const uint32_t* __restrict__ bits,
                                                                            const T* __restrict__ tanh_theta,
                                                                            T* __restrict__ O, int64_t ldo) {
  constexpr int E = 16 / (int)sizeof(T);
  const int64_t s = (int64_t)blockIdx.x * (32 * LD_WARPS / TPR) + threadIdx.x / TPR;
  if (s >= n_samples) return;
  const int lane = threadIdx.x % TPR, P = ns + nh + ns * nh;            // P < 2^31
  const uint32_t* w = bits + s * n_words(ns);
  T* row = O + s * ldo;
  const T* t = tanh_theta + s * nh;
  auto at = [&](int k) {
    if (k < ns) return scal(sigma_of(w, k), ScalarTraits<T>::one());
    if (k < ns + nh) return t[k - ns];
    const int q = k - ns - nh, i = q / nh;
    return scal(sigma_of(w, i), t[q - i * nh]);
  };
  const int mis = (int)((reinterpret_cast<uintptr_t>(row) & 15) / sizeof(T));
  const int head = min(P, (E - mis) % E), nv = (P - head) / E, tail = P - head - nv * E;
  if (blockIdx.y == 0) {
    if (lane < head) row[lane] = at(lane);
    if (lane < tail) row[P - tail + lane] = at(P - tail + lane);
  }
  float4* v = reinterpret_cast<float4*>(row + head);
  for (int64_t q = (int64_t)blockIdx.y * TPR + lane; q < nv; q += TPR * gridDim.y) {
    const int k = head + (int)q * E;
    T x[E];
    if (k < ns + nh) {
#pragma unroll
      for (int e = 0; e < E; ++e) x[e] = at(k + e);
    } else {
      int i = (k - ns - nh) / nh, m = (k - ns - nh) - i * nh;
      float sg = sigma_of(w, i);
#pragma unroll
      for (int e = 0; e < E; ++e) {
        x[e] = scal(sg, t[m]);
        if (++m == nh && e + 1 < E) {                                  // not past the last site
          m = 0;
          sg = sigma_of(w, ++i);
        }
      }
    }
    float4 o;
    if constexpr (ScalarTraits<T>::is_complex) o = make_float4(x[0].x, x[0].y, x[1].x, x[1].y);
    else o = make_float4(x[0], x[1], x[2], x[3]);
    v[q] = o;
  }
}

template <class T>
static int launch_log_derivatives(int ns, int nh, int64_t n, const uint32_t* bits, const T* tt, T* O, int64_t ldo,
                                  cudaStream_t st) {
  constexpr int E = 16 / (int)sizeof(T);
  const int64_t P = (int64_t)ns + nh + (int64_t)ns * nh;
  const bool flat = nh <= LD_FLAT && P < (1ll << 31);
  const int tpr = flat && P <= 64 * E ? 32 : 32 * LD_WARPS, rpb = 32 * LD_WARPS / tpr;   // threads per row, rows per block
  // rows of several blocks where they are too few to fill the chip
  const int64_t most = flat ? (P / E + tpr - 1) / tpr : (ns + LD_WARPS - 1) / LD_WARPS;
  // parts of 2^30 rows, below the limit of a grid's x
  constexpr int64_t part = 1ll << 30;
  for (int64_t r0 = 0; r0 < n; r0 += part) {
    const int64_t nr = std::min(part, n - r0), nb = (nr + rpb - 1) / rpb;
    const dim3 grid((unsigned)nb, (unsigned)std::clamp<int64_t>(LD_BLOCKS / nb, 1, std::clamp<int64_t>(most, 1, 65535)));
    auto kern = !flat ? log_derivatives_kernel<T> : tpr == 32 ? log_derivatives_flat_kernel<T, 32>
                                                              : log_derivatives_flat_kernel<T, 32 * LD_WARPS>;
    kern<<<grid, 32 * LD_WARPS, 0, st>>>(ns, nh, nr, bits + r0 * n_words(ns), tt + r0 * nh, O + r0 * ldo, ldo);
    QES_LAUNCH_CHECK();
  }
  return QES_OK;
}

extern "C" int qes_rbm_log_derivatives(int dtype, int ns, int nh, int64_t n_samples, const uint32_t* bits,
                                       const void* tanh_theta, void* O_out, int64_t ldo, void* stream) {
  QES_ARG_CHECK(ns > 0 && nh > 0 && n_samples >= 0, "qes_rbm_log_derivatives: bad sizes");
  const int64_t P = (int64_t)ns + nh + (int64_t)ns * nh;
  QES_ARG_CHECK(ldo >= P, "qes_rbm_log_derivatives: ldo < P");
  if (n_samples == 0) return QES_OK;
  QES_ARG_CHECK(bits && tanh_theta && O_out, "qes_rbm_log_derivatives: null pointer");
  if (dtype == QES_DTYPE_F32)
    return launch_log_derivatives<float>(ns, nh, n_samples, bits, (const float*)tanh_theta, (float*)O_out, ldo, (cudaStream_t)stream);
  return launch_log_derivatives<float2>(ns, nh, n_samples, bits, (const float2*)tanh_theta, (float2*)O_out, ldo, (cudaStream_t)stream);
}

// ----------------------------------------------------------------------------
// float64 parameter update  master += lr * x ; params = (float) master
// ----------------------------------------------------------------------------
__global__ void param_update_kernel(int64_t n, double lr, const double* __restrict__ x, double* __restrict__ master,
                                    float* __restrict__ params) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    const double v = master[k] + lr * x[k];
    master[k] = v;
    params[k] = (float)v;
  }
}

extern "C" int qes_param_update(int dtype, int64_t n_params, double lr, const void* x, void* master, void* params,
                                void* stream) {
  QES_ARG_CHECK(n_params >= 0 && x && master && params, "qes_param_update: bad arguments");
  QES_ARG_CHECK(dtype == QES_DTYPE_F32 || dtype == QES_DTYPE_C64, "qes_param_update: bad dtype");
  const int64_t n = (dtype == QES_DTYPE_C64) ? 2 * n_params : n_params;   // interleaved re/im
  if (n == 0) return QES_OK;
  const int bs = 256;
  const unsigned grid = (unsigned)std::min<int64_t>((n + bs - 1) / bs, 4096);
  param_update_kernel<<<grid, bs, 0, (cudaStream_t)stream>>>(n, lr, (const double*)x, (double*)master,
                                                             (float*)params);
  QES_LAUNCH_CHECK();
  return QES_OK;
}

// ----------------------------------------------------------------------------
// Batched problems
// ----------------------------------------------------------------------------
constexpr int BMT_THREADS = 256;

// items (b, first element / BMT_THREADS): one thread per table element
template <class T>
__global__ void __launch_bounds__(BMT_THREADS) batch_move_tables_kernel(
    const qes_batch_instance* __restrict__ inst, int mode, const int4* __restrict__ items,
    const T* __restrict__ params, const int32_t* __restrict__ mi, const int32_t* __restrict__ mj,
    const int32_t* __restrict__ mk, T* __restrict__ Ct, T* __restrict__ St, T* __restrict__ A) {
  const int4 it = items[blockIdx.x];
  const qes_batch_instance I = inst[it.x];
  const int nh = I.nh;
  const T* a = params + I.param_off;
  const T* W = a + I.ns + nh;
  const int K = (mode == 0) ? I.ns : I.n_moves;
  const int64_t idx = (int64_t)it.y * BMT_THREADS + threadIdx.x;
  if (idx >= (int64_t)K * nh) return;
  int m, k, i, j, kind;
  if (mode == 0) {                       // single flips, move-major
    m = (int)(idx % nh); k = (int)(idx / nh);
    i = k; j = k; kind = QES_MOVE_FLIP1;
  } else {                               // lowered moves, m-major
    m = (int)(idx / K); k = (int)(idx % K);
    i = mi[I.move_off + k]; j = mj[I.move_off + k]; kind = mk[I.move_off + k];
  }
  T d;
  if (kind == QES_MOVE_FLIP1) d = W[(int64_t)i * nh + m];
  else if (kind == QES_MOVE_PAIR_ANTI) d = addx(W[(int64_t)i * nh + m], scal(-1.f, W[(int64_t)j * nh + m]));
  else d = addx(W[(int64_t)i * nh + m], W[(int64_t)j * nh + m]);
  T c, s;
  cosh_sinh2(d, c, s);
  const int64_t off = (mode == 0) ? I.flip_off : I.move_table_off;
  Ct[off + idx] = c;
  St[off + idx] = s;
  if (mode == 1 && m == 0 && A) {
    T av = a[i];
    if (kind == QES_MOVE_PAIR_ANTI) av = addx(av, scal(-1.f, a[j]));
    else if (kind == QES_MOVE_PAIR_PAR) av = addx(av, a[j]);
    A[I.move_off + k] = av;
  }
}

extern "C" int qes_batch_move_tables(int dtype, int n_inst, const qes_batch_instance* inst, int mode, int n_items,
                                     const int32_t* items, const void* params, const int32_t* move_i,
                                     const int32_t* move_j, const int32_t* move_kind, void* Ct, void* St, void* A,
                                     void* stream) {
  QES_ARG_CHECK(dtype == QES_DTYPE_F32 || dtype == QES_DTYPE_C64, "qes_batch_move_tables: bad dtype");
  QES_ARG_CHECK(mode == 0 || mode == 1, "qes_batch_move_tables: mode must be 0 (flips) or 1 (moves)");
  QES_ARG_CHECK(n_inst >= 0 && n_items >= 0, "qes_batch_move_tables: bad sizes");
  if (n_items == 0) return QES_OK;
  QES_ARG_CHECK(inst && items && params && Ct && St, "qes_batch_move_tables: null pointer");
  QES_ARG_CHECK(mode == 0 || (move_i && move_j && move_kind && A), "qes_batch_move_tables: null move arrays");
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == QES_DTYPE_F32)
    batch_move_tables_kernel<float><<<n_items, BMT_THREADS, 0, st>>>(inst, mode, (const int4*)items,
                                                                     (const float*)params, move_i, move_j, move_kind,
                                                                     (float*)Ct, (float*)St, (float*)A);
  else
    batch_move_tables_kernel<float2><<<n_items, BMT_THREADS, 0, st>>>(inst, mode, (const int4*)items,
                                                                      (const float2*)params, move_i, move_j,
                                                                      move_kind, (float2*)Ct, (float2*)St,
                                                                      (float2*)A);
  QES_LAUNCH_CHECK();
  return QES_OK;
}

// items (b, sample block of FWD_SB)
template <class T>
__global__ void __launch_bounds__(FWD_THREADS) batch_forward_kernel(const qes_batch_instance* __restrict__ inst,
                                                                   const int4* __restrict__ items,
                                                                   const T* __restrict__ params,
                                                                   const uint32_t* __restrict__ bits,
                                                                   T* __restrict__ tanh_out, T* __restrict__ logpsi_out) {
  const int4 it = items[blockIdx.x];
  const qes_batch_instance I = inst[it.x];
  const T* a = params + I.param_off;
  const T* b = a + I.ns;
  const T* W = b + I.nh;
  const int64_t rows = (int64_t)I.n_chains * I.num_samples;
  extern __shared__ __align__(16) uint8_t fwd_sm[];
  rbm_forward_block<T, 2, false, true, ScalarTraits<T>::is_complex>(fwd_sm, (int64_t)it.y * FWD_SB, I.ns, I.nh, rows, bits + I.sample_word_off, a, b, W,
                       nullptr, tanh_out ? tanh_out + I.tanh_off : nullptr,
                       logpsi_out ? logpsi_out + I.sample_off : nullptr);
}

extern "C" int qes_batch_rbm_forward(int dtype, int n_inst, const qes_batch_instance* inst, int n_items,
                                     const int32_t* items, const void* params, const uint32_t* sample_bits,
                                     void* tanh_out, void* logpsi_out, void* stream) {
  QES_ARG_CHECK(dtype == QES_DTYPE_F32 || dtype == QES_DTYPE_C64, "qes_batch_rbm_forward: bad dtype");
  QES_ARG_CHECK(n_inst >= 0 && n_items >= 0, "qes_batch_rbm_forward: bad sizes");
  if (n_items == 0) return QES_OK;
  QES_ARG_CHECK(inst && items && params && sample_bits, "qes_batch_rbm_forward: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  static QesSmemAttr attr;
  QES_CUDA_CHECK((attr.set<fwd_smem<float2, 2>()>(batch_forward_kernel<float2>)));
  if (dtype == QES_DTYPE_F32)
    batch_forward_kernel<float><<<n_items, FWD_THREADS, fwd_smem<float, 2>(), st>>>(inst, (const int4*)items, (const float*)params,
                                                                  sample_bits, (float*)tanh_out, (float*)logpsi_out);
  else
    batch_forward_kernel<float2><<<n_items, FWD_THREADS, fwd_smem<float2, 2>(), st>>>(inst, (const int4*)items, (const float2*)params,
                                                                   sample_bits, (float2*)tanh_out,
                                                                   (float2*)logpsi_out);
  QES_LAUNCH_CHECK();
  return QES_OK;
}

// ----------------------------------------------------------------------------
// replica swap of a region (Renyi-2 estimator): out_a takes region A from b and
// the rest from a, out_b the opposite (QES/NQS/src/nqs_entropy.py:311-460)
// ----------------------------------------------------------------------------
__global__ void swap_region_kernel(int64_t n_words_total, int nw, const uint32_t* __restrict__ mask,
                                   const uint32_t* __restrict__ a, const uint32_t* __restrict__ b,
                                   uint32_t* __restrict__ oa, uint32_t* __restrict__ ob) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n_words_total;
       k += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t m = mask[k % nw], x = a[k], y = b[k];
    oa[k] = (x & ~m) | (y & m);
    ob[k] = (y & ~m) | (x & m);
  }
}

extern "C" int qes_swap_region(int64_t n_samples, int ns, const uint32_t* mask_words, const uint32_t* bits_a,
                               const uint32_t* bits_b, uint32_t* out_a, uint32_t* out_b, void* stream) {
  QES_ARG_CHECK(n_samples >= 0 && ns > 0, "qes_swap_region: bad sizes");
  if (n_samples == 0) return QES_OK;
  QES_ARG_CHECK(mask_words && bits_a && bits_b && out_a && out_b, "qes_swap_region: null pointer");
  const int nw = n_words(ns);
  const int64_t total = n_samples * nw;
  const int bs = 256;
  const unsigned grid = (unsigned)std::min<int64_t>((total + bs - 1) / bs, 148 * 16);
  swap_region_kernel<<<grid, bs, 0, (cudaStream_t)stream>>>(total, nw, mask_words, bits_a, bits_b, out_a, out_b);
  QES_LAUNCH_CHECK();
  return QES_OK;
}
