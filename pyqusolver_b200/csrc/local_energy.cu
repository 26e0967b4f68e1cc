// Fused local-energy kernel and float64 energy statistics.
//
// E_loc(s) = diag(s) + sum_k active_k(s) conj(c_k(s)) exp(-2 sigma_i A_k)
//                        prod_m (C_km - sigma_i tanh(theta_sm) S_km)
//
// The reference evaluates the full network on every connected state
// (O(K*N*M) per sample); here each psi ratio is a product over hidden units
// of one complex FMA against per-move tables that depend only on W, so the
// work is O(K*M) per sample with no transcendental in the inner loop.
//
// One problem runs eloc_tile_kernel (moves x samples in register tiles, tables and tanh rows staged in
// shared memory), the batched form eloc_moves_block: 32 moves (threadIdx.x, one warp row) x
// ELOC_ROWS sample groups (threadIdx.y) of ELOC_SPT samples each.  Tables are stored m-major (Ct[m][k])
// so a warp reads 32 consecutive moves of one hidden unit per load.  Both write one partial sum per 32
// moves and sample in the same order (bit-identical), reduced by eloc_reduce_kernel together with the
// diagonal part.
#include "common.cuh"

#define QES_ARG_CHECK(cond, msg) do { if (!(cond)) { qes_set_last_message(msg); return QES_ERR_ARG; } } while (0)

constexpr int ELOC_SPT = 4;     // samples per thread
constexpr int ELOC_ROWS = 8;    // sample groups per block
constexpr int ELOC_SB = ELOC_SPT * ELOC_ROWS;   // samples per block
constexpr int ELOC_RENORM = 16; // hidden units between renormalisations

// Move block kb (32 moves) x sample block sb (ELOC_SB samples) of one problem.
template <class T>
QES_D void eloc_moves_block(int kb, int64_t sb, int ns, int nh, int64_t n_samples, const uint32_t* __restrict__ bits,
                            const T* __restrict__ tanh_theta, int K, const int32_t* __restrict__ mi,
                            const int32_t* __restrict__ mj, const int32_t* __restrict__ mkind,
                            const float4* __restrict__ mcoef, const T* __restrict__ Ct, const T* __restrict__ St,
                            const T* __restrict__ A, float2* __restrict__ partial /* [kblocks][n_samples] */) {
  const int nw = n_words(ns);
  const int k = kb * 32 + threadIdx.x;
  const int64_t s_base = sb * ELOC_SB + (int64_t)threadIdx.y * ELOC_SPT;
  const bool kval = k < K;

  int kind = 0, i = 0, j = 0;
  float4 cf = make_float4(0.f, 0.f, 0.f, 0.f);
  T Ak = ScalarTraits<T>::zero();
  if (kval) {
    kind = mkind[k]; i = mi[k]; j = mj[k]; cf = mcoef[k]; Ak = A[k];
  }

  float g[ELOC_SPT];        // -sigma_i per sample
  bool act[ELOC_SPT];
  const T* trow[ELOC_SPT];
#pragma unroll
  for (int q = 0; q < ELOC_SPT; ++q) {
    const int64_t s = s_base + q;
    const bool sval = s < n_samples;
    const int64_t sc = sval ? s : 0;
    const uint32_t* w = bits + sc * nw;
    const uint32_t bi = kval ? bit_of(w, i) : 0u;
    bool a = kval && sval;
    if (kind == QES_MOVE_PAIR_ANTI) a = a && (bit_of(w, j) != bi);
    else if (kind == QES_MOVE_PAIR_PAR) a = a && (bit_of(w, j) == bi);
    act[q] = a;
    g[q] = bi ? -1.f : 1.f;
    trow[q] = tanh_theta + sc * nh;
  }

  T acc[ELOC_SPT];
  int ex[ELOC_SPT];
#pragma unroll
  for (int q = 0; q < ELOC_SPT; ++q) { acc[q] = ScalarTraits<T>::one(); ex[q] = 0; }

  if (kval) {
    // whole blocks of ELOC_RENORM units unrolled, then the tail; the same factor order and the same
    // renormalisation points as one loop over m
    const T* cp = Ct + k;
    const T* sp = St + k;
    int m0 = 0;
    for (; m0 + ELOC_RENORM <= nh; m0 += ELOC_RENORM) {
#pragma unroll
      for (int u = 0; u < ELOC_RENORM; ++u) {
        const int m = m0 + u;
        const T c = cp[(int64_t)m * K];
        const T s = sp[(int64_t)m * K];
#pragma unroll
        for (int q = 0; q < ELOC_SPT; ++q) acc[q] = mulx(acc[q], ratio_factor(c, g[q], trow[q][m], s));
      }
#pragma unroll
      for (int q = 0; q < ELOC_SPT; ++q) renorm(acc[q], ex[q]);
    }
    if (m0 < nh) {
      for (int m = m0; m < nh; ++m) {
        const T c = cp[(int64_t)m * K];
        const T s = sp[(int64_t)m * K];
#pragma unroll
        for (int q = 0; q < ELOC_SPT; ++q) acc[q] = mulx(acc[q], ratio_factor(c, g[q], trow[q][m], s));
      }
#pragma unroll
      for (int q = 0; q < ELOC_SPT; ++q) renorm(acc[q], ex[q]);
    }
  }

  // contribution = coef * exp(g*2*A + ex*ln2) * acc   (g = -sigma_i)
#pragma unroll
  for (int q = 0; q < ELOC_SPT; ++q) {
    float2 v = make_float2(0.f, 0.f);
    if (act[q]) {
      const float sig = -g[q];
      const float2 coef = make_float2(cf.x + sig * cf.z, cf.y + sig * cf.w);
      // exp(-2 sigma_i A_k) with the power-of-two exponent folded into the modulus
      const float2 z = to_c(scal(2.f * g[q], Ak));
      const float2 e = to_c(expx(make_float2(z.x + 0.69314718055994531f * (float)ex[q], z.y)));
      v = coef * (e * to_c(acc[q]));
    }
    v = warp_sum(v);
    if (threadIdx.x == 0) {
      const int64_t s = s_base + q;
      if (s < n_samples) partial[(int64_t)kb * n_samples + s] = v;
    }
  }
}

// ----------------------------------------------------------------------------
// Register-tiled form for one problem.  A block takes 32 moves x 32 RS samples with 8 x 32 threads; a thread
// owns 4 consecutive moves x RS samples (row, row + 32, ...).  Per chunk of ELOC_RENORM units the block holds C
// and S (unit-major, real and imaginary parts apart) and T (sample-major) in shared memory, double-buffered:
// T by asynchronous copies, C and S through registers, both requested a chunk ahead.  A factor is C + t (g S)
// with g = -sigma_i: the sign goes into t by one xor.  The sign bit of (move, sample) shares a register with the
// product's exponent (biased, so that it cannot carry into the sign).
// Factors, roundings and the order of the sum over the 32 moves are those of the form above, so the energies
// are bit-identical to it: in a stochastic-reconfiguration step even the last bits of E_loc reach the
// weights through the near-null directions of S.  Products run at 2^8 times the form above's and are renormalised only
// once they have left 1 .. 2^16, so that they never lose digits to underflow where that form would not; one that overflows
// where it need not (a chunk's factors multiply up to 2^112 .. 2^127) comes out as infinite or NaN and is taken again
// the way of the form above.
// Bound by the FP32 and integer pipes: 2 multiply-adds and 1 xor per real factor, 8 and 2 per complex one.
// Measured (B200, 16,384 samples unless stated), the form above / this one: 20x20 TFIM x 1,600 real 3.81 / 1.54 ms
// (0.57 ms at the FP32 rate), TFIM-100 x 200 real 173 / 88 us, 10x10 x 200 complex 452 / 385 us, 6x6 J1-J2 x 144
// complex, 8,192 samples, 139 / 122 us.  Packed f32x2 multiply-adds ran the same (1.53 ms against 1.51, 425 us against
// 401); four complex samples per thread at 128 registers 413 us against 401.
// ----------------------------------------------------------------------------
constexpr int ELT_K = 4;                 // moves per thread
constexpr int ELT_COLS = 8;              // thread columns: 32 moves
constexpr int ELT_ROWS = 32;             // thread rows
constexpr int ELT_THREADS = ELT_COLS * ELT_ROWS;
constexpr uint32_t ELT_EX0 = 1u << 30;   // bias of the exponent field
constexpr int ELT_UP = 8;                // products carry this power of two
constexpr float ELT_SCALE = 256.f;       // 2^ELT_UP

QES_D float xor_sign(float t, uint32_t v) { return __uint_as_float(__float_as_uint(t) ^ (v & 0x80000000u)); }
// the product over all units of move k and one sample (t its row of T), renormalised every ELOC_RENORM units
QES_D float mul_fixed(float a, float b) { return a * b; }
QES_D float2 mul_fixed(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
template <class T>
__device__ __noinline__ T eloc_product(int nh, int K, int k, const T* __restrict__ Ct, const T* __restrict__ St,
                                       const T* __restrict__ t, float g, int* ex_out) {
  T acc = ScalarTraits<T>::one();
  int ex = 0;
  for (int m = 0; m < nh; ++m) {
    acc = mul_fixed(acc, ratio_factor(Ct[(int64_t)m * K + k], g, t[m], St[(int64_t)m * K + k]));
    if (m % ELOC_RENORM == ELOC_RENORM - 1) renorm(acc, ex);
  }
  *ex_out = ex;
  return acc;
}
// VEC: rows of C, S and T start on 16-byte boundaries every 4 (real) / 2 (complex) elements; TAIL: a last chunk of fewer units
// is not padded to a whole one
template <class T, int RS, bool VEC, bool TAIL>
__global__ void __launch_bounds__(ELT_THREADS, ScalarTraits<T>::is_complex ? 3 : 2) eloc_tile_kernel(
    int ns, int nh, int64_t n_samples, const uint32_t* __restrict__ bits, const T* __restrict__ tanh_theta, int K,
    const int32_t* __restrict__ mi, const int32_t* __restrict__ mj,
    const int32_t* __restrict__ mkind, const float4* __restrict__ mcoef, const T* __restrict__ Ct,
    const T* __restrict__ St, const T* __restrict__ A, float2* __restrict__ partial /* [gridDim.x][n_samples] */) {
  constexpr bool CPLX = ScalarTraits<T>::is_complex;
  constexpr int H = CPLX ? 2 : 1;
  constexpr int UM = ELOC_RENORM;
  constexpr int TK = ELT_K * ELT_COLS, TS = RS * ELT_ROWS;
  constexpr int TW = H * UM + 4;                                     // floats per staged T row
  constexpr int NT = 2 * H;                                          // C, S | C.re, C.im, S.re, S.im
  extern __shared__ __align__(16) float elt_sm[];
  float* s_cs = elt_sm;                                              // [2][NT][UM][TK]
  float* s_t = elt_sm + 2 * NT * UM * TK;                            // [2][TS][TW]
  float2* s_red = reinterpret_cast<float2*>(elt_sm);                 // [ELT_COLS][TS], after the products
  const int tid = threadIdx.x;
  const int col = tid % ELT_COLS, row = tid / ELT_COLS;
  const int k0 = blockIdx.x * TK;
  const int64_t s0 = (int64_t)blockIdx.y * TS;
  const int nw = n_words(ns);

  // staging: this thread's C or S entries (table, unit, 4 moves) and its share of T
  const int st_tab = tid >> 7, st_u = (tid >> 3) & (UM - 1), st_k = k0 + ELT_K * (tid & 7);
  float cs[H][ELT_K];
  auto load_cs = [&](int m0) {
    const int m = m0 + st_u;
    const T* src = (st_tab ? St : Ct) + (int64_t)m * K + st_k;
    const T fill = st_tab ? ScalarTraits<T>::zero() : ScalarTraits<T>::one();
    if (VEC && m < nh && st_k + ELT_K <= K) {
      if constexpr (CPLX) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(src)), y = __ldg(reinterpret_cast<const float4*>(src) + 1);
        cs[0][0] = x.x; cs[1][0] = x.y; cs[0][1] = x.z; cs[1][1] = x.w;
        cs[0][2] = y.x; cs[1][2] = y.y; cs[0][3] = y.z; cs[1][3] = y.w;
      } else {
        const float4 x = __ldg(reinterpret_cast<const float4*>(src));
        cs[0][0] = x.x; cs[0][1] = x.y; cs[0][2] = x.z; cs[0][3] = x.w;
      }
    } else {
#pragma unroll
      for (int a = 0; a < ELT_K; ++a) {
        const T x = (m < nh && st_k + a < K) ? src[a] : fill;        // a factor of one past the units and moves
        if constexpr (CPLX) {
          cs[0][a] = x.x;
          cs[1][a] = x.y;
        } else {
          cs[0][a] = x;
        }
      }
    }
  };
  auto store_cs = [&](int buf) {
    float* o = s_cs + ((buf * NT + H * st_tab) * UM + st_u) * TK + ELT_K * (tid & 7);
#pragma unroll
    for (int h = 0; h < H; ++h)
      *reinterpret_cast<float4*>(o + h * UM * TK) = make_float4(cs[h][0], cs[h][1], cs[h][2], cs[h][3]);
  };
  auto copy_t = [&](int m0, int buf) {
    constexpr int PER = VEC ? 16 / (int)sizeof(T) : 1;               // elements per copy
    constexpr int CPR = UM / PER;                                    // copies per row
#pragma unroll
    for (int e = tid; e < TS * CPR; e += ELT_THREADS) {
      const int ss = e / CPR, u = (e % CPR) * PER;
      const bool ok = s0 + ss < n_samples && m0 + u < nh;            // VEC: nh is a multiple of PER
      cp_async<PER * (int)sizeof(T)>(s_t + (size_t)(buf * TS + ss) * TW + H * u,
                                     ok ? tanh_theta + (s0 + ss) * nh + m0 + u : tanh_theta, ok);
    }
    cp_async_commit();
  };
  copy_t(0, 0);
  load_cs(0);

  // sign bit and activity of every (move, sample) of the thread
  uint32_t v[ELT_K][RS];
  uint32_t act = 0;
#pragma unroll
  for (int a = 0; a < ELT_K; ++a) {
    const int k = k0 + ELT_K * col + a;
    const bool kval = k < K;
    const int kind = kval ? mkind[k] : 0, i = kval ? mi[k] : 0;
    const int j = (kval && kind != QES_MOVE_FLIP1) ? mj[k] : i;
#pragma unroll
    for (int q = 0; q < RS; ++q) {
      const int64_t s = s0 + ELT_ROWS * q + row;
      const bool ok = kval && s < n_samples;
      const uint32_t* w = bits + (ok ? s : 0) * nw;
      const uint32_t bi = bit_of(w, i), bj = bit_of(w, j);
      v[a][q] = (bi << 31) | (ELT_EX0 - ELT_UP);                     // g = -sigma_i: negative for spin up
      const bool on = ok && (kind == QES_MOVE_FLIP1 || ((kind == QES_MOVE_PAIR_ANTI) == (bi != bj)));
      act |= (on ? 1u : 0u) << (a * RS + q);
    }
  }
  float accr[ELT_K][RS], acci[ELT_K][RS];
#pragma unroll
  for (int a = 0; a < ELT_K; ++a)
#pragma unroll
    for (int q = 0; q < RS; ++q) {
      accr[a][q] = ELT_SCALE;
      acci[a][q] = 0.f;
    }
  store_cs(0);
  cp_async_wait_all();
  __syncthreads();

  const int nchunk = (nh + UM - 1) / UM;
  for (int ch = 0; ch < nchunk; ++ch) {
    const int buf = ch & 1;
    if (ch + 1 < nchunk) {
      copy_t((ch + 1) * UM, buf ^ 1);
      load_cs((ch + 1) * UM);
    }
    const float* cb = s_cs + buf * NT * UM * TK + ELT_K * col;
    const float* tb = s_t + (size_t)buf * TS * TW + (size_t)row * TW;
    constexpr int UV = 4 / H;                                        // units per 16-byte load of T
    auto units = [&](int u0) {
      float4 t4[RS];
#pragma unroll
      for (int q = 0; q < RS; ++q) t4[q] = *reinterpret_cast<const float4*>(tb + (size_t)q * ELT_ROWS * TW + H * u0);
#pragma unroll
      for (int uu = 0; uu < UV; ++uu) {
        float c[2 * H][ELT_K];
#pragma unroll
        for (int h = 0; h < 2 * H; ++h) {
          const float4 x = *reinterpret_cast<const float4*>(cb + (h * UM + u0 + uu) * TK);
          c[h][0] = x.x; c[h][1] = x.y; c[h][2] = x.z; c[h][3] = x.w;
        }
#pragma unroll
        for (int q = 0; q < RS; ++q) {
          const float tv[4] = {t4[q].x, t4[q].y, t4[q].z, t4[q].w};
#pragma unroll
          for (int a = 0; a < ELT_K; ++a) {
            if constexpr (CPLX) {
              const float tr = xor_sign(tv[2 * uu], v[a][q]), ti = xor_sign(tv[2 * uu + 1], v[a][q]);
              const float fr = __fmaf_rn(tr, c[2][a], __fmaf_rn(-ti, c[3][a], c[0][a]));
              const float fi = __fmaf_rn(tr, c[3][a], __fmaf_rn(ti, c[2][a], c[1][a]));
              // contractions written out: the same roundings in every instantiation
              const float r = __fmaf_rn(accr[a][q], fr, -__fmul_rn(acci[a][q], fi));
              acci[a][q] = __fmaf_rn(accr[a][q], fi, __fmul_rn(acci[a][q], fr));
              accr[a][q] = r;
            } else {
              accr[a][q] *= __fmaf_rn(xor_sign(tv[uu], v[a][q]), c[1][a], c[0][a]);
            }
          }
        }
      }
    };
    if (!TAIL || nh - ch * UM >= UM) {
#pragma unroll
      for (int u0 = 0; u0 < UM; u0 += UV) units(u0);
    } else {
      // the last chunk, up to a multiple of UV; units past nh: C = 1, S = 0, t = 0, an exact factor of one
#pragma unroll 1
      for (int u0 = 0; u0 < nh - ch * UM; u0 += UV) units(u0);
    }
    // power-of-two renormalisation (exact) of a thread whose products have left 1 .. 2^16: most never do.
    // An exponent e in [127, 142] has e + 1 = 1000xxxx in binary.
    uint32_t far = 0;
#pragma unroll
    for (int a = 0; a < ELT_K; ++a)
#pragma unroll
      for (int q = 0; q < RS; ++q) {
        const float m = CPLX ? fmaxf(fabsf(accr[a][q]), fabsf(acci[a][q])) : accr[a][q];
        far |= (__float_as_uint(m) + (1u << 23)) ^ 0x40000000u;
      }
    if (far & 0x78000000u) {
#pragma unroll
      for (int a = 0; a < ELT_K; ++a)
#pragma unroll
        for (int q = 0; q < RS; ++q) {
          int ex = 0;
          if constexpr (CPLX) {
            float2 z = make_float2(accr[a][q], acci[a][q]);
            renorm(z, ex);
            accr[a][q] = ELT_SCALE * z.x;
            acci[a][q] = ELT_SCALE * z.y;
          } else {
            renorm(accr[a][q], ex);
            accr[a][q] *= ELT_SCALE;
          }
          v[a][q] += (uint32_t)(ex - ELT_UP);                        // (a zero or infinity: not read)  |sum| < 2^30: no carry into the sign bit
        }
    }
    if (ch + 1 < nchunk) {
      store_cs(buf ^ 1);                                             // its last readers passed the previous barrier
      cp_async_wait_all();
    }
    __syncthreads();
  }

  // products that came out as zero, infinite or NaN
  bool again = false;
#pragma unroll
  for (int a = 0; a < ELT_K; ++a)
#pragma unroll
    for (int q = 0; q < RS; ++q) {
      const float size = CPLX ? fabsf(accr[a][q]) + fabsf(acci[a][q]) : fabsf(accr[a][q]);
      again |= !(size > 0.f && size <= 3.402823466e38f);
    }
  if (again) {
#pragma unroll
    for (int a = 0; a < ELT_K; ++a)
#pragma unroll
      for (int q = 0; q < RS; ++q) {
        const float size = CPLX ? fabsf(accr[a][q]) + fabsf(acci[a][q]) : fabsf(accr[a][q]);
        if (((act >> (a * RS + q)) & 1u) && !(size > 0.f && size <= 3.402823466e38f)) {
          int ex = 0;
          const T p = eloc_product(nh, K, k0 + ELT_K * col + a, Ct, St, tanh_theta + (s0 + ELT_ROWS * q + row) * nh,
                                   (v[a][q] >> 31) ? -1.f : 1.f, &ex);
          if constexpr (CPLX) {
            accr[a][q] = p.x;
            acci[a][q] = p.y;
          } else {
            accr[a][q] = p;
          }
          v[a][q] = (v[a][q] & 0x80000000u) | (ELT_EX0 + (uint32_t)ex);
        }
      }
  }

  // contribution = coef * exp(g*2*A + ex*ln2) * acc   (g = -sigma_i), summed over the 32 moves as a warp
  // would by xor shuffles: move distances 16, 8, 4 (thread columns), then 2 and 1 (a thread's own moves)
  float2 sum[ELT_K];
#pragma unroll
  for (int a = 0; a < ELT_K; ++a) {
    const int k = k0 + ELT_K * col + a;
    float4 cf = make_float4(0.f, 0.f, 0.f, 0.f);
    T Ak = ScalarTraits<T>::zero();
    if (k < K) {
      cf = mcoef[k];
      Ak = A[k];
    }
    __syncthreads();                                                 // the staged operands, the previous move's sums
#pragma unroll
    for (int q = 0; q < RS; ++q) {
      float2 e = make_float2(0.f, 0.f);
      if ((act >> (a * RS + q)) & 1u) {
        const float g = (v[a][q] >> 31) ? -1.f : 1.f;
        int ex = (int)(v[a][q] & 0x7fffffffu) - (int)ELT_EX0;
        const float sig = -g;
        const float2 coef = make_float2(cf.x + sig * cf.z, cf.y + sig * cf.w);
        const float2 z = to_c(scal(2.f * g, Ak));
        if constexpr (CPLX) {
          float2 acc = make_float2(accr[a][q], acci[a][q]);
          renorm(acc, ex);
          const float lx = __fmul_rn(0.69314718055994531f, (float)ex);
          const float2 x = expx(make_float2(__fadd_rn(z.x, lx), z.y));
          e = coef * (x * acc);
        } else {
          float acc = accr[a][q];
          renorm(acc, ex);
          const float lx = __fmul_rn(0.69314718055994531f, (float)ex);
          const float m = expf(__fadd_rn(z.x, lx)) * acc;
          e = make_float2(coef.x * m, coef.y * m);
        }
      }
      s_red[col * TS + ELT_ROWS * q + row] = e;
    }
    __syncthreads();
    if (tid < TS)
      sum[a] = ((s_red[tid] + s_red[4 * TS + tid]) + (s_red[2 * TS + tid] + s_red[6 * TS + tid])) +
               ((s_red[TS + tid] + s_red[5 * TS + tid]) + (s_red[3 * TS + tid] + s_red[7 * TS + tid]));
  }
  if (tid < TS && s0 + tid < n_samples)
    partial[(int64_t)blockIdx.x * n_samples + s0 + tid] = (sum[0] + sum[2]) + (sum[1] + sum[3]);
}

QES_HD int eloc_kblocks(int K) { return (K + 31) / 32; }

template <class T, int RS>
constexpr size_t eloc_tile_smem() {
  constexpr int H = ScalarTraits<T>::is_complex ? 2 : 1, NT = 2 * H;
  return std::max((size_t)(2 * NT * ELOC_RENORM * ELT_K * ELT_COLS + 2 * RS * ELT_ROWS * (H * ELOC_RENORM + 4)) * sizeof(float),
                  (size_t)ELT_COLS * RS * ELT_ROWS * sizeof(float2));
}

template <class T, int RS>
static int launch_eloc_tiles(int ns, int nh, int64_t n, const uint32_t* bits, const T* tt, const qes_hamiltonian* ham,
                             const T* Ct, const T* St, const T* A, float2* partial, cudaStream_t st) {
  const int K = ham->n_moves;
  const int64_t nsb = (n + RS * ELT_ROWS - 1) / (RS * ELT_ROWS);
  QES_ARG_CHECK(nsb <= 65535, "qes_local_energy: too many samples for one launch");
  constexpr int E = 16 / (int)sizeof(T);
  const uintptr_t al = reinterpret_cast<uintptr_t>(tt) | reinterpret_cast<uintptr_t>(Ct) | reinterpret_cast<uintptr_t>(St);
  const bool vec = nh % E == 0 && K % E == 0 && (al & 15) == 0;
  constexpr size_t smem = eloc_tile_smem<T, RS>();
  // complex only, where a padded unit costs 10 instructions: 82 sites x 4 units, 36,395 samples 62 -> 43 us, 4 x 37 68 -> 60,
  // 10x10 x 200 396 -> 380.  A real factor costs 2, and the second loop slows the first: 2 x 334 107 -> 111 us
  constexpr bool C = ScalarTraits<T>::is_complex;
  const bool tail = C && nh % ELOC_RENORM != 0;
  auto kern = tail ? (vec ? eloc_tile_kernel<T, RS, true, C> : eloc_tile_kernel<T, RS, false, C>)
                   : (vec ? eloc_tile_kernel<T, RS, true, false> : eloc_tile_kernel<T, RS, false, false>);
  static QesSmemAttr attr[4];
  QES_CUDA_CHECK(attr[2 * tail + vec].set<(int)smem>(kern));
  kern<<<dim3(eloc_kblocks(K), (unsigned)nsb), ELT_THREADS, smem, st>>>(ns, nh, n, bits, tt, K, ham->move_i, ham->move_j,
                                                                       ham->move_kind, (const float4*)ham->move_coef, Ct,
                                                                       St, A, partial);
  QES_LAUNCH_CHECK();
  return QES_OK;
}

// samples per thread: as many as leave two blocks per SM (complex: at most two, three blocks of 80 registers
// per SM), down to one
template <class T>
static int launch_eloc_moves(int ns, int nh, int64_t n, const uint32_t* bits, const T* tt, const qes_hamiltonian* ham,
                             const T* Ct, const T* St, const T* A, float2* partial, cudaStream_t st) {
  auto blocks = [&](int rs) {
    return (int64_t)eloc_kblocks(ham->n_moves) * ((n + rs * ELT_ROWS - 1) / (rs * ELT_ROWS));
  };
  if constexpr (!ScalarTraits<T>::is_complex)
    if (blocks(4) >= 2 * 148) return launch_eloc_tiles<T, 4>(ns, nh, n, bits, tt, ham, Ct, St, A, partial, st);
  if (blocks(2) >= 2 * 148) return launch_eloc_tiles<T, 2>(ns, nh, n, bits, tt, ham, Ct, St, A, partial, st);
  return launch_eloc_tiles<T, 1>(ns, nh, n, bits, tt, ham, Ct, St, A, partial, st);
}

// diagonal part + move partials of sample s
QES_D void eloc_reduce_sample(int64_t s, int ns, int64_t n_samples, const uint32_t* __restrict__ bits, int nkb,
                              const float2* __restrict__ partial, int n_zf, const int32_t* __restrict__ zf_site,
                              const float* __restrict__ zf_h, int n_zz, const int32_t* __restrict__ zz_i,
                              const int32_t* __restrict__ zz_j, const float* __restrict__ zz_J,
                              float2* __restrict__ eloc) {
  const int nw = n_words(ns);
  const uint32_t* w = bits + s * nw;
  float d = 0.f;
  for (int t = 0; t < n_zf; ++t) d += zf_h[t] * sigma_of(w, zf_site[t]);
  for (int t = 0; t < n_zz; ++t) d += zz_J[t] * ((bit_of(w, zz_i[t]) == bit_of(w, zz_j[t])) ? 1.f : -1.f);
  float2 e = make_float2(d, 0.f);
  for (int b = 0; b < nkb; ++b) e = e + partial[(int64_t)b * n_samples + s];
  eloc[s] = e;
}

// A thread per sample, the terms in order.  Spin words and the terms are staged in shared memory (word-major and
// 128 terms at a time): reading both through L1 for each of the 800 bonds of a 20x20 lattice left the
// threads waiting on loads.
constexpr int ELR_THREADS = 64, ELR_TERMS = 128, ELR_WORDS = 64;     // more words than this are read from global memory
__global__ void __launch_bounds__(ELR_THREADS) eloc_reduce_kernel(int ns, int64_t n_samples, const uint32_t* __restrict__ bits,
                                                                 int nkb, const float2* __restrict__ partial, int n_zf,
                                                                 const int32_t* __restrict__ zf_site,
                                                                 const float* __restrict__ zf_h, int n_zz,
                                                                 const int32_t* __restrict__ zz_i,
                                                                 const int32_t* __restrict__ zz_j,
                                                                 const float* __restrict__ zz_J,
                                                                 float2* __restrict__ eloc) {
  __shared__ uint32_t s_w[ELR_WORDS][ELR_THREADS];
  __shared__ int2 s_ij[ELR_TERMS];
  __shared__ float s_J[ELR_TERMS];
  const int tid = threadIdx.x, nw = n_words(ns);
  const int64_t s0 = (int64_t)blockIdx.x * ELR_THREADS, s = s0 + tid;
  const int rows = (int)min((int64_t)ELR_THREADS, n_samples - s0);
  const bool staged = nw <= ELR_WORDS;
  if (staged)
    for (int e = tid; e < rows * nw; e += ELR_THREADS) s_w[e % nw][e / nw] = bits[s0 * nw + e];
  const uint32_t* gw = bits + (s < n_samples ? s : s0) * nw;
  auto bit = [&](int i) { return ((staged ? s_w[i >> 5][tid] : gw[i >> 5]) >> (i & 31)) & 1u; };
  float d = 0.f;
  for (int t0 = 0; t0 < n_zf + n_zz; t0 += ELR_TERMS) {
    __syncthreads();                                                 // words staged; previous terms consumed
    for (int q = tid; q < ELR_TERMS && t0 + q < n_zf + n_zz; q += ELR_THREADS) {
      const int t = t0 + q;
      s_ij[q] = t < n_zf ? make_int2(zf_site[t], -1) : make_int2(zz_i[t - n_zf], zz_j[t - n_zf]);
      s_J[q] = t < n_zf ? zf_h[t] : zz_J[t - n_zf];
    }
    __syncthreads();
    const int nt = min(ELR_TERMS, n_zf + n_zz - t0);
#pragma unroll 4
    for (int q = 0; q < nt; ++q) {
      const int2 ij = s_ij[q];
      const uint32_t bi = bit(ij.x), bj = ij.y < 0 ? 1u : bit(ij.y);
      d += s_J[q] * (bi == bj ? 1.f : -1.f);                         // a field term: sigma_i
    }
  }
  if (s >= n_samples) return;
  float2 e = make_float2(d, 0.f);
  for (int b = 0; b < nkb; ++b) e = e + partial[(int64_t)b * n_samples + s];
  eloc[s] = e;
}

extern "C" int qes_local_energy_workspace_bytes(int dtype, int ns, int nh, int64_t n_samples, int n_moves,
                                                size_t* bytes) {
  QES_ARG_CHECK(bytes != nullptr && n_samples >= 0 && n_moves >= 0, "qes_local_energy_workspace_bytes: bad args");
  (void)dtype; (void)ns; (void)nh;
  *bytes = (size_t)eloc_kblocks(n_moves) * (size_t)n_samples * sizeof(float2);
  return QES_OK;
}

extern "C" int qes_local_energy(int dtype, int ns, int nh, int64_t n_samples, const uint32_t* bits,
                                const void* tanh_theta, const qes_hamiltonian* ham, const void* Ct, const void* St,
                                const void* A, void* workspace, size_t workspace_bytes, void* eloc_out,
                                void* stream) {
  QES_ARG_CHECK(ham != nullptr && ns > 0 && nh > 0 && n_samples >= 0, "qes_local_energy: bad sizes");
  QES_ARG_CHECK(dtype == QES_DTYPE_F32 || dtype == QES_DTYPE_C64, "qes_local_energy: bad dtype");
  if (n_samples == 0) return QES_OK;
  QES_ARG_CHECK(bits && eloc_out, "qes_local_energy: null pointer");
  const int K = ham->n_moves;
  size_t need = 0;
  qes_local_energy_workspace_bytes(dtype, ns, nh, n_samples, K, &need);
  if (workspace_bytes < need || (need > 0 && workspace == nullptr)) {
    qes_set_last_message("qes_local_energy: workspace too small");
    return QES_ERR_WORKSPACE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  float2* partial = (float2*)workspace;
  if (K > 0) {
    QES_ARG_CHECK(tanh_theta && Ct && St && A && ham->move_i && ham->move_j && ham->move_kind && ham->move_coef,
                  "qes_local_energy: null move pointer");
    const int rc = dtype == QES_DTYPE_F32
                       ? launch_eloc_moves<float>(ns, nh, n_samples, bits, (const float*)tanh_theta, ham, (const float*)Ct,
                                                  (const float*)St, (const float*)A, partial, st)
                       : launch_eloc_moves<float2>(ns, nh, n_samples, bits, (const float2*)tanh_theta, ham,
                                                   (const float2*)Ct, (const float2*)St, (const float2*)A, partial, st);
    if (rc) return rc;
  }
  eloc_reduce_kernel<<<(unsigned)((n_samples + ELR_THREADS - 1) / ELR_THREADS), ELR_THREADS, 0, st>>>(
      ns, n_samples, bits, K > 0 ? eloc_kblocks(K) : 0, partial, ham->n_zfield, ham->zf_site, ham->zf_h, ham->n_zz, ham->zz_i,
      ham->zz_j, ham->zz_J, (float2*)eloc_out);
  QES_LAUNCH_CHECK();
  return QES_OK;
}

// ----------------------------------------------------------------------------
// float64 statistics of E_loc: mean (complex), variance and std of E_loc,
// Kahan-compensated per thread, then a fixed-order block tree.
// ----------------------------------------------------------------------------
constexpr int STATS_THREADS = 256;
constexpr int STATS_BLOCKS = 148;

__global__ void stats_pass1(int64_t n, const float2* __restrict__ e, const float* __restrict__ w,
                            double* __restrict__ part /* [blocks][4] : sw, swre, swim */) {
  double s0 = 0, s1 = 0, s2 = 0, c0 = 0, c1 = 0, c2 = 0;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    const double wk = w ? (double)w[k] : 1.0;
    const double y0 = wk - c0, y1 = wk * (double)e[k].x - c1, y2 = wk * (double)e[k].y - c2;
    const double t0 = s0 + y0, t1 = s1 + y1, t2 = s2 + y2;
    c0 = (t0 - s0) - y0; c1 = (t1 - s1) - y1; c2 = (t2 - s2) - y2;
    s0 = t0; s1 = t1; s2 = t2;
  }
  __shared__ double red[3][STATS_THREADS];
  red[0][threadIdx.x] = s0; red[1][threadIdx.x] = s1; red[2][threadIdx.x] = s2;
  __syncthreads();
  for (int o = STATS_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o)
      for (int q = 0; q < 3; ++q) red[q][threadIdx.x] += red[q][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int q = 0; q < 3; ++q) part[blockIdx.x * 4 + q] = red[q][0];
}

// The blocks' partials are added in order, by one thread, from shared memory (one thread walking them in global
// memory took 9-12 us for the mean and 6-8 for the variance, a quarter of a small batch's step); every block of the
// second pass forms the mean itself.
__global__ void stats_pass2(int64_t n, const float2* __restrict__ e, const float* __restrict__ w,
                            double* __restrict__ part, double* __restrict__ out) {
  __shared__ double pm[2][STATS_BLOCKS], mean[2];
  for (int b = threadIdx.x; b < STATS_BLOCKS; b += blockDim.x) { pm[0][b] = part[b * 4 + 1]; pm[1][b] = part[b * 4 + 2]; }
  __syncthreads();
  if (threadIdx.x < 2) {
    double m = 0;
#pragma unroll 4
    for (int b = 0; b < STATS_BLOCKS; ++b) m += pm[threadIdx.x][b];
    m /= (double)n;                          // weights are normalised to sum n
    mean[threadIdx.x] = m;
    if (blockIdx.x == 0) out[threadIdx.x] = m;
  }
  __syncthreads();
  const double mr = mean[0], mi = mean[1];
  double s = 0, c = 0;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    const double wk = w ? (double)w[k] : 1.0;
    const double dr = (double)e[k].x - mr, di = (double)e[k].y - mi;
    const double y = wk * (dr * dr + di * di) - c;
    const double t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __shared__ double red[STATS_THREADS];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = STATS_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x * 4 + 3] = red[0];
}

__global__ void stats_final(int64_t n, const double* __restrict__ part, double* __restrict__ out) {
  __shared__ double p[STATS_BLOCKS];
  for (int b = threadIdx.x; b < STATS_BLOCKS; b += blockDim.x) p[b] = part[b * 4 + 3];
  __syncthreads();
  if (threadIdx.x != 0) return;
  double v = 0;
#pragma unroll 4
  for (int b = 0; b < STATS_BLOCKS; ++b) v += p[b];
  v /= (double)n;
  out[2] = v;
  out[3] = sqrt(v);
}

extern "C" int qes_loss_stats_workspace_bytes(int64_t n_samples, size_t* bytes) {
  QES_ARG_CHECK(bytes != nullptr && n_samples >= 0, "qes_loss_stats_workspace_bytes: bad args");
  *bytes = (size_t)STATS_BLOCKS * 4 * sizeof(double);
  return QES_OK;
}

extern "C" int qes_loss_stats(int64_t n_samples, const void* eloc, const float* probs, double* out, void* workspace,
                              size_t workspace_bytes, void* stream) {
  QES_ARG_CHECK(n_samples > 0 && eloc && out, "qes_loss_stats: bad args");
  if (workspace_bytes < (size_t)STATS_BLOCKS * 4 * sizeof(double) || !workspace) {
    qes_set_last_message("qes_loss_stats: workspace too small");
    return QES_ERR_WORKSPACE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  double* part = (double*)workspace;
  stats_pass1<<<STATS_BLOCKS, STATS_THREADS, 0, st>>>(n_samples, (const float2*)eloc, probs, part);
  stats_pass2<<<STATS_BLOCKS, STATS_THREADS, 0, st>>>(n_samples, (const float2*)eloc, probs, part, out);
  stats_final<<<1, STATS_THREADS, 0, st>>>(n_samples, part, out);
  QES_LAUNCH_CHECK_N(3);
  return QES_OK;
}

// ----------------------------------------------------------------------------
// Step diagnostics: Gelman-Rubin R-hat over n_groups contiguous blocks of
// Re E_loc and sigma^2 = var(Re E_loc) (uniform weights, ddof 0), float64.
// One warp per block computes its mean and ddof-1 variance (two passes); a
// single CTA then combines the blocks in a fixed order.
// ----------------------------------------------------------------------------
constexpr int RHAT_FINAL_THREADS = 1024;

__global__ void rhat_groups_kernel(int64_t n_groups, int64_t glen, const float2* __restrict__ e,
                                   double2* __restrict__ gstat) {
  const int lane = threadIdx.x & 31;
  const int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (g >= n_groups) return;
  const float2* x = e + g * glen;
  double s = 0;
  for (int64_t k = lane; k < glen; k += 32) s += (double)x[k].x;
  const double m = warp_sum(s) / (double)glen;
  double v = 0;
  for (int64_t k = lane; k < glen; k += 32) {
    const double d = (double)x[k].x - m;
    v += d * d;
  }
  v = warp_sum(v);
  if (lane == 0) gstat[g] = make_double2(m, glen > 1 ? v / (double)(glen - 1) : 0.0);
}

__global__ void __launch_bounds__(RHAT_FINAL_THREADS) rhat_final_kernel(int64_t n_groups, int64_t glen, int valid,
                                                                      const double2* __restrict__ gstat,
                                                                      double* __restrict__ out) {
  __shared__ double red[2][RHAT_FINAL_THREADS];
  double sm = 0, sv = 0;
  for (int64_t g = threadIdx.x; g < n_groups; g += blockDim.x) { sm += gstat[g].x; sv += gstat[g].y; }
  red[0][threadIdx.x] = sm; red[1][threadIdx.x] = sv;
  __syncthreads();
  for (int o = RHAT_FINAL_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) { red[0][threadIdx.x] += red[0][threadIdx.x + o]; red[1][threadIdx.x] += red[1][threadIdx.x + o]; }
    __syncthreads();
  }
  const double mm = red[0][0] / (double)n_groups;   // grand mean (equal block lengths)
  const double W = red[1][0] / (double)n_groups;    // mean within-block variance
  __syncthreads();
  double sb = 0;
  for (int64_t g = threadIdx.x; g < n_groups; g += blockDim.x) {
    const double d = gstat[g].x - mm;
    sb += d * d;
  }
  red[0][threadIdx.x] = sb;
  __syncthreads();
  for (int o = RHAT_FINAL_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[0][threadIdx.x] += red[0][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double L = (double)glen, G = (double)n_groups, ssb = red[0][0];
    // total variance of the n = G*L values, ddof 0: within + between blocks
    out[1] = ((L - 1.0) * W * G + L * ssb) / (G * L);
    if (valid) {
      const double B = L * ssb / (G - 1.0);
      const double var_hat = ((L - 1.0) / L) * W + B / L;
      out[0] = sqrt(var_hat / fmax(W, 1e-12));
    } else {
      out[0] = nan("");
    }
  }
}

extern "C" int qes_loss_rhat_workspace_bytes(int64_t n_samples, int n_chains, size_t* bytes) {
  QES_ARG_CHECK(bytes != nullptr && n_samples >= 0, "qes_loss_rhat_workspace_bytes: bad args");
  *bytes = (size_t)std::max<int64_t>(1, std::max<int64_t>(n_chains, 1)) * sizeof(double2);
  return QES_OK;
}

extern "C" int qes_loss_rhat(int64_t n_samples, int n_chains, const void* eloc, double* out, void* workspace,
                             size_t workspace_bytes, void* stream) {
  QES_ARG_CHECK(n_samples > 0 && eloc && out && workspace, "qes_loss_rhat: bad args");
  const int64_t nch = std::max(n_chains, 1);
  const bool valid = nch > 1 && n_samples > nch && n_samples % nch == 0 && n_samples / nch > 1;
  const int64_t G = valid ? nch : 1, L = n_samples / G;
  if (workspace_bytes < (size_t)G * sizeof(double2)) {
    qes_set_last_message("qes_loss_rhat: workspace too small");
    return QES_ERR_WORKSPACE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  double2* gstat = (double2*)workspace;
  const int warps = 8;
  rhat_groups_kernel<<<(unsigned)((G + warps - 1) / warps), 32 * warps, 0, st>>>(G, L, (const float2*)eloc, gstat);
  rhat_final_kernel<<<1, RHAT_FINAL_THREADS, 0, st>>>(G, L, valid ? 1 : 0, gstat, out);
  QES_LAUNCH_CHECK_N(2);
  return QES_OK;
}

// ----------------------------------------------------------------------------
// Allocation-free local energy.
//
// Some callers cannot allocate device memory at all: hosts that hand this
// library a fixed device budget at start-up and forbid cudaMalloc afterwards,
// latency-critical loops where cudaMalloc's implicit device synchronisation is
// not acceptable, and foreign-language bindings (cgo, JNI, plain C) that have
// no allocator of their own to hand out scratch buffers.  For them this entry
// point keeps the local energy's only scratch -- one float2 partial sum per
// (32-move block, sample) -- in a fixed array compiled into the library.
//
// The array lives in every GPU that loads the library until the process
// exits.  The host never dereferences the symbol itself: the array's device
// address is looked up with cudaGetSymbolAddress on the first call made on
// each device (with that device current) and cached, so that first call per
// device should come before any stream capture.  All calls share the one
// array: each call overwrites the part it reads before reading it, so no
// clearing is needed, but calls that overlap on the GPU (several streams or
// host threads at once) race on it and must be serialised by the caller.
// ----------------------------------------------------------------------------
#include <mutex>

static __device__ __align__(256) float2 g_eloc_noalloc_scratch[QES_NOALLOC_ELOC_SCRATCH_BYTES / sizeof(float2)];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
void* g_noalloc_ptr[kMaxDevices] = {};
}  // namespace

static int eloc_noalloc_scratch(void** out) {
  int dev = -1;
  QES_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) {
    qes_set_last_message("qes_local_energy_noalloc: device ordinal beyond the supported 64");
    return QES_ERR_SIZE;
  }
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (g_noalloc_ptr[dev] == nullptr) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_eloc_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) {
      qes_set_last_error(e, "qes_local_energy_noalloc: cudaGetSymbolAddress of the static scratch");
      return QES_ERR_CUDA;
    }
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return QES_OK;
}

extern "C" int qes_local_energy_noalloc(int dtype, int ns, int nh, int64_t n_samples, const uint32_t* bits,
                                        const void* tanh_theta, const qes_hamiltonian* ham, const void* Ct,
                                        const void* St, const void* A, void* eloc_out, void* stream) {
  QES_ARG_CHECK(ham != nullptr && ns > 0 && nh > 0 && n_samples >= 0, "qes_local_energy_noalloc: bad sizes");
  size_t need = 0;
  const int rc0 = qes_local_energy_workspace_bytes(dtype, ns, nh, n_samples, ham->n_moves, &need);
  if (rc0 != QES_OK) return rc0;
  if (need > (size_t)QES_NOALLOC_ELOC_SCRATCH_BYTES) {
    qes_set_last_message("qes_local_energy_noalloc: ceil(n_moves/32) * n_samples * 8 bytes exceeds the "
                         "8 MiB static scratch; use qes_local_energy with a caller workspace");
    return QES_ERR_SIZE;
  }
  void* scratch = nullptr;
  const int rc = eloc_noalloc_scratch(&scratch);
  if (rc != QES_OK) return rc;
  return qes_local_energy(dtype, ns, nh, n_samples, bits, tanh_theta, ham, Ct, St, A, scratch,
                          (size_t)QES_NOALLOC_ELOC_SCRATCH_BYTES, eloc_out, stream);
}

// ----------------------------------------------------------------------------
// Batched problems
// ----------------------------------------------------------------------------
// move items (b, move block, sample block)
template <class T>
__global__ void __launch_bounds__(32 * ELOC_ROWS) batch_eloc_moves_kernel(
    const qes_batch_instance* __restrict__ inst, const int4* __restrict__ items, const uint32_t* __restrict__ bits,
    const T* __restrict__ tanh_theta, const int32_t* __restrict__ mi, const int32_t* __restrict__ mj,
    const int32_t* __restrict__ mkind, const float4* __restrict__ mcoef, const T* __restrict__ Ct,
    const T* __restrict__ St, const T* __restrict__ A, float2* __restrict__ partial) {
  const int4 it = items[blockIdx.x];
  const qes_batch_instance I = inst[it.x];
  const int64_t rows = (int64_t)I.n_chains * I.num_samples;
  eloc_moves_block<T>(it.y, it.z, I.ns, I.nh, rows, bits + I.sample_word_off, tanh_theta + I.tanh_off, I.n_moves,
                      mi + I.move_off, mj + I.move_off, mkind + I.move_off, mcoef + I.move_off,
                      Ct + I.move_table_off, St + I.move_table_off, A + I.move_off, partial + I.eloc_part_off);
}

// reduce items (b, sample block of 256)
__global__ void batch_eloc_reduce_kernel(const qes_batch_instance* __restrict__ inst, const int4* __restrict__ items,
                                         const uint32_t* __restrict__ bits, const float2* __restrict__ partial,
                                         const int32_t* __restrict__ zf_site, const float* __restrict__ zf_h,
                                         const int32_t* __restrict__ zz_i, const int32_t* __restrict__ zz_j,
                                         const float* __restrict__ zz_J, float2* __restrict__ eloc) {
  const int4 it = items[blockIdx.x];
  const qes_batch_instance I = inst[it.x];
  const int64_t rows = (int64_t)I.n_chains * I.num_samples;
  const int64_t s = (int64_t)it.y * blockDim.x + threadIdx.x;
  if (s >= rows) return;
  eloc_reduce_sample(s, I.ns, rows, bits + I.sample_word_off, I.n_moves > 0 ? eloc_kblocks(I.n_moves) : 0,
                     partial + I.eloc_part_off, I.n_zfield, zf_site + I.zf_off, zf_h + I.zf_off, I.n_zz,
                     zz_i + I.zz_off, zz_j + I.zz_off, zz_J + I.zz_off, eloc + I.sample_off);
}

extern "C" int qes_batch_local_energy(int dtype, int n_inst, const qes_batch_instance* inst, int n_move_items,
                                      const int32_t* move_items, int n_red_items, const int32_t* red_items,
                                      const uint32_t* sample_bits, const void* tanh_theta, const int32_t* move_i,
                                      const int32_t* move_j, const int32_t* move_kind, const float* move_coef,
                                      const void* Ct, const void* St, const void* A, const int32_t* zf_site,
                                      const float* zf_h, const int32_t* zz_i, const int32_t* zz_j,
                                      const float* zz_J, void* partial, void* eloc_out, void* stream) {
  QES_ARG_CHECK(dtype == QES_DTYPE_F32 || dtype == QES_DTYPE_C64, "qes_batch_local_energy: bad dtype");
  QES_ARG_CHECK(n_inst >= 0 && n_move_items >= 0 && n_red_items >= 0, "qes_batch_local_energy: bad sizes");
  if (n_red_items == 0) return QES_OK;
  QES_ARG_CHECK(inst && red_items && sample_bits && eloc_out, "qes_batch_local_energy: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  if (n_move_items > 0) {
    QES_ARG_CHECK(move_items && tanh_theta && move_i && move_j && move_kind && move_coef && Ct && St && A && partial,
                  "qes_batch_local_energy: null move pointer");
    dim3 block(32, ELOC_ROWS);
    if (dtype == QES_DTYPE_F32)
      batch_eloc_moves_kernel<float><<<n_move_items, block, 0, st>>>(
          inst, (const int4*)move_items, sample_bits, (const float*)tanh_theta, move_i, move_j, move_kind,
          (const float4*)move_coef, (const float*)Ct, (const float*)St, (const float*)A, (float2*)partial);
    else
      batch_eloc_moves_kernel<float2><<<n_move_items, block, 0, st>>>(
          inst, (const int4*)move_items, sample_bits, (const float2*)tanh_theta, move_i, move_j, move_kind,
          (const float4*)move_coef, (const float2*)Ct, (const float2*)St, (const float2*)A, (float2*)partial);
    QES_LAUNCH_CHECK();
  }
  batch_eloc_reduce_kernel<<<n_red_items, 256, 0, st>>>(inst, (const int4*)red_items, sample_bits,
                                                        (const float2*)partial, zf_site, zf_h, zz_i, zz_j, zz_J,
                                                        (float2*)eloc_out);
  QES_LAUNCH_CHECK();
  return QES_OK;
}

// one block per problem: float64 mean (complex), variance, std of its E_loc rows (uniform weights)
constexpr int BSTAT_THREADS = 256;
__global__ void __launch_bounds__(BSTAT_THREADS) batch_stats_kernel(const qes_batch_instance* __restrict__ inst,
                                                                   const float2* __restrict__ eloc,
                                                                   double* __restrict__ out) {
  const qes_batch_instance I = inst[blockIdx.x];
  const int64_t rows = (int64_t)I.n_chains * I.num_samples;
  const float2* e = eloc + I.sample_off;
  __shared__ double red[2][BSTAT_THREADS];
  double sr = 0, si = 0;
  for (int64_t k = threadIdx.x; k < rows; k += blockDim.x) { sr += e[k].x; si += e[k].y; }
  red[0][threadIdx.x] = sr; red[1][threadIdx.x] = si;
  __syncthreads();
  for (int o = BSTAT_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) { red[0][threadIdx.x] += red[0][threadIdx.x + o]; red[1][threadIdx.x] += red[1][threadIdx.x + o]; }
    __syncthreads();
  }
  const double n = (double)(rows > 0 ? rows : 1);
  const double mr = red[0][0] / n, mi = red[1][0] / n;
  __syncthreads();
  double v = 0;
  for (int64_t k = threadIdx.x; k < rows; k += blockDim.x) {
    const double dr = e[k].x - mr, di = e[k].y - mi;
    v += dr * dr + di * di;
  }
  red[0][threadIdx.x] = v;
  __syncthreads();
  for (int o = BSTAT_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[0][threadIdx.x] += red[0][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double var = red[0][0] / n;
    out[4 * blockIdx.x + 0] = mr;
    out[4 * blockIdx.x + 1] = mi;
    out[4 * blockIdx.x + 2] = var;
    out[4 * blockIdx.x + 3] = sqrt(var);
  }
}

extern "C" int qes_batch_loss_stats(int n_inst, const qes_batch_instance* inst, const void* eloc, double* out,
                                    void* stream) {
  QES_ARG_CHECK(n_inst >= 0, "qes_batch_loss_stats: bad sizes");
  if (n_inst == 0) return QES_OK;
  QES_ARG_CHECK(inst && eloc && out, "qes_batch_loss_stats: null pointer");
  batch_stats_kernel<<<n_inst, BSTAT_THREADS, 0, (cudaStream_t)stream>>>(inst, (const float2*)eloc, out);
  QES_LAUNCH_CHECK();
  return QES_OK;
}
