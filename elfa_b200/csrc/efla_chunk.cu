// EFLA recurrence in chunks of 32 tokens on the tensor cores.
//
// Per (batch, head) with state S [d, d] (row = key index, column = value index), K, V [32, d] the tokens of a chunk, lam_t = |k_t|^2,
// c_t = (1 - exp(-beta lam_t)) / lam_t and ex_t = 1 - c_t lam_t = exp(-beta lam_t), the recurrence S += c k (v - S^T k)^T of the chunk is
//   E0 = V - K S0          errors against the state at the chunk's start
//   E  = (I + strict_lower(K K^T) diag(c))^{-1} E0 = E0 + N E0,  N strictly lower triangular and independent of the state
//   O  = V - diag(ex) E    (o_t = S_t^T k_t)
//   S1 = S0 + K^T diag(c) E
// (the WY form of a product of rank-one updates). efla_prep_kernel computes N, c and ex of all chunks in parallel, one warp each;
// efla_chunk_fwd_kernel walks the chunks with the state in registers.
//
// Precision: the state, E0, E and N are fp32. K and V are bf16 as given; every fp32 operand of a product enters as the sum of three bf16
// numbers (24 bits, exact), products of two split operands keep the six terms above 2^-24, the accumulators are fp32, and both E and S are
// updated by one fp32 addition per chunk, so the error of the state is that of the token-by-token fp32 recurrence or smaller
// (64-bit comparison at T 2048, 16 heads of 64: 2.2e-7 relative; token by token 2.4e-7).
//
// Values that are not finite: as in the recurrence, one in K or V reaches its own token and later ones, one in dO its own token and earlier
// ones, and V and dO their own columns only (for dV; a row of dK adds up all columns). Inside a chunk the products of the chunked form
// would carry 0 x NaN to the other tokens, so every kernel asks at its end whether a state or a key gradient came out not finite and, if so,
// runs once more in a checked form that walks the chunks concerned token by token (efla_walk) and overwrites its results. On finite data
// that costs one barrier. (Asked for inside the walk over the chunks it stood in the chain of dependent products: forward 105 us against 94,
// state gradient 98 against 92 at B 8, T 2048, 16 heads of 64, when it was moved.) Gradients of such tokens are not finite; whether infinity or NaN is not kept.
//
// reference: kernels/cuda/efla.cu:121-271,534-552 (chunks are scanned one after the other, the bf16 state in global memory).
#include <algorithm>

#include "common.cuh"
#include "elfa_native.h"
#include "mma_sync.cuh"

namespace elfa {
namespace {

constexpr int EC = 32;                     // tokens of a chunk
constexpr int EN_LD = 40;                  // row pitch of a warp's split tiles in shared memory (bf16)
constexpr int EN_ELEMS = 3 * EC * EC;      // one chunk's N: [split][t][s] bf16, the four 16-byte pieces of a row exchanged (efla_n_piece)
constexpr int EC_COEF = 4 * EC;            // one chunk's coefficients in global memory

// Byte offset of piece c (columns 8 c ..) of row t of one split of N, in global and in shared memory alike: eight rows of 64 bytes, read at one
// piece by ldmatrix, lie in different banks, and a chunk's N is one contiguous copy
__device__ __forceinline__ int efla_n_piece(int t, int c) { return t * 64 + ((c ^ (t >> 1 & 3)) << 4); }

// ------------------------------------------------------------------------------------------------ state-independent part
// One warp per (batch, head, chunk): Gram matrix by mma.sync (exact bf16 products), then lane s eliminates column s of the unit
// lower triangular matrix by forward substitution in fp32 registers (496 multiply-adds, rows broadcast from shared memory).
// coef: [.., 0][t] = c, [1] = ex, [2] = lam, [3] = dc / dlam, evaluated in fp64 and rounded once (one exponential per token; the gradient of
// beta is a long sum of terms dc_t ex_t in which an error of lam or ex common to all tokens would not average out). Tokens past the
// end have k = 0: they change neither the state nor another token.
template <int D>
__global__ void __launch_bounds__(64) efla_prep_kernel(const __nv_bfloat16* __restrict__ k, const float* __restrict__ beta_ptr,
                                                       __nv_bfloat16* __restrict__ nmat, float* __restrict__ coef, int T, int H,
                                                       int nchunks, long long total) {
  constexpr int LD = D + 8;
  __shared__ __align__(16) __nv_bfloat16 sk_all[2][EC * LD];
  __shared__ __align__(16) float sg_all[2][EC][36];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const long long id = (long long)blockIdx.x * 2 + warp;
  if (id >= total) return;
  const int bh = (int)(id / nchunks), ch = (int)(id % nchunks), b = bh / H, h = bh % H;
  const int t0 = ch * EC, n = min(EC, T - t0);
  __nv_bfloat16* sk = sk_all[warp];
  float(*sg)[36] = sg_all[warp];
  const __nv_bfloat16* kb = k + (((long long)b * T + t0) * H + h) * D;
  uint4 kq[D / 8];                         // every load of the chunk in flight before the first store
#pragma unroll
  for (int u = 0; u < D / 8; ++u) {
    const int i = u * 32 + lane, r = i / (D / 8), c = i % (D / 8);
    kq[u] = make_uint4(0, 0, 0, 0);
    if (r < n) kq[u] = *reinterpret_cast<const uint4*>(kb + (long long)r * H * D + c * 8);
  }
#pragma unroll
  for (int u = 0; u < D / 8; ++u) {
    const int i = u * 32 + lane, r = i / (D / 8), c = i % (D / 8);
    *reinterpret_cast<uint4*>(sk + r * LD + c * 8) = kq[u];
  }
  __syncwarp();
  const uint32_t ks = smem_u32(sk);
#pragma unroll
  for (int mi = 0; mi < 2; ++mi) {
    float acc[4][4];
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      uint32_t a[4];
      ldsm4(a, ks + ((mi * 16 + (lane & 15)) * LD + kk * 16 + (lane >> 4) * 8) * 2);
#pragma unroll
      for (int np = 0; np <= mi; ++np) {   // token columns 16 np .. 16 np + 15: the strictly upper tiles are not needed
        uint32_t bq[4];
        ldsm4(bq, ks + ((np * 16 + (lane & 7) + (lane >> 4) * 8) * LD + kk * 16 + ((lane >> 3) & 1) * 8) * 2);
        if (kk == 0) {
          mma_bf16_first(acc[2 * np], a, bq[0], bq[1]);
          mma_bf16_first(acc[2 * np + 1], a, bq[2], bq[3]);
        } else {
          mma_bf16(acc[2 * np], a, bq[0], bq[1]);
          mma_bf16(acc[2 * np + 1], a, bq[2], bq[3]);
        }
      }
    }
#pragma unroll
    for (int nj = 0; nj < 2 * mi + 2; ++nj) {
      *reinterpret_cast<float2*>(&sg[mi * 16 + g][nj * 8 + 2 * q]) = make_float2(acc[nj][0], acc[nj][1]);
      *reinterpret_cast<float2*>(&sg[mi * 16 + g + 8][nj * 8 + 2 * q]) = make_float2(acc[nj][2], acc[nj][3]);
    }
  }
  __syncwarp();
  double lam = 0.;
#pragma unroll
  for (int i = 0; i < D / 8; ++i) {
    const uint4 v = *reinterpret_cast<const uint4*>(sk + lane * LD + i * 8);
    const uint32_t* pv = reinterpret_cast<const uint32_t*>(&v);
    float p[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) p[j] = bf16_lo(pv[j]) * bf16_lo(pv[j]) + bf16_hi(pv[j]) * bf16_hi(pv[j]);
    lam += (double)((p[0] + p[1]) + (p[2] + p[3]));
  }
  const double beta = *beta_ptr, x_ = beta * lam;
  double c, ex, dl;
  if (fabs(x_) < 1e-3) {                   // series: 1 - ex would cancel
    c = beta * (1. - x_ * (0.5 - x_ * (1. / 6. - x_ / 24.)));
    ex = 1. - c * lam;
    dl = beta * beta * (x_ * (1. / 3. - x_ / 8.) - 0.5);
  } else {
    const double inv = 1. / lam;
    ex = exp(-x_);
    c = (1. - ex) * inv;
    dl = (beta * ex - c) * inv;
  }
  const float c_ = (float)c;
  float* cf = coef + id * EC_COEF;
  cf[lane] = c_;
  cf[EC + lane] = (float)ex;
  cf[2 * EC + lane] = (float)lam;
  cf[3 * EC + lane] = (float)dl;
  __syncwarp();
  for (int t = 0; t < EC; ++t)
    if (lane < t) sg[t][lane] *= c_;       // A[t][r] = G[t][r] c_r
  __syncwarp();
  // column `lane` of (I + A)^{-1}: x_t = [t == lane] - sum_{r < t} A[t][r] x_r
  float x[EC];
#pragma unroll
  for (int t = 0; t < EC; ++t) {
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
    for (int r = 0; r + 3 < t; r += 4) {
      const float4 a = *reinterpret_cast<const float4*>(&sg[t][r]);
      s0 += a.x * x[r];
      s1 += a.y * x[r + 1];
      s2 += a.z * x[r + 2];
      s3 += a.w * x[r + 3];
    }
#pragma unroll
    for (int r = t / 4 * 4; r < t; ++r) s0 += sg[t][r] * x[r];
    const float s = (s0 + s1) + (s2 + s3);
    x[t] = t < lane ? 0.f : (t == lane ? 1.f : -s);
  }
  // neighbouring lanes trade halves so that a store carries two columns: even lanes write row t, odd lanes row t + 1
  uint32_t* out = reinterpret_cast<uint32_t*>(nmat + id * EN_ELEMS) + (lane >> 1 & 3);
  auto put = [&](int split, int t, uint32_t v) {
    const uint32_t w = __shfl_xor_sync(0xffffffffu, v, 1);
    out[split * (EC * EC / 2) + efla_n_piece(t + (lane & 1), lane >> 3) / 4] = (lane & 1) ? __byte_perm(w, v, 0x7632) : __byte_perm(v, w, 0x5410);
  };
#pragma unroll
  for (int t = 0; t < EC; t += 2) {
    uint32_t hi, mid, lo;
    split3(t > lane ? x[t] : 0.f, t + 1 > lane ? x[t + 1] : 0.f, hi, mid, lo);
    put(0, t, hi);
    put(1, t, mid);
    put(2, t, lo);
  }
}

// ------------------------------------------------------------------------------------------------ sequential part
// Warps per CTA: each owns 16 value columns and all d key rows of the state, as the accumulator tiles of S^T (16 x d), so that the
// products of a chunk chain through registers and warps exchange nothing. The CTA shares the staged K / N tiles of its head.
template <int D> constexpr int ec_warps() { return D == 32 ? 2 : (D == 96 ? 3 : 4); }
constexpr int EC_STAGES = 4;

template <int D>
struct EflaStage {                         // byte offsets inside one stage of the shared-memory ring
  static constexpr int VC = 16 * ec_warps<D>();
  static constexpr int KLD = D + 8, VLD = VC + 8;
  static constexpr int K = 0, V = K + EC * KLD * 2, N = V + EC * VLD * 2, C = N + EN_ELEMS * 2, BYTES = C + 2 * EC * 4;
};

// A thread's place in the copies of a chunk's K and V tiles: it takes 16 bytes of every KR-th row of K, every VR-th row of V. N and the
// coefficients are copied as they lie. With indices worked out per copy (and N in rows of a wider pitch) the copies took 690 of the 2600 cycles of a
// chunk to issue; the walks are chains that nothing hides it behind.
template <int D>
struct EflaLoader {
  using L = EflaStage<D>;
  static constexpr int NT = 32 * ec_warps<D>(), KR = NT / (D / 8), VR = NT / (L::VC / 8);
  static_assert(NT % (D / 8) == 0 && NT % (L::VC / 8) == 0 && EC % KR == 0 && EC % VR == 0, "whole passes");
  const __nv_bfloat16 *k, *v;              // this thread's vectors in the first chunk's first rows; v: null without values
  const __nv_bfloat16* n;
  const float* c;
  long long rs;
  uint32_t ring;
  int krow, vrow, T;
  __device__ __forceinline__ EflaLoader(const __nv_bfloat16* kb, const __nv_bfloat16* vb, const __nv_bfloat16* nb, const float* cb, long long rs_,
                                        uint32_t ring_, int T_)
      : n(nb + threadIdx.x * 8), c(cb + threadIdx.x * 4), rs(rs_), ring(ring_), krow(threadIdx.x / (D / 8)), vrow(threadIdx.x / (L::VC / 8)), T(T_) {
    k = kb + krow * rs + threadIdx.x % (D / 8) * 8;
    v = vb ? vb + vrow * rs + threadIdx.x % (L::VC / 8) * 8 : nullptr;
  }
  // chunk ch as the it-th of the ring's uses
  __device__ __forceinline__ void operator()(int it, int ch) const {
    const uint32_t st = ring + it % EC_STAGES * L::BYTES;
    const __nv_bfloat16* ns = n + (long long)ch * EN_ELEMS;
    static_assert(EN_ELEMS / 8 % NT == 0, "whole passes");
#pragma unroll
    for (int p = 0; p < EN_ELEMS / 8 / NT; ++p) cp_async16(st + L::N + (threadIdx.x + p * NT) * 16, ns + p * NT * 8, true);
    if (threadIdx.x < 2 * EC / 4) cp_async16(st + L::C + threadIdx.x * 16, c + (long long)ch * EC_COEF, true);
    const int rows = T - ch * EC;
    const long long at = (long long)ch * EC * rs;
    const uint32_t kd = st + L::K + (krow * L::KLD + threadIdx.x % (D / 8) * 8) * 2, vd = st + L::V + (vrow * L::VLD + threadIdx.x % (L::VC / 8) * 8) * 2;
    if (rows >= EC && v) {
      const __nv_bfloat16 *ks = k + at, *vs = v + at;
#pragma unroll
      for (int p = 0; p < EC / KR; ++p) cp_async16(kd + p * KR * L::KLD * 2, ks + p * KR * rs, true);
#pragma unroll
      for (int p = 0; p < EC / VR; ++p) cp_async16(vd + p * VR * L::VLD * 2, vs + p * VR * rs, true);
    } else {                               // rows past the end, and values where there are none, become zero
#pragma unroll
      for (int p = 0; p < EC / KR; ++p) {
        const bool in = krow + p * KR < rows;
        cp_async16(kd + p * KR * L::KLD * 2, in ? k + at + p * KR * rs : n, in);
      }
#pragma unroll
      for (int p = 0; p < EC / VR; ++p) {
        const bool in = v && vrow + p * VR < rows;
        cp_async16(vd + p * VR * L::VLD * 2, in ? v + at + p * VR * rs : n, in);
      }
    }
  }
};

// e += N e for a warp's 16 x 32 tile (four C tiles, columns = tokens): six products of the splits, small ones first.
// TRANS: the transposed matrix (e_r += sum_t N[t][r] e_t), for the gradient.
template <bool TRANS>
__device__ __forceinline__ void efla_apply_n(float (&e)[4][4], uint32_t nbase, int lane) {
  uint32_t ah[2][4], am[2][4], al[2][4];
#pragma unroll
  for (int ks = 0; ks < 2; ++ks) split3_a(ah[ks], am[ks], al[ks], e[2 * ks], e[2 * ks + 1]);
  // the four token tiles advance together: a dependent mma.sync waits for the one before it, and there is one warp per scheduler
  float acc[4][4];
#pragma unroll
  for (int p = 2; p >= 0; --p) {           // splits of N, small ones first
    uint32_t bf[4][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      if (TRANS) ldsm4_t(bf[nt], nbase + p * (EC * EC * 2) + efla_n_piece(lane, nt));        // rows t, columns r of tile nt
      else ldsm4(bf[nt], nbase + p * (EC * EC * 2) + efla_n_piece(nt * 8 + (lane & 7), lane >> 3));
    }
#pragma unroll
    for (int m = 2 - p; m >= 0; --m)       // splits of e that still count against this split of N
#pragma unroll
      for (int ks = 0; ks < 2; ++ks)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          if (TRANS ? (nt >= 2 && ks == 0) : (nt < 2 && ks == 1)) continue;                 // zero blocks of the triangle
          if (p == 2 && ks == (TRANS && nt >= 2)) mma_bf16_first(acc[nt], ah[ks], bf[nt][2 * ks], bf[nt][2 * ks + 1]);
          else mma_bf16(acc[nt], m == 0 ? ah[ks] : (m == 1 ? am[ks] : al[ks]), bf[nt][2 * ks], bf[nt][2 * ks + 1]);
        }
  }
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) put_pair(e[nt], hf, add_f32x2(pair_of(e[nt], hf), pair_of(acc[nt], hf)));
}

// p[16 x 32] = S^T K^T for the warp's S^T tiles (rows = value columns, columns = tokens)
template <int D>
__device__ __forceinline__ void efla_state_times_k(float (&p)[4][4], const float (&S)[D / 8][4], uint32_t kbase, int lane) {
  constexpr int LD = EflaStage<D>::KLD;
#pragma unroll
  for (int k2 = 0; k2 < D / 32; ++k2) {
    uint32_t bq[4][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) ldsm4(bq[nt], kbase + ((nt * 8 + (lane & 7)) * LD + k2 * 32 + (lane >> 3) * 8) * 2);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      uint32_t hi[4], mid[4], lo[4];
      split3_a(hi, mid, lo, S[4 * k2 + 2 * u], S[4 * k2 + 2 * u + 1]);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        if (k2 == 0 && u == 0) mma_bf16_first(p[nt], lo, bq[nt][0], bq[nt][1]);
        else mma_bf16(p[nt], lo, bq[nt][2 * u], bq[nt][2 * u + 1]);
      }
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) mma_bf16(p[nt], mid, bq[nt][2 * u], bq[nt][2 * u + 1]);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) mma_bf16(p[nt], hi, bq[nt][2 * u], bq[nt][2 * u + 1]);
    }
  }
}

// S^T (+/-)= u K for the warp's tiles, u [16 x 32] fp32; one fp32 addition per state element
template <int D, bool SUB>
__device__ __forceinline__ void efla_state_update(float (&S)[D / 8][4], const float (&u)[4][4], uint32_t kbase, int lane) {
  constexpr int LD = EflaStage<D>::KLD;
  uint32_t hi[2][4], mid[2][4], lo[2][4];
#pragma unroll
  for (int ks = 0; ks < 2; ++ks) split3_a(hi[ks], mid[ks], lo[ks], u[2 * ks], u[2 * ks + 1]);
#pragma unroll
  for (int n0 = 0; n0 < D / 8; n0 += 4) {  // four independent accumulator chains
    uint32_t bq[4][4];
    float acc[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n) ldsm4_t(bq[n], kbase + (lane * LD + (n0 + n) * 8) * 2);
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
      for (int ks = 0; ks < 2; ++ks)
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          if (p == 0 && ks == 0) mma_bf16_first(acc[n], lo[0], bq[n][0], bq[n][1]);
          else mma_bf16(acc[n], p == 0 ? lo[ks] : (p == 1 ? mid[ks] : hi[ks]), bq[n][2 * ks], bq[n][2 * ks + 1]);
        }
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const uint64_t s = pair_of(S[n0 + n], hf), a = pair_of(acc[n], hf);
        put_pair(S[n0 + n], hf, SUB ? fma_f32x2(a, pack_f32x2(-1.f, -1.f), s) : add_f32x2(s, a));
      }
  }
}

// One chunk token by token, for the columns in which a product of the chunked form is not finite: there 0 x NaN inside a product would reach
// tokens that the recurrence keeps apart. first[hf] is the token from which on value column g + 8 hf takes these results (EC: the column is
// left alone); its state rows walk all n tokens. Plain fp32 multiply-adds and a quad's shuffles: only the checked forms come here.
// sp: the state [D / 8][4] in local memory, read and written. OUT: outputs o_t = p + (1 - ex) e go to so [token][24]; otherwise the errors go
// to ep [4][4] in local memory.
template <int D, int KLD, int VLD, bool OUT>
__device__ __noinline__ void efla_walk(float* sp, float* ep, const __nv_bfloat16* sk, const __nv_bfloat16* sv, const float* cf,
                                       __nv_bfloat16* so, int first0, int first1, int n) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  float S[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 2; ++i) S[i / 4][i % 4] = sp[i];
#pragma unroll 1
  for (int t = 0; t < n; ++t) {
    float p0 = 0.f, p1 = 0.f;
#pragma unroll
    for (int i = 0; i < D / 8; ++i) {
      const float2 kk = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sk + t * KLD + i * 8 + 2 * q));
      p0 += kk.x * S[i][0] + kk.y * S[i][1];
      p1 += kk.x * S[i][2] + kk.y * S[i][3];
    }
#pragma unroll
    for (int m = 1; m < 4; m <<= 1) {
      p0 += __shfl_xor_sync(0xffffffffu, p0, m);
      p1 += __shfl_xor_sync(0xffffffffu, p1, m);
    }
    const float c = cf[t], w = 1.f - cf[EC + t];
    const float e0 = __bfloat162float(sv[t * VLD + g]) - p0, e1 = __bfloat162float(sv[t * VLD + g + 8]) - p1;
    const bool put = OUT ? q == 0 : q == (t & 7) >> 1;
    if (put && t >= first0) {
      if (OUT) so[t * 24 + g] = __float2bfloat16(p0 + w * e0);
      else ep[(t >> 3) * 4 + (t & 1)] = e0;
    }
    if (put && t >= first1) {
      if (OUT) so[t * 24 + g + 8] = __float2bfloat16(p1 + w * e1);
      else ep[(t >> 3) * 4 + 2 + (t & 1)] = e1;
    }
    const float u0 = c * e0, u1 = c * e1;
#pragma unroll
    for (int i = 0; i < D / 8; ++i) {
      const float2 kk = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sk + t * KLD + i * 8 + 2 * q));
      if (first0 < EC) {
        S[i][0] += kk.x * u0;
        S[i][1] += kk.y * u0;
      }
      if (first1 < EC) {
        S[i][2] += kk.x * u1;
        S[i][3] += kk.y * u1;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < D / 2; ++i) sp[i] = S[i / 4][i % 4];
}

// The same for the gradient of the state, from the last token to the first: de_t = c y - ex dO with y = dS^T k, dS -= k de. All columns; the
// de go to ep.
template <int D, int KLD, int VLD>
__device__ __noinline__ void efla_walk_back(float* sp, float* ep, const __nv_bfloat16* sk, const __nv_bfloat16* so, const float* cf, int n) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  float S[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 2; ++i) S[i / 4][i % 4] = sp[i];
#pragma unroll 1
  for (int t = n - 1; t >= 0; --t) {
    float y0 = 0.f, y1 = 0.f;
#pragma unroll
    for (int i = 0; i < D / 8; ++i) {
      const float2 kk = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sk + t * KLD + i * 8 + 2 * q));
      y0 += kk.x * S[i][0] + kk.y * S[i][1];
      y1 += kk.x * S[i][2] + kk.y * S[i][3];
    }
#pragma unroll
    for (int m = 1; m < 4; m <<= 1) {
      y0 += __shfl_xor_sync(0xffffffffu, y0, m);
      y1 += __shfl_xor_sync(0xffffffffu, y1, m);
    }
    const float d0 = cf[t] * y0 - cf[EC + t] * __bfloat162float(so[t * VLD + g]);
    const float d1 = cf[t] * y1 - cf[EC + t] * __bfloat162float(so[t * VLD + g + 8]);
    if (q == (t & 7) >> 1) {
      ep[(t >> 3) * 4 + (t & 1)] = d0;
      ep[(t >> 3) * 4 + 2 + (t & 1)] = d1;
    }
#pragma unroll
    for (int i = 0; i < D / 8; ++i) {
      const float2 kk = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sk + t * KLD + i * 8 + 2 * q));
      S[i][0] -= kk.x * d0;
      S[i][1] -= kk.y * d0;
      S[i][2] -= kk.x * d1;
      S[i][3] -= kk.y * d1;
    }
  }
#pragma unroll
  for (int i = 0; i < D / 2; ++i) sp[i] = S[i / 4][i % 4];
}

// y_t = dS^T k_t of every token, put where the errors are put
template <int D, int KLD>
__device__ __noinline__ void efla_rows(const float* sp, float* ep, const __nv_bfloat16* sk, int n) {
  const int lane = threadIdx.x & 31, q = lane & 3;
#pragma unroll 1
  for (int t = 0; t < n; ++t) {
    float y0 = 0.f, y1 = 0.f;
#pragma unroll 4
    for (int i = 0; i < D / 8; ++i) {
      const float2 kk = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sk + t * KLD + i * 8 + 2 * q));
      y0 += kk.x * sp[i * 4] + kk.y * sp[i * 4 + 1];
      y1 += kk.x * sp[i * 4 + 2] + kk.y * sp[i * 4 + 3];
    }
#pragma unroll
    for (int m = 1; m < 4; m <<= 1) {
      y0 += __shfl_xor_sync(0xffffffffu, y0, m);
      y1 += __shfl_xor_sync(0xffffffffu, y1, m);
    }
    if (q == (t & 7) >> 1) {
      ep[(t >> 3) * 4 + (t & 1)] = y0;
      ep[(t >> 3) * 4 + 2 + (t & 1)] = y1;
    }
  }
}

// a state tile holds a value that is not finite
template <int D>
__device__ __forceinline__ bool efla_not_finite(const float (&S)[D / 8][4]) {
  float chk = 0.f;
#pragma unroll
  for (int i = 0; i < D / 8; ++i)
#pragma unroll
    for (int x = 0; x < 4; ++x) chk = fmaf(S[i][x], 0.f, chk);
  return chk != 0.f;
}
// any lane of the warp holds a value that is not finite
__device__ __forceinline__ bool efla_any_bad(const float (&e)[4][4]) {
  float chk = 0.f;
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int x = 0; x < 4; ++x) chk = fmaf(e[nt][x], 0.f, chk);
  return __any_sync(0xffffffffu, chk != 0.f);
}
// first[hf] = the earliest token at which column g + 8 hf is not finite, at most what it was; those entries become 0
__device__ __forceinline__ void efla_take_bad(float (&e)[4][4], int (&first)[2], int q) {
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int x = 0; x < 4; ++x)
      if (!(fabsf(e[nt][x]) <= 3.402823466e38f)) {
        first[x >> 1] = min(first[x >> 1], nt * 8 + 2 * q + (x & 1));
        e[nt][x] = 0.f;
      }
#pragma unroll
  for (int hf = 0; hf < 2; ++hf) {
    first[hf] = min(first[hf], __shfl_xor_sync(0xffffffffu, first[hf], 1));
    first[hf] = min(first[hf], __shfl_xor_sync(0xffffffffu, first[hf], 2));
  }
}

// e = V - e for a warp's tile, V^T as read by ldmatrix
__device__ __forceinline__ void efla_errors(float (&e)[4][4], const uint32_t (&vq)[2][4]) {
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int hf = 0; hf < 2; ++hf)
      put_pair(e[nt], hf, fma_f32x2(pair_of(e[nt], hf), pack_f32x2(-1.f, -1.f), pack_f32x2(bf16_lo(vq[hf][nt]), bf16_hi(vq[hf][nt]))));
}

// Chunk-boundary states are stored as the warps hold them: [B, H, chunk][d / 16 value blocks][d / 8 tiles][lane] float4.
template <int D>
__device__ __forceinline__ long long efla_state_slot(long long chunk_id, int vblock, int lane) {
  return ((chunk_id * (D / 16) + vblock) * (D / 8)) * 32 + lane;      // float4 units; tile n at + 32 n
}

// A walk over the chunks [c0, c1) of one head. state0: null (zero) or the head's [d, d] start; identity: start from the identity instead.
// With vals = outs = null and ckpt = null only the state is walked; state_out (or null) gets the last one.
struct EflaWalk {
  int c0, c1;
  bool identity;
  const float* state0;
  float* state_out;
};

// k, v, o: [B, T, H, d] bf16; v and o may be null (see EflaWalk). ckpt (or null): the state at the start of every chunk.
// Bound by the dependent chain of a chunk (132 mma.sync and about 880 instructions of one warp per scheduler), not by memory. With the
// preparation, B 1, T 8192, 16 heads of 64, no gradient: 342 us in one walk, token by token (with its checkpoints) 2364 us; in the training step
// of B 8, T 2048 the forward went from about 750 to 85 us and 28 us for the preparation.
template <int D, bool CHECKED, bool CUT>
__device__ __forceinline__ bool efla_fwd_walk(
    const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v, const __nv_bfloat16* __restrict__ nmat,
    const float* __restrict__ coef, __nv_bfloat16* __restrict__ o, float4* __restrict__ ckpt, int T, int H, int nchunks, EflaWalk w) {
  using L = EflaStage<D>;
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int bh = blockIdx.x, b = bh / H, h = bh % H;
  const int ccol = blockIdx.y * L::VC, wcol = ccol + warp * 16;       // first value column of the CTA / of this warp
  const uint32_t ring = smem_u32(smem);
  const int c0 = CUT ? w.c0 : 0, c1 = CUT ? w.c1 : nchunks;
  __nv_bfloat16* stage_o = reinterpret_cast<__nv_bfloat16*>(smem + EC_STAGES * L::BYTES) + warp * EC * 24;   // [32 tokens][16 + 8]
  const long long row0 = ((long long)b * T * H + h) * D, rs = (long long)H * D;
  const __nv_bfloat16 *kb = k + row0, *vb = !CUT || v ? v + row0 + ccol : nullptr;
  const __nv_bfloat16* nb = nmat + (long long)bh * nchunks * EN_ELEMS;
  const float* cb = coef + (long long)bh * nchunks * EC_COEF;

  float S[D / 8][4];                       // S^T: value column g (+ 8), key row 8 n + 2q (+ 1)
#pragma unroll
  for (int n = 0; n < D / 8; ++n)
#pragma unroll
    for (int x = 0; x < 4; ++x)
    {
      const int row = n * 8 + 2 * q + (x & 1), col = wcol + g + (x >> 1) * 8;
      S[n][x] = CUT && w.identity ? (row == col ? 1.f : 0.f) : (w.state0 ? w.state0[row * D + col] : 0.f);
    }

  const EflaLoader<D> load(kb, vb, nb, cb, rs, ring, T);
  auto fetch = [&](int ch) {
    if (ch < c1) load(ch, ch);
    cp_async_commit();
  };
#pragma unroll
  for (int i = 0; i < EC_STAGES - 1; ++i) fetch(c0 + i);
  for (int ch = c0; ch < c1; ++ch) {
    const int stage = ch % EC_STAGES;
    cp_async_wait<EC_STAGES - 2>();
    __syncthreads();                       // chunk ch has landed for every thread; the stage of chunk ch - 1 is free
    fetch(ch + EC_STAGES - 1);
    const uint32_t st = ring + stage * L::BYTES;
    const float* cf = reinterpret_cast<const float*>(smem + stage * L::BYTES + L::C);
    if (ckpt) {
      float4* dst = ckpt + efla_state_slot<D>((long long)bh * nchunks + ch, wcol / 16, lane);
#pragma unroll
      for (int n = 0; n < D / 8; ++n) dst[n * 32] = make_float4(S[n][0], S[n][1], S[n][2], S[n][3]);
    }
    float e[4][4];
    efla_state_times_k<D>(e, S, st + L::K, lane);
    uint32_t vq[2][4];                     // V^T tiles: [value half][token tile], tokens 2q, 2q + 1 of column g
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) ldsm4_t(vq[hf], st + L::V + (lane * L::VLD + warp * 16 + hf * 8) * 2);
    efla_errors(e, vq);
    efla_apply_n<false>(e, st + L::N, lane);
    int first[2] = {EC, EC};
    if (CHECKED && efla_any_bad(e)) {      // once more, without the entries at fault: the other columns and the tokens before keep their bits
      efla_state_times_k<D>(e, S, st + L::K, lane);
      efla_errors(e, vq);
      efla_take_bad(e, first, q);
      efla_apply_n<false>(e, st + L::N, lane);
      efla_take_bad(e, first, q);
    }
    const bool bad = CHECKED && __any_sync(0xffffffffu, first[0] < EC || first[1] < EC);
    uint32_t oq[2][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const float2 ex = *reinterpret_cast<const float2*>(cf + EC + nt * 8 + 2 * q);
      const float2 cc = *reinterpret_cast<const float2*>(cf + nt * 8 + 2 * q);
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        float o0, o1;
        unpack_f32x2(fma_f32x2(pack_f32x2(-ex.x, -ex.y), pair_of(e[nt], hf), pack_f32x2(bf16_lo(vq[hf][nt]), bf16_hi(vq[hf][nt]))), o0, o1);
        oq[hf][nt] = pack_bf16(o0, o1);
        put_pair(e[nt], hf, mul_f32x2(pair_of(e[nt], hf), pack_f32x2(cc.x, cc.y)));
      }
    }
    if (bad) {
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (first[x >> 1] < EC) e[nt][x] = 0.f;                     // the walk below moves these columns
    }
    if (!CUT || o) {                       // the outputs change their layout while the state is updated
      const uint32_t so = smem_u32(stage_o);
      __syncwarp();
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) stsm4_t(so + (lane * 24 + hf * 8) * 2, oq[hf][0], oq[hf][1], oq[hf][2], oq[hf][3]);
      __syncwarp();
    }
    efla_state_update<D, false>(S, e, st + L::K, lane);
    if (bad) {
      const unsigned char* sst = smem + stage * L::BYTES;
      float sl[D / 2];
#pragma unroll
      for (int n = 0; n < D / 2; ++n) sl[n] = S[n / 4][n % 4];
      efla_walk<D, L::KLD, L::VLD, true>(sl, nullptr, reinterpret_cast<const __nv_bfloat16*>(sst + L::K),
                                         reinterpret_cast<const __nv_bfloat16*>(sst + L::V) + warp * 16, cf, stage_o, first[0], first[1],
                                         min(EC, T - ch * EC));
#pragma unroll
      for (int n = 0; n < D / 2; ++n) S[n / 4][n % 4] = sl[n];
      __syncwarp();
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int t = u * 16 + (lane >> 1), hf = lane & 1;
      if ((!CUT || o) && ch * EC + t < T)
        *reinterpret_cast<uint4*>(o + row0 + ((long long)ch * EC + t) * rs + wcol + hf * 8) = *reinterpret_cast<const uint4*>(stage_o + t * 24 + hf * 8);
    }
  }
  cp_async_wait<0>();
  if (w.state_out) {
#pragma unroll
    for (int n = 0; n < D / 8; ++n)
#pragma unroll
      for (int x = 0; x < 4; ++x) w.state_out[(n * 8 + 2 * q + (x & 1)) * D + wcol + g + (x >> 1) * 8] = S[n][x];
  }
  // an error that was not finite anywhere has left its state column not finite (mma.sync: also 0 x NaN)
  return efla_not_finite<D>(S);
}

template <int D, bool CUT>
__device__ __noinline__ void efla_fwd_again(const __nv_bfloat16* k, const __nv_bfloat16* v, const __nv_bfloat16* nmat, const float* coef,
                                            __nv_bfloat16* o, float4* ckpt, int T, int H, int nchunks, EflaWalk w) {
  efla_fwd_walk<D, true, CUT>(k, v, nmat, coef, o, ckpt, T, H, nchunks, w);
}

// Segments. A walk of n chunks is cut into P segments of `seg` chunks, since a chunk's update is affine in the state (S1 = A S0 + B):
//   FIRST  segment 0 from its known start, with its outputs; segments 1 .. P - 2 from zero (their B) and, without values, from the identity
//          (their A), states only: 2 P - 3 walks per head side by side
//   (efla_combine_kernel: start of segment p + 1 = A_p start_p + B_p)
//   REST   segments 1 .. P - 1 from their starts, with their outputs
// The walk in one piece is compiled apart (CUT = false): asking for what may be absent in it cost 5 us of 94.
// Three times the work in 2 / P of the steps: worth it where the heads alone leave the chip idle (see efla_segments). With beta >= 0 the maps
// contract (the eigenvalues of a token's factor, exp(-beta |k|^2) and 1, lie in (0, 1]), so an error of a start dies out along its segment.
// beta is learned and may turn negative: then a map of many tokens grows past the range of fp32 where the states that it would multiply are
// zero, and the heads are walked in one piece: the first CTA of FIRST takes all chunks and the other launches leave at once. The host does not know
// beta; the sign of a token's coefficient is that of beta.
// work: start [P], A [P], B [P], each [B H, d, d] fp32.
enum { EFLA_FIRST, EFLA_REST };

__device__ __forceinline__ bool efla_in_one_piece(const float* __restrict__ coef, int bh, int nchunks) {
  return !(coef[(long long)bh * nchunks * EC_COEF] >= 0.f);
}

__device__ __forceinline__ float* efla_work(float* work, int which, int P, int p, int bh, int dd) {
  return work + (((long long)which * P + p) * gridDim.x + bh) * dd;
}

// Grid (B * H, d / columns of a CTA, walks). state0 / state_out: [B, H, d, d] fp32 or null.
template <int D, bool CUT>
__global__ void __launch_bounds__(32 * ec_warps<D>()) efla_chunk_fwd_kernel(
    const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v, const __nv_bfloat16* __restrict__ nmat,
    const float* __restrict__ coef, const float* state0, __nv_bfloat16* __restrict__ o, float* state_out,
    float4* __restrict__ ckpt, float* work, int T, int H, int nchunks, int P, int seg, int phase) {
  const int bh = blockIdx.x, z = blockIdx.z;
  EflaWalk w{0, nchunks, false, state0 ? state0 + (long long)bh * D * D : nullptr, state_out ? state_out + (long long)bh * D * D : nullptr};
  const bool whole = !CUT || efla_in_one_piece(coef, bh, nchunks);
  if (CUT && whole && (phase == EFLA_REST || z > 0)) return;
  if (!whole) {
    const bool map = phase == EFLA_FIRST && z > 0;                       // a segment's A or B
    const int p = phase == EFLA_REST ? z + 1 : (z > P - 2 ? z - (P - 2) : z);
    w.c0 = p * seg;
    w.c1 = min(nchunks, w.c0 + seg);
    if (map) {
      w.identity = z > P - 2;
      w.state0 = nullptr;
      w.state_out = efla_work(work, w.identity ? 1 : 2, P, p, bh, D * D);
      if (w.identity) v = nullptr;
      o = nullptr;
      ckpt = nullptr;
    } else {
      if (p > 0) w.state0 = efla_work(work, 0, P, p, bh, D * D);
      if (p < P - 1) w.state_out = p == 0 ? efla_work(work, 0, P, 1, bh, D * D) : nullptr;
    }
  }
  if (__syncthreads_or(efla_fwd_walk<D, false, CUT>(k, v, nmat, coef, o, ckpt, T, H, nchunks, w)))
    efla_fwd_again<D, CUT>(k, v, nmat, coef, o, ckpt, T, H, nchunks, w);
}

// the i-th of the six products of two split operands, small ones first
__device__ __forceinline__ void mma_split(float (&acc)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][4], int o, int i, bool first) {
  const int ai = i == 0 || i == 3 ? 1 : (i == 1 ? 2 : 0), bi = i == 0 || i == 4 ? 1 : (i == 2 ? 2 : 0);
  if (first) mma_bf16_first(acc, a[ai], b[bi][o], b[bi][o + 1]);
  else mma_bf16(acc, a[ai], b[bi][o], b[bi][o + 1]);
}

// start[p + dir] = A[p] start[p] + B[p] for the P - 2 inner segments, in order, on the tensor cores: a CTA owns 16 columns of a head, warp w the rows
// 16 w .. 16 w + 15. Both operands are split in three (24 bits each; the six products above 2^-24, small ones first, in three sums joined at the end), so a
// start is as close to the 64-bit one as with fp32 multiply-adds (which the walks' errors hide either way: final state, B 1, T 8192, 16 heads of 64, 10
// segments, 2.2e-7 relative). The next A is copied to shared memory while this one is used; the start goes to the next step as splits in shared memory.
// Bound by the chain of a step: the sums, the splits of the start, one barrier. Per step of 128 and 64 rows 1.9 and 1.1 us, with fp32 multiply-adds 6.3 and
// 1.6. Grid (B * H, d / 16).
template <int D>
struct EflaCombineSmem {
  static constexpr int ALD = D + 8, SLD = D + 8;                             // A fp32; splits of the start, a row per column
  static constexpr int A = 0, S = 2 * D * ALD * 4, BYTES = S + 2 * 3 * 16 * SLD * 2;
};
template <int D>
__global__ void __launch_bounds__(2 * D) efla_combine_kernel(const float* __restrict__ coef, float* __restrict__ work, int nchunks, int P, int dir) {
  using L = EflaCombineSmem<D>;
  extern __shared__ __align__(16) unsigned char smem[];
  const uint32_t base = smem_u32(smem);
  const int bh = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, r0 = warp * 16 + g, c0 = blockIdx.y * 16 + 2 * q;
  if (efla_in_one_piece(coef, bh, nchunks)) return;
  int p = dir > 0 ? 1 : P - 2;
  auto fetch = [&](int n, int at) {                    // A of the n-th step
    const float* a = efla_work(work, 1, P, at, bh, D * D);
    for (int i = threadIdx.x; i < D * D / 4; i += 2 * D)
      cp_async16(base + L::A + ((n & 1) * D * L::ALD + i / (D / 4) * L::ALD + i % (D / 4) * 4) * 4, a + i * 4, true);
    cp_async_commit();
  };
  // tile j of eight columns, half hf of the warp's rows: row r0 + 8 hf, columns c0 + 8 j and the next
  auto put_start = [&](int n, const float (&s)[2][4]) {
    uint32_t t[3][4];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) split3(s[j][2 * hf], s[j][2 * hf + 1], t[0][2 * j + hf], t[1][2 * j + hf], t[2][2 * j + hf]);
    const int col = (lane >> 4) * 8 + (lane & 7), row = warp * 16 + (lane >> 3 & 1) * 8;
#pragma unroll
    for (int x = 0; x < 3; ++x)
      stsm4_t(base + L::S + (((n & 1) * 3 + x) * 16 * L::SLD + col * L::SLD + row) * 2, t[x][0], t[x][1], t[x][2], t[x][3]);
  };
  auto at = [&](float* m, int j, int hf) { return reinterpret_cast<float2*>(m + (r0 + 8 * hf) * D + c0 + 8 * j); };
  fetch(0, p);
  float s[2][4], bn[2][4];
  auto read = [&](float (&to)[2][4], float* m) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const float2 f = *at(m, j, hf);
        to[j][2 * hf] = f.x;
        to[j][2 * hf + 1] = f.y;
      }
  };
  read(s, efla_work(work, 0, P, p, bh, D * D));
  read(bn, efla_work(work, 2, P, p, bh, D * D));
  put_start(0, s);
  for (int n = 0; n < P - 2; ++n, p += dir) {
    cp_async_wait<0>();
    __syncthreads();                                   // A and the start have landed; the buffers of the step before are free
    float b[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int x = 0; x < 4; ++x) b[j][x] = bn[j][x];
    if (n + 1 < P - 2) {
      fetch(n + 1, p + dir);
      read(bn, efla_work(work, 2, P, p + dir, bh, D * D));
    }
    float acc[3][2][4];                                // the smallest products, the middle ones, the large ones
    const float* sa = reinterpret_cast<const float*>(smem + L::A) + (n & 1) * D * L::ALD;
#pragma unroll
    for (int k = 0; k < D / 16; ++k) {
      uint32_t a[3][4], f[3][4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {                    // a0, a1: rows g, g + 8; a2, a3: the columns 8 further
        const float2 v = *reinterpret_cast<const float2*>(sa + (r0 + (x & 1) * 8) * L::ALD + k * 16 + (x >> 1) * 8 + 2 * q);
        split3(v.x, v.y, a[0][x], a[1][x], a[2][x]);
      }
#pragma unroll
      for (int x = 0; x < 3; ++x)
        ldsm4(f[x], base + L::S + (((n & 1) * 3 + x) * 16 * L::SLD + ((lane >> 4) * 8 + (lane & 7)) * L::SLD + k * 16 + (lane >> 3 & 1) * 8) * 2);
#pragma unroll
      for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) mma_split(acc[i < 3 ? 0 : (i < 5 ? 1 : 2)][j], a, f, 2 * j, i, k == 0 && (i == 0 || i == 3 || i == 5));
    }
    float* out = efla_work(work, 0, P, p + dir, bh, D * D);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
        for (int x = 2 * hf; x < 2 * hf + 2; ++x) s[j][x] = ((acc[0][j][x] + acc[1][j][x]) + acc[2][j][x]) + b[j][x];
        *at(out, j, hf) = make_float2(s[j][2 * hf], s[j][2 * hf + 1]);
      }
    if (n + 1 < P - 2) put_start(n + 1, s);
  }
}

template <int D>
int launch_combine(const float* coef, float* work, int BH, int nchunks, int P, int dir, cudaStream_t s) {
  if (P < 3) return ELFA_OK;
  constexpr int bytes = EflaCombineSmem<D>::BYTES;
  ELFA_CUDA(allow_shared<efla_combine_kernel<D>>(bytes));
  efla_combine_kernel<D><<<dim3(BH, D / 16), 2 * D, bytes, s>>>(coef, work, nchunks, P, dir);
  ELFA_CUDA(cudaGetLastError());
  ::elfa::count_launches(1);
  return ELFA_OK;
}

template <int D>
int launch_chunk_fwd(const void* k, const void* v, const float* beta, const float* state0, void* o, float* state_out, float* ckpt,
                     void* nmat, float* coef, float* work, int P, int B, int T, int H, cudaStream_t s) {
  using L = EflaStage<D>;
  const int nchunks = (T + EC - 1) / EC;
  const long long total = (long long)B * H * nchunks;
  ELFA_REQUIRE((total + 1) / 2 < (1ll << 31), "efla_chunk_fwd: too many chunks");
  efla_prep_kernel<D><<<(unsigned)((total + 1) / 2), 64, 0, s>>>(static_cast<const __nv_bfloat16*>(k), beta, static_cast<__nv_bfloat16*>(nmat),
                                                                 coef, T, H, nchunks, total);
  ELFA_CUDA(cudaGetLastError());
  constexpr int bytes = EC_STAGES * L::BYTES + ec_warps<D>() * EC * 24 * 2;
  int seg = nchunks;
  if (P > 1) {
    seg = (nchunks + P - 1) / P;
    P = (nchunks + seg - 1) / seg;
  }
  auto kernel = P > 1 ? efla_chunk_fwd_kernel<D, true> : efla_chunk_fwd_kernel<D, false>;
  ELFA_CUDA((P > 1 ? allow_shared<efla_chunk_fwd_kernel<D, true>>(bytes) : allow_shared<efla_chunk_fwd_kernel<D, false>>(bytes)));
  auto walk = [&](int phase, int walks) {
    kernel<<<dim3(B * H, D / L::VC, walks), 32 * ec_warps<D>(), bytes, s>>>(
        static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v), static_cast<const __nv_bfloat16*>(nmat), coef, state0,
        static_cast<__nv_bfloat16*>(o), state_out, reinterpret_cast<float4*>(ckpt), work, T, H, nchunks, P, seg, phase);
    ::elfa::count_launches(1);
  };
  ::elfa::count_launches(1);
  if (P <= 1) {
    walk(EFLA_FIRST, 1);
  } else {
    walk(EFLA_FIRST, 2 * P - 3);
    ELFA_CUDA(cudaGetLastError());
    const int rc = launch_combine<D>(coef, work, B * H, nchunks, P, 1, s);
    if (rc != ELFA_OK) return rc;
    walk(EFLA_REST, P - 1);
  }
  ELFA_CUDA(cudaGetLastError());
  return ELFA_OK;
}

// ------------------------------------------------------------------------------------------------ backward
// With dS1 the gradient of the state behind a chunk, Y = K dS1 and U = diag(c) E:
//   dE  = -diag(ex) dO + diag(c) Y        dE0 = dE + N^T dE        dV = dO + dE0        dS0 = dS1 - K^T dE0
//   dK  = U dS1^T - dE0 S0^T + (dG + dG^T + 2 diag(dlam)) K       dG_ts = -(dE0 E^T)_ts c_s  (t > s)
//   dc_t = sum_j (Y E)_tj + lam_t sum_j (dO E)_tj - sum_{r > t} (dE0 E^T)_rt (K K^T)_rt
//   dlam_t = c_t sum_j (dO E)_tj + dc_t dc/dlam,   dbeta = sum_t dc_t ex_t
// Only dS is sequential: efla_chunk_bwd_state_kernel walks the chunks backwards with dS in registers and writes the dS1 of every chunk;
// efla_chunk_bwd_kernel then handles all chunks in parallel from the two chunk-boundary states.
// B 8, T 2048, 16 heads of 64: 76 us and 257 us (token by token, the states of a chunk through a global workspace: 2352 us and 130 us more to
// finish). The parallel kernel issues about 400 mma.sync per warp and chunk (94 us of tensor time at 8.3 cycles each) and reads 370 MB
// (55 us); it is bound by the chain of its two warps per scheduler (five cycles per instruction of a warp, a third of the issue slots). A third CTA
// per SM, at 168 registers, did not make it faster; nor did a tenth fewer instructions (packed remainders of the splits, first products without zeroed
// sums, per-token sums halved from lane to lane) with 64-wide heads. With 128-wide ones, one CTA per SM, these, the start's states asked for into L2 one
// round of CTAs ahead and read a second time behind the products of the other term took it from 99 to 91.5 us (B 2, T 1531, 8 heads).
template <int D, bool CHECKED, bool CUT>
__device__ __forceinline__ bool efla_bwd_walk(
    const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ nmat,
    const float* __restrict__ coef, float4* __restrict__ dckpt, int T, int H, int nchunks, EflaWalk w) {
  using L = EflaStage<D>;
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int bh = blockIdx.x, b = bh / H, h = bh % H;
  const int ccol = blockIdx.y * L::VC, wcol = ccol + warp * 16;
  const uint32_t ring = smem_u32(smem);
  const int c0 = CUT ? w.c0 : 0, c1 = CUT ? w.c1 : nchunks;
  const long long row0 = ((long long)b * T * H + h) * D, rs = (long long)H * D;
  const __nv_bfloat16 *kb = k + row0, *ob = !CUT || dout ? dout + row0 + ccol : nullptr;
  const __nv_bfloat16* nb = nmat + (long long)bh * nchunks * EN_ELEMS;
  const float* cb = coef + (long long)bh * nchunks * EC_COEF;

  float S[D / 8][4];                       // dS^T, laid out as the state of the forward kernel
#pragma unroll
  for (int n = 0; n < D / 8; ++n)
#pragma unroll
    for (int x = 0; x < 4; ++x)
    {
      const int row = n * 8 + 2 * q + (x & 1), col = wcol + g + (x >> 1) * 8;
      S[n][x] = CUT && w.identity ? (row == col ? 1.f : 0.f) : (w.state0 ? w.state0[row * D + col] : 0.f);
    }

  const EflaLoader<D> load(kb, ob, nb, cb, rs, ring, T);
  auto fetch = [&](int i) {                // i-th chunk from the end
    const int ch = c1 - 1 - i;
    if (ch >= c0) load(i, ch);
    cp_async_commit();
  };
#pragma unroll
  for (int i = 0; i < EC_STAGES - 1; ++i) fetch(i);
  for (int i = 0; i < c1 - c0; ++i) {
    const int stage = i % EC_STAGES;
    cp_async_wait<EC_STAGES - 2>();
    __syncthreads();
    fetch(i + EC_STAGES - 1);
    const uint32_t st = ring + stage * L::BYTES;
    const float* cf = reinterpret_cast<const float*>(smem + stage * L::BYTES + L::C);
    if (!CUT || dckpt) {
      float4* dst = dckpt + efla_state_slot<D>((long long)bh * nchunks + c1 - 1 - i, wcol / 16, lane);
#pragma unroll
      for (int n = 0; n < D / 8; ++n) dst[n * 32] = make_float4(S[n][0], S[n][1], S[n][2], S[n][3]);
    }
    float e[4][4];
    efla_state_times_k<D>(e, S, st + L::K, lane);
    uint32_t oq[2][4];
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) ldsm4_t(oq[hf], st + L::V + (lane * L::VLD + warp * 16 + hf * 8) * 2);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const float2 cc = *reinterpret_cast<const float2*>(cf + nt * 8 + 2 * q);
      const float2 ex = *reinterpret_cast<const float2*>(cf + EC + nt * 8 + 2 * q);
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const uint64_t o = mul_f32x2(pack_f32x2(-ex.x, -ex.y), pack_f32x2(bf16_lo(oq[hf][nt]), bf16_hi(oq[hf][nt])));
        put_pair(e[nt], hf, fma_f32x2(pack_f32x2(cc.x, cc.y), pair_of(e[nt], hf), o));
      }
    }
    efla_apply_n<true>(e, st + L::N, lane);
    if (!(CHECKED && efla_any_bad(e))) {
      efla_state_update<D, true>(S, e, st + L::K, lane);
    } else {                               // e.g. a NaN in dO: it reaches its own and the earlier tokens only
      float sl[D / 2], unused[16];
#pragma unroll
      for (int n = 0; n < D / 2; ++n) sl[n] = S[n / 4][n % 4];
      const unsigned char* sst = smem + stage * L::BYTES;
      efla_walk_back<D, L::KLD, L::VLD>(sl, unused, reinterpret_cast<const __nv_bfloat16*>(sst + L::K),
                                        reinterpret_cast<const __nv_bfloat16*>(sst + L::V) + warp * 16, cf,
                                        min(EC, T - (c1 - 1 - i) * EC));
#pragma unroll
      for (int n = 0; n < D / 2; ++n) S[n / 4][n % 4] = sl[n];
    }
  }
  cp_async_wait<0>();
  if (w.state_out) {
#pragma unroll
    for (int n = 0; n < D / 8; ++n)
#pragma unroll
      for (int x = 0; x < 4; ++x) w.state_out[(n * 8 + 2 * q + (x & 1)) * D + wcol + g + (x >> 1) * 8] = S[n][x];
  }
  return efla_not_finite<D>(S);
}

template <int D, bool CUT>
__device__ __noinline__ void efla_bwd_again(const __nv_bfloat16* k, const __nv_bfloat16* dout, const __nv_bfloat16* nmat, const float* coef,
                                            float4* dckpt, int T, int H, int nchunks, EflaWalk w) {
  efla_bwd_walk<D, true, CUT>(k, dout, nmat, coef, dckpt, T, H, nchunks, w);
}

// Segments as in the forward kernel, from the last one to the first: FIRST walks the last segment from dstate_out and the inner ones from zero
// and (without dO) from the identity, which gives the transposed maps.
template <int D, bool CUT>
__global__ void __launch_bounds__(32 * ec_warps<D>()) efla_chunk_bwd_state_kernel(
    const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ nmat,
    const float* __restrict__ coef, const float* dstate_out, float4* __restrict__ dckpt, float* dstate0, float* work, int T, int H,
    int nchunks, int P, int seg, int phase) {
  const int bh = blockIdx.x, z = blockIdx.z;
  EflaWalk w{0, nchunks, false, dstate_out ? dstate_out + (long long)bh * D * D : nullptr, dstate0 ? dstate0 + (long long)bh * D * D : nullptr};
  const bool whole = !CUT || efla_in_one_piece(coef, bh, nchunks);
  if (CUT && whole && (phase == EFLA_REST || z > 0)) return;
  if (!whole) {
    const bool map = phase == EFLA_FIRST && z > 0;
    const int p = phase == EFLA_REST ? z : (z == 0 ? P - 1 : (z > P - 2 ? z - (P - 2) : z));
    w.c0 = p * seg;
    w.c1 = min(nchunks, w.c0 + seg);
    if (map) {
      w.identity = z > P - 2;
      w.state0 = nullptr;
      w.state_out = efla_work(work, w.identity ? 1 : 2, P, p, bh, D * D);
      if (w.identity) dout = nullptr;
      dckpt = nullptr;
    } else {
      if (p < P - 1) w.state0 = efla_work(work, 0, P, p, bh, D * D);
      if (p > 0) w.state_out = p == P - 1 ? efla_work(work, 0, P, P - 2, bh, D * D) : nullptr;
    }
  }
  if (__syncthreads_or(efla_bwd_walk<D, false, CUT>(k, dout, nmat, coef, dckpt, T, H, nchunks, w)))
    efla_bwd_again<D, CUT>(k, dout, nmat, coef, dckpt, T, H, nchunks, w);
}

// One CTA per chunk, d / 16 warps; warp w owns value columns 16 w .. 16 w + 15 and all key rows. E, Y, dE0 are recomputed from the
// chunk-boundary states with the products of the sequential kernels; the contractions over the value columns (dK, dE0 E^T) are
// partial per warp and added up in warp order through shared memory. A warp's scratch holds transposed splits first, its dK partial
// last.
template <int D>
struct EflaBwdSmem {
  static constexpr int W = D / 16;
  static constexpr int LD = D + 8;                                       // K, V, dO tiles and the split state tile (bf16)
  static constexpr int TILE = EC * LD * 2;
  static constexpr int SCR_E = 3 * 16 * EN_LD * 2, SCR_S = 3 * 16 * LD * 2, RED_LD = D + 4;
  static constexpr int SCR = SCR_E + SCR_S > EC * RED_LD * 4 ? SCR_E + SCR_S : EC * RED_LD * 4;
  static constexpr int GLD = 36;
  static constexpr int K = 0, V = K + TILE, O = V + TILE, N = O + TILE, C = N + EN_ELEMS * 2, G = C + EC_COEF * 4,
                       DA = G + EC * GLD * 4, SUM = DA + W * EC * GLD * 4, DC = SUM + W * 2 * EC * 4, SCRATCH = DC + W * EC * 4,
                       BYTES = SCRATCH + W * SCR;
};

__device__ __forceinline__ void stsm4(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}

// Three splits of a 16 x 32 tile (rows = value columns j, columns = tokens) into scratch [3][16][EN_LD].
__device__ __forceinline__ void efla_put_tokens(uint32_t scr, const float (&e)[4][4], int lane) {
#pragma unroll
  for (int hf = 0; hf < 2; ++hf) {
    uint32_t s[3][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) split3(e[nt][2 * hf], e[nt][2 * hf + 1], s[0][nt], s[1][nt], s[2][nt]);
#pragma unroll
    for (int p = 0; p < 3; ++p)
      stsm4(scr + (p * 16 * EN_LD + (hf * 8 + (lane & 7)) * EN_LD + (lane >> 3) * 8) * 2, s[p][0], s[p][1], s[p][2], s[p][3]);
  }
}
// ... read back as the A operand (rows = tokens 16 mi .., k = value columns)
__device__ __forceinline__ void efla_get_a(uint32_t (&a)[3][4], uint32_t scr, int mi, int lane) {
#pragma unroll
  for (int p = 0; p < 3; ++p)
    ldsm4_t(a[p], scr + (p * 16 * EN_LD + ((lane & 7) + (lane >> 4) * 8) * EN_LD + mi * 16 + ((lane >> 3) & 1) * 8) * 2);
}
// ... or as the B operand of two tiles (k = value columns, columns = x 16 np .. 16 np + 15), from a scratch of row pitch LD
template <int LD>
__device__ __forceinline__ void efla_get_b(uint32_t (&b)[3][4], uint32_t scr, int np, int lane) {
#pragma unroll
  for (int p = 0; p < 3; ++p) ldsm4_t(b[p], scr + (p * 16 * LD + (lane & 15) * LD + np * 16 + (lane >> 4) * 8) * 2);
}
template <int D, bool CHECKED>
__device__ __forceinline__ bool efla_bwd_chunk(
    const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v, const __nv_bfloat16* __restrict__ dout,
    const __nv_bfloat16* __restrict__ nmat, const float* __restrict__ coef, const float4* __restrict__ ckpt,
    const float4* __restrict__ dckpt, __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv,
    float* __restrict__ dbeta, bool by_chunk, int T, int H, int nchunks, int ahead) {
  using L = EflaBwdSmem<D>;
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const long long id = blockIdx.x;
  const int bh = (int)(id / nchunks), ch = (int)(id % nchunks), b = bh / H, h = bh % H;
  const int t0 = ch * EC, n = min(EC, T - t0);
  const uint32_t base = smem_u32(smem);
  const long long rs = (long long)H * D, off = (((long long)b * T + t0) * H + h) * D;
  const float* cf = reinterpret_cast<const float*>(smem + L::C);

  for (int i = tid; i < EC * (D / 8); i += 2 * D) {
    const int r = i / (D / 8), c = i % (D / 8);
    const long long src = off + (r < n ? r : 0) * rs + c * 8;
    const uint32_t dst = (r * L::LD + c * 8) * 2;
    cp_async16(base + L::K + dst, k + src, r < n);
    cp_async16(base + L::V + dst, v + src, r < n);
    cp_async16(base + L::O + dst, dout + src, r < n);
  }
  for (int i = tid; i < 3 * EC * 4; i += 2 * D) cp_async16(base + L::N + i * 16, nmat + id * EN_ELEMS + i * 8, true);
  if (tid < EC_COEF / 4) cp_async16(base + L::C + tid * 16, coef + id * EC_COEF + tid * 4, true);
  const float4* sp = ckpt + efla_state_slot<D>(id, warp, lane);
  const uint32_t scr_e = base + L::SCRATCH + warp * L::SCR, scr_s = scr_e + L::SCR_E;
  {                                        // dS1 waits in the scratch (every lane reads back its own vectors) until E is done
    const float4* dp = dckpt + efla_state_slot<D>(id, warp, lane);
#pragma unroll
    for (int i = 0; i < D / 8; ++i) cp_async16(scr_s + (i * 32 + lane) * 16, dp + i * 32, true);
  }
  cp_async_commit();
  float S[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i) {
    const float4 f = sp[i * 32];
    S[i][0] = f.x; S[i][1] = f.y; S[i][2] = f.z; S[i][3] = f.w;
  }
  if (tid == 0 && id + ahead < gridDim.x) {                             // the states of the chunk that follows on this SM, into L2
    const long long at = (id + ahead) * (D * D);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<const float*>(ckpt) + at), "r"(D * D * 4) : "memory");
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<const float*>(dckpt) + at), "r"(D * D * 4) : "memory");
  }
  cp_async_wait<0>();
  __syncthreads();

  float* sG = reinterpret_cast<float*>(smem + L::G);
  if (warp < 2) {                          // rows 16 warp .. of the Gram matrix, lower tiles
    float acc[4][4];
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      uint32_t a[4];
      ldsm4(a, base + L::K + ((warp * 16 + (lane & 15)) * L::LD + kk * 16 + (lane >> 4) * 8) * 2);
#pragma unroll
      for (int np = 0; np < 2; ++np) {
        uint32_t bq[4];
        ldsm4(bq, base + L::K + ((np * 16 + (lane & 7) + (lane >> 4) * 8) * L::LD + kk * 16 + ((lane >> 3) & 1) * 8) * 2);
        if (kk == 0) {
          mma_bf16_first(acc[2 * np], a, bq[0], bq[1]);
          mma_bf16_first(acc[2 * np + 1], a, bq[2], bq[3]);
        } else {
          mma_bf16(acc[2 * np], a, bq[0], bq[1]);
          mma_bf16(acc[2 * np + 1], a, bq[2], bq[3]);
        }
      }
    }
#pragma unroll
    for (int nj = 0; nj < 4; ++nj) {
      *reinterpret_cast<float2*>(&sG[(warp * 16 + g) * L::GLD + nj * 8 + 2 * q]) = make_float2(acc[nj][0], acc[nj][1]);
      *reinterpret_cast<float2*>(&sG[(warp * 16 + g + 8) * L::GLD + nj * 8 + 2 * q]) = make_float2(acc[nj][2], acc[nj][3]);
    }
  }

  // E and dE0, and the per-token sums over this warp's value columns
  float e[4][4], de[4][4];
  efla_state_times_k<D>(e, S, base + L::K, lane);
  uint32_t vq[2][4], oq[2][4];
#pragma unroll
  for (int hf = 0; hf < 2; ++hf) {
    ldsm4_t(vq[hf], base + L::V + (lane * L::LD + warp * 16 + hf * 8) * 2);
    ldsm4_t(oq[hf], base + L::O + (lane * L::LD + warp * 16 + hf * 8) * 2);
  }
  efla_errors(e, vq);
  efla_apply_n<false>(e, base + L::N, lane);
  const float4* ds1 = reinterpret_cast<const float4*>(smem + L::SCRATCH + warp * L::SCR + L::SCR_E) + lane;
#pragma unroll
  for (int i = 0; i < D / 8; ++i) {
    const float4 f = ds1[i * 32];
    S[i][0] = f.x; S[i][1] = f.y; S[i][2] = f.z; S[i][3] = f.w;
  }
  efla_state_times_k<D>(de, S, base + L::K, lane);
  float* ssum = reinterpret_cast<float*>(smem + L::SUM) + warp * 2 * EC;
  auto sums_and_de = [&]() {               // the sums of Y E and dO E over the warp's columns; de: from Y to dE
    float t[16];                           // [Y E, dO E][token tile][token 2 q, 2 q + 1]
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const float2 cc = *reinterpret_cast<const float2*>(cf + nt * 8 + 2 * q);
      const float2 ex = *reinterpret_cast<const float2*>(cf + EC + nt * 8 + 2 * q);
      float ye[2] = {0.f, 0.f}, oe[2] = {0.f, 0.f};
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const float o0 = bf16_lo(oq[hf][nt]), o1 = bf16_hi(oq[hf][nt]);
        ye[0] += de[nt][2 * hf] * e[nt][2 * hf];
        ye[1] += de[nt][2 * hf + 1] * e[nt][2 * hf + 1];
        oe[0] += o0 * e[nt][2 * hf];
        oe[1] += o1 * e[nt][2 * hf + 1];
        de[nt][2 * hf] = cc.x * de[nt][2 * hf] - ex.x * o0;
        de[nt][2 * hf + 1] = cc.y * de[nt][2 * hf + 1] - ex.y * o1;
      }
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        t[nt * 2 + x] = ye[x];
        t[8 + nt * 2 + x] = oe[x];
      }
    }
    // over the eight lanes of a q: every step adds half of the sums and hands the others to the lane that adds them (14 exchanges, not 48)
#pragma unroll
    for (int st = 0; st < 3; ++st) {
      const int n = 8 >> st, m = 4 << st;
      const bool upper = lane & m;
#pragma unroll
      for (int i = 0; i < n; ++i) {
        const float give = upper ? t[i] : t[i + n], keep = upper ? t[i + n] : t[i];
        t[i] = keep + __shfl_xor_sync(0xffffffffu, give, m);
      }
    }
    // lane bits 2, 3, 4 say which: Y E or dO E, upper or lower two token tiles, which of the two
    const int nt = (lane >> 3 & 1) * 2 + (lane >> 4 & 1);
    *reinterpret_cast<float2*>(ssum + (lane >> 2 & 1) * EC + nt * 8 + 2 * q) = make_float2(t[0], t[1]);
  };
  sums_and_de();
  efla_apply_n<true>(de, base + L::N, lane);
  if (CHECKED && (efla_any_bad(e) || efla_any_bad(de))) {             // token by token: see efla_walk
    const __nv_bfloat16* tile = reinterpret_cast<const __nv_bfloat16*>(smem);
    float sl[D / 2], el[16], dl[16];
    auto fill = [&](const float4* from) {
#pragma unroll
      for (int i = 0; i < D / 8; ++i) {
        const float4 f = from[i * 32];
        sl[4 * i] = f.x; sl[4 * i + 1] = f.y; sl[4 * i + 2] = f.z; sl[4 * i + 3] = f.w;
      }
    };
    const bool bad_e = efla_any_bad(e), bad_de = efla_any_bad(de);
    float keep[16];
#pragma unroll
    for (int x = 0; x < 16; ++x) {
      keep[x] = de[x / 4][x % 4];
      el[x] = dl[x] = 0.f;                 // tokens past the end
    }
    if (bad_e) {
      fill(sp);
      efla_walk<D, L::LD, L::LD, false>(sl, el, tile + L::K / 2, tile + L::V / 2 + warp * 16, cf, nullptr, 0, 0, n);
#pragma unroll
      for (int x = 0; x < 16; ++x) e[x / 4][x % 4] = el[x];
    }
    fill(ds1);
    efla_rows<D, L::LD>(sl, dl, tile + L::K / 2, n);
#pragma unroll
    for (int x = 0; x < 16; ++x) de[x / 4][x % 4] = dl[x];
    __syncwarp();                          // the sums are written anew
    sums_and_de();
    if (bad_de) efla_walk_back<D, L::LD, L::LD>(sl, dl, tile + L::K / 2, tile + L::O / 2 + warp * 16, cf, n);
#pragma unroll
    for (int x = 0; x < 16; ++x) de[x / 4][x % 4] = bad_de ? dl[x] : keep[x];
  }

  {                                        // dV = dO + dE0, transposed through the scratch
    uint32_t d2[2][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int hf = 0; hf < 2; ++hf)
        d2[hf][nt] = pack_bf16(bf16_lo(oq[hf][nt]) + de[nt][2 * hf], bf16_hi(oq[hf][nt]) + de[nt][2 * hf + 1]);
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) stsm4_t(scr_e + (lane * 24 + hf * 8) * 2, d2[hf][0], d2[hf][1], d2[hf][2], d2[hf][3]);
    __syncwarp();
    const unsigned char* sc = smem + L::SCRATCH + warp * L::SCR;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int t = u * 16 + (lane >> 1), hf = lane & 1;
      if (t < n) *reinterpret_cast<uint4*>(dv + off + t * rs + warp * 16 + hf * 8) = *reinterpret_cast<const uint4*>(sc + (t * 24 + hf * 8) * 2);
    }
    __syncwarp();
  }
  // dK partial (2 x d / 8 tiles) = U dS1^T - dE0 S0^T
  float acc[2][D / 8][4];
  uint32_t a[2][3][4];
#pragma unroll
  for (int term = 0; term < 2; ++term) {
    float w[4][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const float2 cc = *reinterpret_cast<const float2*>(cf + nt * 8 + 2 * q);
#pragma unroll
      for (int x = 0; x < 4; ++x) w[nt][x] = term == 0 ? e[nt][x] * ((x & 1) ? cc.y : cc.x) : -de[nt][x];
    }
    efla_put_tokens(scr_e, w, lane);
#pragma unroll
    for (int i4 = 0; i4 < D / 32; ++i4)
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t s[3][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) split3(S[4 * i4 + u][2 * hf], S[4 * i4 + u][2 * hf + 1], s[0][u], s[1][u], s[2][u]);
#pragma unroll
        for (int p = 0; p < 3; ++p)
          stsm4(scr_s + (p * 16 * L::LD + (hf * 8 + (lane & 7)) * L::LD + i4 * 32 + (lane >> 3) * 8) * 2, s[p][0], s[p][1], s[p][2], s[p][3]);
      }
    if (term == 0) {                       // S0 once more, on its way while these products run
#pragma unroll
      for (int i = 0; i < D / 8; ++i) {
        const float4 f = sp[i * 32];
        S[i][0] = f.x; S[i][1] = f.y; S[i][2] = f.z; S[i][3] = f.w;
      }
    }
    __syncwarp();
#pragma unroll
    for (int mi = 0; mi < 2; ++mi) efla_get_a(a[mi], scr_e, mi, lane);
#pragma unroll
    for (int np = 0; np < D / 16; ++np) {
      uint32_t bq[3][4];
      efla_get_b<L::LD>(bq, scr_s, np, lane);
#pragma unroll
      for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int mi = 0; mi < 2; ++mi) {
          mma_split(acc[mi][2 * np], a[mi], bq, 0, i, term == 0 && i == 0);
          mma_split(acc[mi][2 * np + 1], a[mi], bq, 2, i, term == 0 && i == 0);
        }
    }
    __syncwarp();
  }
  // -dE0 E^T (a still holds -dE0), lower tiles
  float* sda = reinterpret_cast<float*>(smem + L::DA) + warp * EC * L::GLD;
  efla_put_tokens(scr_e, e, lane);
  __syncwarp();
#pragma unroll
  for (int np = 0; np < 2; ++np) {
    uint32_t bq[3][4];
    efla_get_b<EN_LD>(bq, scr_e, np, lane);
#pragma unroll
    for (int mi = np; mi < 2; ++mi)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float da[4];
#pragma unroll
        for (int i = 0; i < 6; ++i) mma_split(da, a[mi], bq, 2 * u, i, i == 0);
        *reinterpret_cast<float2*>(&sda[(mi * 16 + g) * L::GLD + np * 16 + u * 8 + 2 * q]) = make_float2(da[0], da[1]);
        *reinterpret_cast<float2*>(&sda[(mi * 16 + g + 8) * L::GLD + np * 16 + u * 8 + 2 * q]) = make_float2(da[2], da[3]);
      }
  }
  __syncwarp();
  float* red = reinterpret_cast<float*>(smem + L::SCRATCH + warp * L::SCR);
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int i = 0; i < D / 8; ++i) {
      *reinterpret_cast<float2*>(&red[(mi * 16 + g) * L::RED_LD + i * 8 + 2 * q]) = make_float2(acc[mi][i][0], acc[mi][i][1]);
      *reinterpret_cast<float2*>(&red[(mi * 16 + g + 8) * L::RED_LD + i * 8 + 2 * q]) = make_float2(acc[mi][i][2], acc[mi][i][3]);
    }
  __syncthreads();
  // dA = sum over the warps; the symmetric matrix dG + dG^T replaces the first slice of sda, column sums of dA G go to sdc
  float* sym = reinterpret_cast<float*>(smem + L::DA);
  float* sdc = reinterpret_cast<float*>(smem + L::DC);
  {
    float part = 0.f;
    const float c_s = cf[lane];
    for (int t = warp; t < EC; t += L::W) {
      float da = 0.f;
      if (t > lane) {
#pragma unroll
        for (int w = 0; w < L::W; ++w) da += sym[(w * EC + t) * L::GLD + lane];
        part += da * sG[t * L::GLD + lane];
        sym[t * L::GLD + lane] = CHECKED && c_s == 0.f ? 0.f : da * c_s;     // c = 0: a key whose square overflows changes nothing
      }
    }
    sdc[warp * EC + lane] = part;
  }
  __syncthreads();
  if (warp == 0) {
    float ye = 0.f, oe = 0.f, dc = 0.f;
#pragma unroll
    for (int w = 0; w < L::W; ++w) {
      const float* ss = reinterpret_cast<const float*>(smem + L::SUM) + w * 2 * EC;
      ye += ss[lane];
      oe += ss[EC + lane];
      dc += sdc[w * EC + lane];
    }
    dc += ye + cf[2 * EC + lane] * oe;
    sym[lane * L::GLD + lane] = 2.f * (cf[lane] * oe + dc * cf[3 * EC + lane]);
    const float db = lane < n ? dc * cf[EC + lane] : 0.f;
    if (by_chunk) {
      double sum = db;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) dbeta[blockIdx.x] = (float)sum;
    } else if (lane < n) {
      dbeta[((long long)b * T + t0 + lane) * H + h] = db;
    }
  } else {
    for (int t = warp - 1; t < EC; t += L::W - 1)
      if (t < lane) sym[t * L::GLD + lane] = sym[lane * L::GLD + t];
  }
  __syncthreads();
  // key rows 16 warp ..: dK = sum of the partials + sym K
  float dkt[2][2][4];
#pragma unroll
  for (int ks = 0; ks < 2; ++ks) {
    uint32_t b0[4];
    ldsm4_t(b0, base + L::K + ((ks * 16 + (lane & 15)) * L::LD + warp * 16 + (lane >> 4) * 8) * 2);
#pragma unroll
    for (int mi = 0; mi < 2; ++mi) {
      float2 f[4];
      f[0] = *reinterpret_cast<const float2*>(&sym[(mi * 16 + g) * L::GLD + ks * 16 + 2 * q]);
      f[1] = *reinterpret_cast<const float2*>(&sym[(mi * 16 + g + 8) * L::GLD + ks * 16 + 2 * q]);
      f[2] = *reinterpret_cast<const float2*>(&sym[(mi * 16 + g) * L::GLD + ks * 16 + 8 + 2 * q]);
      f[3] = *reinterpret_cast<const float2*>(&sym[(mi * 16 + g + 8) * L::GLD + ks * 16 + 8 + 2 * q]);
      uint32_t hi[4], mid[4], lo[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) split3(f[x].x, f[x].y, hi[x], mid[x], lo[x]);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (ks == 0) mma_bf16_first(dkt[mi][u], lo, b0[2 * u], b0[2 * u + 1]);
        else mma_bf16(dkt[mi][u], lo, b0[2 * u], b0[2 * u + 1]);
        mma_bf16(dkt[mi][u], mid, b0[2 * u], b0[2 * u + 1]);
        mma_bf16(dkt[mi][u], hi, b0[2 * u], b0[2 * u + 1]);
      }
    }
  }
  float chk = 0.f;
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      const int t = mi * 16 + hf * 8 + g;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float2 s = make_float2(dkt[mi][u][2 * hf], dkt[mi][u][2 * hf + 1]);
#pragma unroll
        for (int w = 0; w < L::W; ++w) {
          const float2 r = *reinterpret_cast<const float2*>(reinterpret_cast<const float*>(smem + L::SCRATCH + w * L::SCR) + t * L::RED_LD +
                                                            warp * 16 + u * 8 + 2 * q);
          s.x += r.x;
          s.y += r.y;
        }
        if (t < n) *reinterpret_cast<uint32_t*>(dk + off + t * rs + warp * 16 + u * 8 + 2 * q) = pack_bf16(s.x, s.y);
        chk = fmaf(s.x, 0.f, fmaf(s.y, 0.f, chk));
      }
    }
  return chk != 0.f;                       // an error or gradient that was not finite is in the key gradient of its token
}

template <int D>
__device__ __noinline__ void efla_bwd_chunk_again(const __nv_bfloat16* k, const __nv_bfloat16* v, const __nv_bfloat16* dout,
                                                  const __nv_bfloat16* nmat, const float* coef, const float4* ckpt, const float4* dckpt,
                                                  __nv_bfloat16* dk, __nv_bfloat16* dv, float* dbeta, bool by_chunk, int T, int H, int nchunks) {
  efla_bwd_chunk<D, true>(k, v, dout, nmat, coef, ckpt, dckpt, dk, dv, dbeta, by_chunk, T, H, nchunks, 1 << 30);
}

template <int D>
__global__ void __launch_bounds__(2 * D, D <= 64 ? 2 : 1) efla_chunk_bwd_kernel(
    const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v, const __nv_bfloat16* __restrict__ dout,
    const __nv_bfloat16* __restrict__ nmat, const float* __restrict__ coef, const float4* __restrict__ ckpt,
    const float4* __restrict__ dckpt, __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv,
    float* __restrict__ dbeta, bool by_chunk, int T, int H, int nchunks, int ahead) {
  if (__syncthreads_or(efla_bwd_chunk<D, false>(k, v, dout, nmat, coef, ckpt, dckpt, dk, dv, dbeta, by_chunk, T, H, nchunks, ahead)))
    efla_bwd_chunk_again<D>(k, v, dout, nmat, coef, ckpt, dckpt, dk, dv, dbeta, by_chunk, T, H, nchunks);
}

// out = the sum of the chunks' n terms, in a fixed order and in 64 bits. One CTA is enough: 8192 terms (B 8, T 2048, 16 heads) take what a launch takes, where
// a reduction over the 262144 terms of the tokens took 6 us (whole pass 463 -> 458 us, B 2, T 1531, 8 heads of 128 260 -> 257.5). grid 1, block 1024
__global__ void __launch_bounds__(1024) efla_beta_sum_kernel(const float* __restrict__ part, float* __restrict__ out, int n) {
  __shared__ double red[32];
  double s = 0.;
#pragma unroll 8
  for (int i = threadIdx.x; i < n; i += 1024) s += part[i];
  auto join = [](double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  s = join(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = join(red[threadIdx.x]);
    if (threadIdx.x == 0) *out = (float)s;
  }
}

template <int D>
int launch_chunk_bwd(const void* k, const void* v, const void* nmat, const float* coef, const float* ckpt,
                     const void* dout, const float* dstate_out, void* dk, void* dv, float* dbeta_terms, float* dbeta_sum, float* dstate0, float* dckpt,
                     float* work, int P, int B, int T, int H, cudaStream_t s) {
  using L = EflaStage<D>;
  using M = EflaBwdSmem<D>;
  const int nchunks = (T + EC - 1) / EC;
  const long long total = (long long)B * H * nchunks;
  ELFA_REQUIRE(total < (1ll << 31), "efla_chunk_bwd: too many chunks");
  constexpr int bytes1 = EC_STAGES * L::BYTES;
  const auto* K = static_cast<const __nv_bfloat16*>(k);
  const auto* O = static_cast<const __nv_bfloat16*>(dout);
  const auto* N = static_cast<const __nv_bfloat16*>(nmat);
  ELFA_CUDA(allow_shared<efla_chunk_bwd_kernel<D>>(M::BYTES));
  int seg = nchunks;
  if (P > 1) {
    seg = (nchunks + P - 1) / P;
    P = (nchunks + seg - 1) / seg;
  }
  auto kernel = P > 1 ? efla_chunk_bwd_state_kernel<D, true> : efla_chunk_bwd_state_kernel<D, false>;
  ELFA_CUDA((P > 1 ? allow_shared<efla_chunk_bwd_state_kernel<D, true>>(bytes1) : allow_shared<efla_chunk_bwd_state_kernel<D, false>>(bytes1)));
  auto walk = [&](int phase, int walks) {
    kernel<<<dim3(B * H, D / L::VC, walks), 32 * ec_warps<D>(), bytes1, s>>>(
        K, O, N, coef, dstate_out, reinterpret_cast<float4*>(dckpt), dstate0, work, T, H, nchunks, P, seg, phase);
    ::elfa::count_launches(1);
  };
  if (P <= 1) {
    walk(EFLA_FIRST, 1);
  } else {
    walk(EFLA_FIRST, 2 * P - 3);
    ELFA_CUDA(cudaGetLastError());
    const int rc = launch_combine<D>(coef, work, B * H, nchunks, P, -1, s);
    if (rc != ELFA_OK) return rc;
    walk(EFLA_REST, P - 1);
  }
  ELFA_CUDA(cudaGetLastError());
  efla_chunk_bwd_kernel<D><<<(unsigned)total, 2 * D, M::BYTES, s>>>(
      K, static_cast<const __nv_bfloat16*>(v), O, N, coef, reinterpret_cast<const float4*>(ckpt),
      reinterpret_cast<const float4*>(dckpt), static_cast<__nv_bfloat16*>(dk), static_cast<__nv_bfloat16*>(dv), dbeta_terms, dbeta_sum != nullptr, T, H,
      nchunks, (D <= 64 ? 2 : 1) * (device_sm_count() > 0 ? device_sm_count() : 148));
  ELFA_CUDA(cudaGetLastError());
  ::elfa::count_launches(1);
  if (dbeta_sum) {
    efla_beta_sum_kernel<<<1, 1024, 0, s>>>(dbeta_terms, dbeta_sum, (int)total);
    ELFA_CUDA(cudaGetLastError());
    ::elfa::count_launches(1);
  }
  return ELFA_OK;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace
}  // namespace elfa

using namespace elfa;

// How many segments a walk over T tokens is cut into (1: none), and with them how large `work` is: 3 * segments * B * H * d * d floats.
// One walk takes nchunks steps; cut, FIRST takes nchunks / P steps of (2 P - 3) walks per head and column block and REST as many of P - 1. Measured
// per head dimension: a step with one CTA per SM, with as many as its registers and shared memory hold (whole rounds beyond), and the
// two launches and joints more. Kernels and joints, forward / state gradient, us: B 1 x 8192, 16 heads of 64, P 1 328 / 292, 6 122 / 117, 8 117 / 114,
// 10 100 / 97, 12 128 / 122 (a second round); B 2 x 1531, 8 heads of 128, P 1 106 / 95, 4 82 / 80, 5 74 / 69, 6 79 / 78; B 1 x 4096, 16 heads of 32, P 1
// 110 / 117, 10 33 / 31, 16 33 / 32; not cut: B 4 x 1024, 8 heads of 128, 72 / 65; B 8 x 2048, 16 heads of 64, 86 / 78. Both walks are cut alike: on
// eleven shapes the rule's number is the best for both, or within 5 % of it.
// A cut costs the host two launches and an allocation per walk (6 to 8 us), which only a walk longer than the host's part of the call pays for: about 30 us
// without a gradient, 70 with one, where the rest of the pass runs meanwhile (B 1 x 500, 8 heads of 32, training, cut whatever its length: 159 -> 208 us).
static int efla_segments(int B, int T, int H, int d, double least) {
  const int nchunks = (T + EC - 1) / EC, sms = device_sm_count() > 0 ? device_sm_count() : 148;
  const long long units = (long long)B * H * (d == 128 || d == 96 ? 2 : 1);
  struct Cost { double one, full; int resident; double launches, joint; };      // microseconds
  const Cost c = d == 128 ? Cost{2.1, 3.6, 2, 16, 2.2} : (d == 96 ? Cost{1.76, 2.6, 2, 9, 1.6} : (d == 64 ? Cost{1.4, 1.9, 2, 6, 0.9} : Cost{1.16, 1.4, 4, 4, 0.5}));
  auto steps = [&](long long walks) {
    const long long ctas = units * walks, round = (long long)c.resident * sms, rest = ctas % round;
    return c.full * (double)(ctas / round) + (rest == 0 ? 0. : (rest <= sms ? c.one : c.full));
  };
  const double whole = nchunks * steps(1);
  if (whole < least) return 1;
  double best = 0.9 * whole;                     // cut only where that is clearly less
  int at = 1;
  for (int P = 3; P <= 16 && nchunks / P >= 4; ++P) {
    const int seg = (nchunks + P - 1) / P;
    const double t = seg * (steps(2 * P - 3) + steps(P - 1)) + c.launches + c.joint * (P - 2);
    if (t < best) {
      best = t;
      at = P;
    }
  }
  return at;
}
ELFA_API int elfa_efla_segments(int B, int T, int H, int d) { return efla_segments(B, T, H, d, 30); }
ELFA_API int elfa_efla_segments_train(int B, int T, int H, int d) { return efla_segments(B, T, H, d, 70); }

// k, v, o: [B, T, H, d] bf16, 16-byte aligned; beta: 1 float; state0 (optional) / state_out: [B, H, d, d] fp32; ckpt: null or
// B * H * ceil(T / 32) * d * d floats (chunk-start states in the kernels' own order, needed by backward). nmat: [B * H * ceil(T / 32), 3, 32, 32] bf16 and
// coef: [B * H * ceil(T / 32), 4, 32] fp32, 16-byte aligned, are written here. No output may share memory with an input (a call may run twice).
ELFA_API int elfa_efla_chunk_fwd(const void* k, const void* v, const float* beta, const float* state0, void* o, float* state_out,
                                 float* ckpt, void* nmat, float* coef, int B, int T, int H, int d, void* stream) {
  return elfa_efla_chunk_fwd_cut(k, v, beta, state0, o, state_out, ckpt, nmat, coef, nullptr, 1, B, T, H, d, stream);
}

// The same with the walk in `segments` segments (from elfa_efla_segments, or 1 to T / 128), work: 16-byte aligned scratch of that size.
ELFA_API int elfa_efla_chunk_fwd_cut(const void* k, const void* v, const float* beta, const float* state0, void* o, float* state_out,
                                     float* ckpt, void* nmat, float* coef, float* work, int segments, int B, int T, int H, int d, void* stream) {
  ELFA_REQUIRE(k && v && beta && o && nmat && coef && B > 0 && T > 0 && H > 0, "efla_chunk_fwd: bad arguments");
  ELFA_REQUIRE(segments >= 1 && segments <= 16 && (segments == 1 || work), "efla_chunk_fwd: bad segments");
  ELFA_REQUIRE(aligned16(k) && aligned16(v) && aligned16(o) && aligned16(nmat) && aligned16(coef), "efla_chunk_fwd: operands must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (d) {
    case 32: return launch_chunk_fwd<32>(k, v, beta, state0, o, state_out, ckpt, nmat, coef, work, segments, B, T, H, s);
    case 64: return launch_chunk_fwd<64>(k, v, beta, state0, o, state_out, ckpt, nmat, coef, work, segments, B, T, H, s);
    case 96: return launch_chunk_fwd<96>(k, v, beta, state0, o, state_out, ckpt, nmat, coef, work, segments, B, T, H, s);
    case 128: return launch_chunk_fwd<128>(k, v, beta, state0, o, state_out, ckpt, nmat, coef, work, segments, B, T, H, s);
    default: set_last_error("efla_chunk_fwd: head dimension must be 32, 64, 96 or 128"); return ELFA_ERR_UNSUPPORTED;
  }
}

// Gradients of elfa_efla_chunk_fwd from what it left in nmat, coef and ckpt. dout: [B, T, H, d] bf16; dstate_out: null or [B, H, d, d]
// fp32; dk, dv: [B, T, H, d] bf16; dbeta_tok: [B, T, H] per-token terms (add them up); dstate0: null or [B, H, d, d] fp32; dckpt: scratch
// of ckpt's size.
ELFA_API int elfa_efla_chunk_bwd(const void* k, const void* v, const void* nmat, const float* coef, const float* ckpt, const void* dout,
                                 const float* dstate_out, void* dk, void* dv, float* dbeta_tok, float* dstate0,
                                 float* dckpt, int B, int T, int H, int d, void* stream) {
  return elfa_efla_chunk_bwd_cut(k, v, nmat, coef, ckpt, dout, dstate_out, dk, dv, dbeta_tok, dstate0, dckpt, nullptr, 1, B, T, H, d, stream);
}

// The same in segments, see elfa_efla_chunk_fwd_cut. (Training takes the sum below; these two are for callers that want the terms of beta's gradient per
// token, the tests of that sum among them.)
ELFA_API int elfa_efla_chunk_bwd_cut(const void* k, const void* v, const void* nmat, const float* coef, const float* ckpt, const void* dout,
                                     const float* dstate_out, void* dk, void* dv, float* dbeta_tok, float* dstate0,
                                     float* dckpt, float* work, int segments, int B, int T, int H, int d, void* stream) {
  return elfa_efla_chunk_bwd_sum(k, v, nmat, coef, ckpt, dout, dstate_out, dk, dv, dbeta_tok, nullptr, dstate0, dckpt, work, segments, B, T, H, d, stream);
}

// The same with the sum of the terms in dbeta (1 float); dbeta_terms: scratch of B * H * ceil(T / 32) floats then, and [B, T, H] where dbeta is null.
ELFA_API int elfa_efla_chunk_bwd_sum(const void* k, const void* v, const void* nmat, const float* coef, const float* ckpt, const void* dout,
                                     const float* dstate_out, void* dk, void* dv, float* dbeta_terms, float* dbeta, float* dstate0,
                                     float* dckpt, float* work, int segments, int B, int T, int H, int d, void* stream) {
  ELFA_REQUIRE(segments >= 1 && segments <= 16 && (segments == 1 || work), "efla_chunk_bwd: bad segments");
  ELFA_REQUIRE(k && v && nmat && coef && ckpt && dout && dk && dv && dbeta_terms && dckpt && B > 0 && T > 0 && H > 0,
               "efla_chunk_bwd: bad arguments");
  ELFA_REQUIRE(aligned16(k) && aligned16(v) && aligned16(nmat) && aligned16(coef) && aligned16(ckpt) && aligned16(dout) && aligned16(dk) &&
                   aligned16(dv) && aligned16(dckpt),
               "efla_chunk_bwd: operands must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (d) {
    case 32: return launch_chunk_bwd<32>(k, v, nmat, coef, ckpt, dout, dstate_out, dk, dv, dbeta_terms, dbeta, dstate0, dckpt, work, segments, B, T, H, s);
    case 64: return launch_chunk_bwd<64>(k, v, nmat, coef, ckpt, dout, dstate_out, dk, dv, dbeta_terms, dbeta, dstate0, dckpt, work, segments, B, T, H, s);
    case 96: return launch_chunk_bwd<96>(k, v, nmat, coef, ckpt, dout, dstate_out, dk, dv, dbeta_terms, dbeta, dstate0, dckpt, work, segments, B, T, H, s);
    case 128: return launch_chunk_bwd<128>(k, v, nmat, coef, ckpt, dout, dstate_out, dk, dv, dbeta_terms, dbeta, dstate0, dckpt, work, segments, B, T, H, s);
    default: set_last_error("efla_chunk_bwd: head dimension must be 32, 64, 96 or 128"); return ELFA_ERR_UNSUPPORTED;
  }
}
