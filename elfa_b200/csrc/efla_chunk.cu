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
// reference: kernels/cuda/efla.cu:121-271,534-552 (chunks are scanned one after the other, the bf16 state in global memory).
#include "common.cuh"
#include "elfa_native.h"
#include "efla_math.cuh"
#include "mma_sync.cuh"

namespace elfa {
namespace {

constexpr int EC = 32;                     // tokens of a chunk
constexpr int EN_LD = 40;                  // row pitch of N in shared memory (bf16)
constexpr int EN_ELEMS = 3 * EC * EC;      // one chunk's N: [split][t][s] bf16 in global memory

// ------------------------------------------------------------------------------------------------ state-independent part
// One warp per (batch, head, chunk): Gram matrix by mma.sync (exact bf16 products), then lane s eliminates column s of the unit
// lower triangular matrix by forward substitution in fp32 registers (496 multiply-adds, rows broadcast from shared memory).
// coef: [.., 0][t] = c, [.., 1][t] = ex. Tokens past the end have k = 0: they change neither the state nor another token.
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
  for (int i = lane; i < EC * (D / 8); i += 32) {
    const int r = i / (D / 8), c = i % (D / 8);
    const uint4 z = make_uint4(0, 0, 0, 0);
    *reinterpret_cast<uint4*>(sk + r * LD + c * 8) = r < n ? *reinterpret_cast<const uint4*>(kb + (long long)r * H * D + c * 8) : z;
  }
  __syncwarp();
  const uint32_t ks = smem_u32(sk);
#pragma unroll
  for (int mi = 0; mi < 2; ++mi) {
    float acc[4][4];
#pragma unroll
    for (int nj = 0; nj < 4; ++nj)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[nj][e] = 0.f;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      uint32_t a[4];
      ldsm4(a, ks + ((mi * 16 + (lane & 15)) * LD + kk * 16 + (lane >> 4) * 8) * 2);
#pragma unroll
      for (int np = 0; np <= mi; ++np) {   // token columns 16 np .. 16 np + 15: the strictly upper tiles are not needed
        uint32_t bq[4];
        ldsm4(bq, ks + ((np * 16 + (lane & 7) + (lane >> 4) * 8) * LD + kk * 16 + ((lane >> 3) & 1) * 8) * 2);
        mma_bf16(acc[2 * np], a, bq[0], bq[1]);
        mma_bf16(acc[2 * np + 1], a, bq[2], bq[3]);
      }
    }
#pragma unroll
    for (int nj = 0; nj < 2 * mi + 2; ++nj) {
      *reinterpret_cast<float2*>(&sg[mi * 16 + g][nj * 8 + 2 * q]) = make_float2(acc[nj][0], acc[nj][1]);
      *reinterpret_cast<float2*>(&sg[mi * 16 + g + 8][nj * 8 + 2 * q]) = make_float2(acc[nj][2], acc[nj][3]);
    }
  }
  __syncwarp();
  float c_, d1, d2;
  const float lam = sg[lane][lane], beta = *beta_ptr;
  efla_coeff(beta, lam, c_, d1, d2);
  const float ex = lam < 1e-6f ? 1.f - c_ * lam : d1;
  coef[id * 2 * EC + lane] = c_;
  coef[id * 2 * EC + EC + lane] = ex;
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
  __nv_bfloat16* out = nmat + id * EN_ELEMS;
#pragma unroll
  for (int t = 0; t < EC; t += 2) {
    uint32_t hi, mid, lo;
    split3(t > lane ? x[t] : 0.f, t + 1 > lane ? x[t + 1] : 0.f, hi, mid, lo);
    uint16_t* o16 = reinterpret_cast<uint16_t*>(out);
    o16[t * EC + lane] = (uint16_t)hi;
    o16[(t + 1) * EC + lane] = (uint16_t)(hi >> 16);
    o16[EC * EC + t * EC + lane] = (uint16_t)mid;
    o16[EC * EC + (t + 1) * EC + lane] = (uint16_t)(mid >> 16);
    o16[2 * EC * EC + t * EC + lane] = (uint16_t)lo;
    o16[2 * EC * EC + (t + 1) * EC + lane] = (uint16_t)(lo >> 16);
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
  static constexpr int K = 0, V = K + EC * KLD * 2, N = V + EC * VLD * 2, C = N + 3 * EC * EN_LD * 2, BYTES = C + 2 * EC * 4;
};

template <int D>
__device__ __forceinline__ void efla_stage_load(uint32_t st, const __nv_bfloat16* __restrict__ kb, const __nv_bfloat16* __restrict__ vb,
                                                const __nv_bfloat16* __restrict__ nm, const float* __restrict__ cf, long long row_stride,
                                                int n) {
  using L = EflaStage<D>;
  constexpr int NT = 32 * ec_warps<D>();
  for (int i = threadIdx.x; i < EC * (D / 8); i += NT) {
    const int r = i / (D / 8), c = i % (D / 8);
    cp_async16(st + L::K + (r * L::KLD + c * 8) * 2, kb + (r < n ? r : 0) * row_stride + c * 8, r < n);
  }
  for (int i = threadIdx.x; i < EC * (L::VC / 8); i += NT) {
    const int r = i / (L::VC / 8), c = i % (L::VC / 8);
    cp_async16(st + L::V + (r * L::VLD + c * 8) * 2, vb + (r < n ? r : 0) * row_stride + c * 8, r < n);
  }
  for (int i = threadIdx.x; i < 3 * EC * 4; i += NT)
    cp_async16(st + L::N + ((i / 4) * EN_LD + (i % 4) * 8) * 2, nm + i * 8, true);
  if (threadIdx.x < 2 * EC / 4) cp_async16(st + L::C + threadIdx.x * 16, cf + threadIdx.x * 4, true);
}

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
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int x = 0; x < 4; ++x) acc[nt][x] = 0.f;
#pragma unroll
  for (int p = 2; p >= 0; --p) {           // splits of N, small ones first
    uint32_t bf[4][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      if (TRANS) ldsm4_t(bf[nt], nbase + (p * EC * EN_LD + lane * EN_LD + nt * 8) * 2);      // rows t, columns r of tile nt
      else ldsm4(bf[nt], nbase + (p * EC * EN_LD + (nt * 8 + (lane & 7)) * EN_LD + (lane >> 3) * 8) * 2);
    }
#pragma unroll
    for (int m = 2 - p; m >= 0; --m)       // splits of e that still count against this split of N
#pragma unroll
      for (int ks = 0; ks < 2; ++ks)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          if (TRANS ? (nt >= 2 && ks == 0) : (nt < 2 && ks == 1)) continue;                 // zero blocks of the triangle
          mma_bf16(acc[nt], m == 0 ? ah[ks] : (m == 1 ? am[ks] : al[ks]), bf[nt][2 * ks], bf[nt][2 * ks + 1]);
        }
  }
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int x = 0; x < 4; ++x) e[nt][x] += acc[nt][x];
}

// p[16 x 32] = S^T K^T for the warp's S^T tiles (rows = value columns, columns = tokens)
template <int D>
__device__ __forceinline__ void efla_state_times_k(float (&p)[4][4], const float (&S)[D / 8][4], uint32_t kbase, int lane) {
  constexpr int LD = EflaStage<D>::KLD;
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int x = 0; x < 4; ++x) p[nt][x] = 0.f;
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
      for (int nt = 0; nt < 4; ++nt) mma_bf16(p[nt], lo, bq[nt][2 * u], bq[nt][2 * u + 1]);
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
    for (int n = 0; n < 4; ++n) {
      ldsm4_t(bq[n], kbase + (lane * LD + (n0 + n) * 8) * 2);
#pragma unroll
      for (int x = 0; x < 4; ++x) acc[n][x] = 0.f;
    }
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
      for (int ks = 0; ks < 2; ++ks)
#pragma unroll
        for (int n = 0; n < 4; ++n)
          mma_bf16(acc[n], p == 0 ? lo[ks] : (p == 1 ? mid[ks] : hi[ks]), bq[n][2 * ks], bq[n][2 * ks + 1]);
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int x = 0; x < 4; ++x) S[n0 + n][x] = SUB ? S[n0 + n][x] - acc[n][x] : S[n0 + n][x] + acc[n][x];
  }
}

// Grid (B * H, d / columns of a CTA). k, v, o: [B, T, H, d] bf16. state0 / state_out: [B, H, d, d] fp32 or null. ckpt (or null):
// [B, H, nchunks, d, d] fp32, the state at the start of every chunk.
// Bound by the dependent chain of a chunk (about 130 mma.sync and 700 instructions of one warp per scheduler), not by memory. With the
// preparation, B 1, T 8192, 16 heads of 64, no gradient: 397 us, token by token (with its checkpoints) 2364 us; in the training step of
// B 8, T 2048 the forward went from about 0.75 to 0.13 ms.
template <int D>
__global__ void __launch_bounds__(32 * ec_warps<D>()) efla_chunk_fwd_kernel(
    const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v, const __nv_bfloat16* __restrict__ nmat,
    const float* __restrict__ coef, const float* __restrict__ state0, __nv_bfloat16* __restrict__ o, float* __restrict__ state_out,
    float* __restrict__ ckpt, int T, int H, int nchunks) {
  using L = EflaStage<D>;
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int bh = blockIdx.x, b = bh / H, h = bh % H;
  const int ccol = blockIdx.y * L::VC, wcol = ccol + warp * 16;       // first value column of the CTA / of this warp
  const uint32_t ring = smem_u32(smem);
  __nv_bfloat16* stage_o = reinterpret_cast<__nv_bfloat16*>(smem + EC_STAGES * L::BYTES) + warp * EC * 24;   // [32 tokens][16 + 8]
  const long long row0 = ((long long)b * T * H + h) * D, rs = (long long)H * D;
  const __nv_bfloat16 *kb = k + row0, *vb = v + row0 + ccol;
  const __nv_bfloat16* nb = nmat + (long long)bh * nchunks * EN_ELEMS;
  const float* cb = coef + (long long)bh * nchunks * 2 * EC;

  float S[D / 8][4];                       // S^T: value column g (+ 8), key row 8 n + 2q (+ 1)
#pragma unroll
  for (int n = 0; n < D / 8; ++n)
#pragma unroll
    for (int x = 0; x < 4; ++x)
      S[n][x] = state0 ? state0[((long long)bh * D + n * 8 + 2 * q + (x & 1)) * D + wcol + g + (x >> 1) * 8] : 0.f;

  auto fetch = [&](int ch) {
    if (ch < nchunks)
      efla_stage_load<D>(ring + (ch % EC_STAGES) * L::BYTES, kb + (long long)ch * EC * rs, vb + (long long)ch * EC * rs,
                         nb + (long long)ch * EN_ELEMS, cb + (long long)ch * 2 * EC, rs, min(EC, T - ch * EC));
    cp_async_commit();
  };
#pragma unroll
  for (int i = 0; i < EC_STAGES - 1; ++i) fetch(i);
  for (int ch = 0; ch < nchunks; ++ch) {
    cp_async_wait<EC_STAGES - 2>();
    __syncthreads();                       // chunk ch has landed for every thread; the stage of chunk ch - 1 is free
    fetch(ch + EC_STAGES - 1);
    const uint32_t st = ring + (ch % EC_STAGES) * L::BYTES;
    const float* cf = reinterpret_cast<const float*>(smem + (ch % EC_STAGES) * L::BYTES + L::C);
    if (ckpt) {
      float* dst = ckpt + ((long long)bh * nchunks + ch) * D * D + wcol + g;
#pragma unroll
      for (int n = 0; n < D / 8; ++n)
#pragma unroll
        for (int x = 0; x < 4; ++x) dst[(n * 8 + 2 * q + (x & 1)) * D + (x >> 1) * 8] = S[n][x];
    }
    float e[4][4];
    efla_state_times_k<D>(e, S, st + L::K, lane);
    uint32_t vq[2][4];                     // V^T tiles: [value half][token tile], tokens 2q, 2q + 1 of column g
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) ldsm4_t(vq[hf], st + L::V + (lane * L::VLD + warp * 16 + hf * 8) * 2);
    float chk = 0.f;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float vv = (x & 1) ? bf16_hi(vq[x >> 1][nt]) : bf16_lo(vq[x >> 1][nt]);
        e[nt][x] = vv - e[nt][x];
        chk = fmaf(e[nt][x], 0.f, chk);
      }
    // a non-finite error stays with its token and the later ones: it is taken out of the product (0 x NaN would reach the earlier
    // tokens of the chunk) and put back behind it
    const bool bad = __any_sync(0xffffffffu, chk != 0.f);
    int first[2] = {EC, EC};
    if (bad) {
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
    efla_apply_n<false>(e, st + L::N, lane);
    if (bad) {
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (nt * 8 + 2 * q + (x & 1) >= first[x >> 1]) e[nt][x] = __int_as_float(0x7fffffff);
    }
    uint32_t oq[2][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const float2 ex = *reinterpret_cast<const float2*>(cf + EC + nt * 8 + 2 * q);
      const float2 cc = *reinterpret_cast<const float2*>(cf + nt * 8 + 2 * q);
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        oq[hf][nt] = pack_bf16(fmaf(-ex.x, e[nt][2 * hf], bf16_lo(vq[hf][nt])), fmaf(-ex.y, e[nt][2 * hf + 1], bf16_hi(vq[hf][nt])));
        e[nt][2 * hf] *= cc.x;
        e[nt][2 * hf + 1] *= cc.y;
      }
    }
    efla_state_update<D, false>(S, e, st + L::K, lane);
    const uint32_t so = smem_u32(stage_o);
    __syncwarp();
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) stsm4_t(so + (lane * 24 + hf * 8) * 2, oq[hf][0], oq[hf][1], oq[hf][2], oq[hf][3]);
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int t = u * 16 + (lane >> 1), hf = lane & 1;
      if (ch * EC + t < T)
        *reinterpret_cast<uint4*>(o + row0 + ((long long)ch * EC + t) * rs + wcol + hf * 8) = *reinterpret_cast<const uint4*>(stage_o + t * 24 + hf * 8);
    }
  }
  cp_async_wait<0>();
  if (state_out) {
#pragma unroll
    for (int n = 0; n < D / 8; ++n)
#pragma unroll
      for (int x = 0; x < 4; ++x)
        state_out[((long long)bh * D + n * 8 + 2 * q + (x & 1)) * D + wcol + g + (x >> 1) * 8] = S[n][x];
  }
}

template <int D>
int launch_chunk_fwd(const void* k, const void* v, const float* beta, const float* state0, void* o, float* state_out, float* ckpt,
                     void* nmat, float* coef, int B, int T, int H, cudaStream_t s) {
  using L = EflaStage<D>;
  const int nchunks = (T + EC - 1) / EC;
  const long long total = (long long)B * H * nchunks;
  ELFA_REQUIRE((total + 1) / 2 < (1ll << 31), "efla_chunk_fwd: too many chunks");
  efla_prep_kernel<D><<<(unsigned)((total + 1) / 2), 64, 0, s>>>(static_cast<const __nv_bfloat16*>(k), beta, static_cast<__nv_bfloat16*>(nmat),
                                                                 coef, T, H, nchunks, total);
  ELFA_CUDA(cudaGetLastError());
  constexpr int bytes = EC_STAGES * L::BYTES + ec_warps<D>() * EC * 24 * 2;
  ELFA_CUDA(cudaFuncSetAttribute(efla_chunk_fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  efla_chunk_fwd_kernel<D><<<dim3(B * H, D / L::VC), 32 * ec_warps<D>(), bytes, s>>>(
      static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v), static_cast<const __nv_bfloat16*>(nmat), coef, state0,
      static_cast<__nv_bfloat16*>(o), state_out, ckpt, T, H, nchunks);
  ELFA_CUDA(cudaGetLastError());
  ::elfa::count_launches(2);
  return ELFA_OK;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace
}  // namespace elfa

using namespace elfa;

// k, v, o: [B, T, H, d] bf16, 16-byte aligned; beta: 1 float; state0 (optional) / state_out: [B, H, d, d] fp32; ckpt: null or
// [B, H, ceil(T / 32), d, d] fp32 (chunk-start states, needed by backward). nmat: [B * H * ceil(T / 32), 3, 32, 32] bf16 and
// coef: [B * H * ceil(T / 32), 2, 32] fp32, 16-byte aligned, are written here.
ELFA_API int elfa_efla_chunk_fwd(const void* k, const void* v, const float* beta, const float* state0, void* o, float* state_out,
                                 float* ckpt, void* nmat, float* coef, int B, int T, int H, int d, void* stream) {
  ELFA_REQUIRE(k && v && beta && o && nmat && coef && B > 0 && T > 0 && H > 0, "efla_chunk_fwd: bad arguments");
  ELFA_REQUIRE(aligned16(k) && aligned16(v) && aligned16(o) && aligned16(nmat) && aligned16(coef), "efla_chunk_fwd: operands must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (d) {
    case 32: return launch_chunk_fwd<32>(k, v, beta, state0, o, state_out, ckpt, nmat, coef, B, T, H, s);
    case 64: return launch_chunk_fwd<64>(k, v, beta, state0, o, state_out, ckpt, nmat, coef, B, T, H, s);
    case 96: return launch_chunk_fwd<96>(k, v, beta, state0, o, state_out, ckpt, nmat, coef, B, T, H, s);
    case 128: return launch_chunk_fwd<128>(k, v, beta, state0, o, state_out, ckpt, nmat, coef, B, T, H, s);
    default: set_last_error("efla_chunk_fwd: head dimension must be 32, 64, 96 or 128"); return ELFA_ERR_UNSUPPORTED;
  }
}
