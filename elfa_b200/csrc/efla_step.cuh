// The EFLA recurrence and the ShortConv of a stream, a few tokens at a time: the bodies of the kernels in efla.cu, which decode.cu runs inside a whole
// decoding step.
#pragma once
#include "common.cuh"

namespace elfa {

__device__ __forceinline__ float efla_coeff(float beta, float lam) {
  // expm1f: 1 - exp would cancel for short keys (at beta lam = 1e-6 one step of fp32 is 6 %, and the chunked form has c in fp64)
  return lam < 1e-30f ? beta : -expm1f(-beta * lam) / lam;
}

// Token by token, for short blocks without a gradient (generation; the line is in ops/efla.py): one launch, nothing else to prepare.
// k, v, o: [B, T, H, D] bf16. state0 / state_out: [B, H, D, D] fp32.
// The columns of S evolve independently (column j needs k_t, c_t and v_t[j] only), so a CTA owns 32 value columns:
// grid (B*H, D/32). Its four warps split the D key rows: warp w keeps rows [w D/4, (w+1) D/4) of the 32 columns in
// registers (lane = column), so the dependent instruction chain of a step is a quarter as long and the four
// schedulers of the SM all have a warp. A step costs one block barrier: the warps exchange their partial dot
// products through a parity-double-buffered shared array. Time is walked in tiles of EFLA_TT tokens: every warp
// fetches its rows of the tile with all loads in flight together (keys as fp32, the CTA's 32 value columns) and computes
// their lam / c from registers, and the sequential part touches global memory only for the output.
constexpr int EFLA_TT = 32;
constexpr int EFLA_W = 4;

// Shared memory of the four warps, for tiles of TT tokens
template <int D, int TT>
struct EflaStepScratch {
  alignas(16) float k[TT][D];
  float v[TT][32];
  float c[TT], lam[TT];
  float part[2][EFLA_W * 32];
};

// A warp fetches TT / 4 rows and forms their lam / c from what it holds
template <int D, int TT>
__device__ __forceinline__ void efla_load_tile(const __nv_bfloat16* k, const __nv_bfloat16* v, EflaStepScratch<D, TT>& sm, float beta,
                                               long long row0, long long row_stride, int col, int n, int warp, int lane) {
  constexpr int PER = TT / EFLA_W;
  const int r0 = warp * PER;
  if (r0 >= n) return;
  __nv_bfloat16 kq[PER][D / 32], vq[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const long long row = row0 + (long long)min(r0 + u, n - 1) * row_stride;        // clamped: rows past the end re-read the last one
#pragma unroll
    for (int c = 0; c < D / 32; ++c) kq[u][c] = k[row + c * 32 + lane];
    vq[u] = v[row + col];
  }
  float own = 0.f;
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    float lam = 0.f;
#pragma unroll
    for (int c = 0; c < D / 32; ++c) {
      const float x = __bfloat162float(kq[u][c]);
      sm.k[r0 + u][c * 32 + lane] = x;
      lam += x * x;
    }
    sm.v[r0 + u][lane] = __bfloat162float(vq[u]);
    lam = warp_sum(lam);
    if (lane == u) own = lam;
  }
  if (lane < PER) {
    sm.c[r0 + lane] = efla_coeff(beta, own);
    sm.lam[r0 + lane] = own;
  }
}

// One step of the recurrence for this warp's R rows: returns p (complete, after the exchange) and applies the update.
template <int R, typename Sync>
__device__ __forceinline__ float efla_step(float (&S)[R], const float* krow, float c_, float vj, float* part, int warp, int lane, Sync together) {
  const float4* kr = reinterpret_cast<const float4*>(krow);
  float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
#pragma unroll
  for (int i = 0; i < R / 4; ++i) {
    const float4 kk = kr[i];
    p0 += kk.x * S[4 * i];
    p1 += kk.y * S[4 * i + 1];
    p2 += kk.z * S[4 * i + 2];
    p3 += kk.w * S[4 * i + 3];
  }
  part[warp * 32 + lane] = (p0 + p1) + (p2 + p3);
  together();
  const float p = (part[lane] + part[32 + lane]) + (part[64 + lane] + part[96 + lane]);
  const float ce = c_ * (vj - p);
#pragma unroll
  for (int i = 0; i < R / 4; ++i) {
    const float4 kk = kr[i];
    S[4 * i] += kk.x * ce;
    S[4 * i + 1] += kk.y * ce;
    S[4 * i + 2] += kk.z * ce;
    S[4 * i + 3] += kk.w * ce;
  }
  return p;
}

// All T tokens of (batch, head) bh for the value columns 32 block .. 32 block + 31: 128 threads (tid), `together` a barrier of theirs
template <int D, int TT, typename Sync>
__device__ __forceinline__ void efla_scan_block(const __nv_bfloat16* k, const __nv_bfloat16* v, const float* beta_ptr, const float* state0,
                                                __nv_bfloat16* o, float* state_out, int T, int H, int bh, int block, EflaStepScratch<D, TT>& sm,
                                                int tid, Sync together) {
  constexpr int R = D / EFLA_W;
  const int b = bh / H, h = bh % H, lane = tid & 31, warp = tid >> 5;
  const int col = block * 32 + lane, i0 = warp * R;
  const float beta = *beta_ptr;
  float S[R];
#pragma unroll
  for (int i = 0; i < R; ++i) S[i] = state0 ? state0[((long long)bh * D + i0 + i) * D + col] : 0.f;
#pragma unroll 1
  for (int t0 = 0; t0 < T; t0 += TT) {
    const int n = min(TT, T - t0);
    if (t0) together();                                  // the previous tile has been consumed
    efla_load_tile<D, TT>(k, v, sm, beta, (((long long)b * T + t0) * H + h) * D, (long long)H * D, col, n, warp, lane);
    together();
#pragma unroll 1
    for (int r = 0; r < n; ++r) {
      const int t = t0 + r;
      const float c_ = sm.c[r], vj = sm.v[r][lane];
      const float p = efla_step<R>(S, sm.k[r] + i0, c_, vj, sm.part[r & 1], warp, lane, together);
      if (warp == 0) o[(((long long)b * T + t) * H + h) * D + col] = __float2bfloat16(p + c_ * sm.lam[r] * (vj - p));
    }
  }
  if (state_out) {
#pragma unroll
    for (int i = 0; i < R; ++i) state_out[((long long)bh * D + i0 + i) * D + col] = S[i];
  }
}

// Channels c and c + 1 of position t (of T) behind `tails` kept ones; at(i): the two channels at position i of tail and inputs side by side; xb: the
// channels' place in the copy of the two, whose position t (COPY: and at t == 0 the tail) is written here; u: the output's place. RING: see
// shortconv_stream_kernel.
template <bool RING, bool COPY = true, typename At>
__device__ __forceinline__ void shortconv_stream_pair(At at, const __nv_bfloat16* w, const __nv_bfloat16* bias, __nv_bfloat16* xb, __nv_bfloat16* u,
                                                      int tails, int t, int c, int C, int W) {
  if (COPY && t == 0)
#pragma unroll 8
    for (int i = 0; i < tails; ++i) *reinterpret_cast<uint32_t*>(xb + (long long)i * C) = at(i);
  *reinterpret_cast<uint32_t*>(xb + (long long)(tails + t) * C) = at(tails + t);
  float s[2][2] = {{0.f, 0.f}, {0.f, 0.f}};                            // [chain][channel]
  if (bias) {
    s[0][0] = __bfloat162float(bias[c]);
    s[0][1] = __bfloat162float(bias[c + 1]);
  }
  const int taps = min(W, tails + t + 1);
#pragma unroll 8
  for (int j = 0; j < taps; ++j) {
    const uint32_t x = at(tails + t - j);
    const int k = RING ? j & 1 : 0;
    s[k][0] = fmaf(bf16_lo(x), __bfloat162float(w[(long long)c * W + j]), s[k][0]);
    s[k][1] = fmaf(bf16_hi(x), __bfloat162float(w[(long long)(c + 1) * W + j]), s[k][1]);
  }
  if (RING) {
    s[0][0] += s[1][0];
    s[0][1] += s[1][1];
  }
  *reinterpret_cast<uint32_t*>(u) = pack_bf16(s[0][0], s[0][1]);
}

}  // namespace elfa
