// EFLA recurrence token by token (blocks of up to about a hundred tokens without a gradient; the others and backward: efla_chunk.cu) and the causal depthwise
// ShortConv (forward and backward).
//
// EFLA, per (batch, head), state S [d, d] fp32 (row = key index i, column = value index j):
//   lam = |k|^2, c = (1 - exp(-beta lam)) / lam, p = S^T k, e = v - p, S += c k e^T, o = p + c lam e
// (o equals S_new^T k): one CTA of four warps per (batch, head, 32 value columns); its threads keep the state in registers for all
// tokens so it never leaves the chip and is never rounded to bf16 - the reference rounds the bf16 state in global memory on every
// token and launches once per chunk (reference: kernels/cuda/efla.cu:121-197; fp32 variant kernels/cuda/efla_scan.cu:99-152; CPU math
// src/model/efla.zig:27-49,275-329).
//
// ShortConv: y[b,t,c] = bias[c] + sum_w x[b,t-w,c] weight[c,w] (reference:
// kernels/cuda/convolution.cu:4-57,126-189; src/model/prism.zig:948-973). The weight gradient is
// summed in slices of the rows, which are added up in order (no atomics).
#include <algorithm>
#include <type_traits>

#include "efla_step.cuh"
#include "elfa_native.h"

namespace elfa {
namespace {

template <int D>
__global__ void __launch_bounds__(32 * EFLA_W) efla_scan_fwd_kernel(const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v,
                                                                    const float* __restrict__ beta_ptr, const float* __restrict__ state0,
                                                                    __nv_bfloat16* __restrict__ o, float* __restrict__ state_out, int T, int H) {
  __shared__ EflaStepScratch<D, EFLA_TT> sm;
  efla_scan_block<D, EFLA_TT>(k, v, beta_ptr, state0, o, state_out, T, H, blockIdx.x, blockIdx.y, sm, threadIdx.x, [] { __syncthreads(); });
}

// ------------------------------------------------------------------------------------ ShortConv
// Windows of 4, 8 and 16 taps: a warp owns 64 channels (a pair per lane) of one sequence and walks over `span` consecutive time steps with
// the last W inputs and the W weights in registers (the loop is unrolled W steps, so the window is a ring with fixed register names);
// every input element is loaded once per span plus the W - 1 steps of the seam, the next W rows are in flight while the current
// ones are summed, and the sums run on packed fp32 pairs. Other windows (larger rings do not fit the registers) take
// shortconv_tile_kernel / shortconv_dw_kernel below.
// Backward is one walk from late to early: with dy[t .. t + W - 1] as the window, dx[t] = sum_j w[j] dy[t + j] and
// dw[j] += x[t] dy[t + j]; every warp writes its dw / db sums as one slice of part [slices][W + 1][C], added up in order afterwards.
// B 8, T 2048, C 1024, W 16: 25 us forward (67 MB; bound by the packed multiply-adds and the latency of 202- and 128-register warps; 27 with a test and
// a 64-bit multiplication per load, which are kept in backward: 45 us with them, 50 without), 45 + 6 us backward; the
// layer that contains them went from 789 to 454 us when they replaced kernels that took a tap at a time.
// A lane's weights are 4 W consecutive bytes; one at a time they would cost 2 W loads that touch 32 lines each, more than the
// inputs (31.5 against 26.5 us forward).
template <int W>
__device__ __forceinline__ void shortconv_weights(uint64_t (&wf)[W], const __nv_bfloat16* __restrict__ w, int c) {
  uint32_t q[W];                           // channel c in the first half, c + 1 in the second, two taps each
  const __nv_bfloat16* wc = w + (long long)c * W;
  if ((reinterpret_cast<uintptr_t>(w) & 15) == 0) {      // c is even: every lane starts on 16 bytes
#pragma unroll
    for (int i = 0; i < W / 4; ++i) {
      const uint4 v = reinterpret_cast<const uint4*>(wc)[i];
      q[4 * i] = v.x; q[4 * i + 1] = v.y; q[4 * i + 2] = v.z; q[4 * i + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < W; ++i) q[i] = (uint32_t)__bfloat16_as_ushort(wc[2 * i]) | (uint32_t)__bfloat16_as_ushort(wc[2 * i + 1]) << 16;
  }
#pragma unroll
  for (int j = 0; j < W; j += 2) {
    wf[j] = pack_f32x2(bf16_lo(q[j / 2]), bf16_lo(q[W / 2 + j / 2]));
    wf[j + 1] = pack_f32x2(bf16_hi(q[j / 2]), bf16_hi(q[W / 2 + j / 2]));
  }
}
__device__ __forceinline__ uint32_t ld_pair(const __nv_bfloat16* base, long long row, long long C, bool ok) {
  return ok ? *reinterpret_cast<const uint32_t*>(base + row * C) : 0u;
}
// Rows row, row + dir, ...; `inside`: all of them exist (a test and a multiplication less per load), otherwise those of ok(i).
template <int N, class Ok>
__device__ __forceinline__ void ld_rows(uint32_t (&q)[N], const __nv_bfloat16* base, long long row, long long C, int dir, bool inside, Ok ok) {
  if (inside) {
    const __nv_bfloat16* p = base + row * C;
    const long long step = dir * C;
#pragma unroll
    for (int i = 0; i < N; ++i, p += step) q[i] = *reinterpret_cast<const uint32_t*>(p);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) q[i] = ld_pair(base, row + dir * i, C, ok(i));
  }
}
__device__ __forceinline__ uint64_t pair_f32x2(uint32_t v) { return pack_f32x2(bf16_lo(v), bf16_hi(v)); }

// The ring stands in zeros for what lies outside the sequence, and 0 x infinity is NaN. Forward leaves those products out of a sequence's first
// W outputs. Backward looks, where its walk reaches past the end, for values that are not finite (weights; the sums of tap 0 and of the
// bias, which see every input and output gradient of the walk) and then forms the same sums again, in the same order, without them.
__device__ __forceinline__ bool not_finite_f32x2(uint64_t v) {
  float lo, hi;
  unpack_f32x2(v, lo, hi);
  return fmaf(lo, 0.f, hi * 0.f) != 0.f;
}
template <int W>
__device__ __forceinline__ bool shortconv_weights_bad(const uint64_t (&wf)[W]) {
  uint64_t z = 0ull;
#pragma unroll
  for (int j = 0; j < W; ++j) z = fma_f32x2(wf[j], 0ull, z);
  return not_finite_f32x2(z);
}
template <int W>
__device__ __noinline__ void shortconv_bwd_again(const __nv_bfloat16* xb, const __nv_bfloat16* wc, const __nv_bfloat16* gb,
                                                 __nv_bfloat16* ob, float* pb, int t0, int t1, int T, int C) {
  for (int ch = 0; ch < 2; ++ch) {
    float acc[W + 1];
    for (int j = 0; j <= W; ++j) acc[j] = 0.f;
    for (int t = t1 - 1; t >= t0; --t) {
      const float xv = __bfloat162float(xb[(long long)t * C + ch]);
      float s[2] = {0.f, 0.f};
      for (int j = 0; j < W && t + j < T; ++j) {
        const float g = __bfloat162float(gb[(long long)(t + j) * C + ch]);
        s[j & 1] = fmaf(g, __bfloat162float(wc[ch * W + j]), s[j & 1]);
        acc[j] = fmaf(xv, g, acc[j]);
        if (j == 0) acc[W] += g;
      }
      ob[(long long)t * C + ch] = __float2bfloat16(s[0] + s[1]);
    }
    for (int j = 0; j <= W; ++j) pb[(long long)j * C + ch] = acc[j];
  }
}

// grid (ceil(B * spans / 4), ceil(C / 64)), block (32, 4)
template <int W>
__global__ void __launch_bounds__(128) shortconv_ring_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                                 const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ y,
                                                                 int B, int T, int C, int span, int spans) {
  const int c = blockIdx.y * 64 + 2 * threadIdx.x;
  const int unit = blockIdx.x * 4 + threadIdx.y;
  if (c >= C || unit >= B * spans) return;
  const int b = unit / spans, t0 = (unit % spans) * span, t1 = min(T, t0 + span);
  const __nv_bfloat16* xb = x + (long long)b * T * C + c;
  __nv_bfloat16* yb = y + (long long)b * T * C + c;
  uint64_t wf[W], win[W];
  shortconv_weights<W>(wf, w, c);
  const uint64_t b2 = bias ? pack_f32x2(__bfloat162float(bias[c]), __bfloat162float(bias[c + 1])) : 0ull;
#pragma unroll
  for (int j = 1; j < W; ++j) win[W - j] = pair_f32x2(ld_pair(xb, t0 - j, C, t0 - j >= 0));
  win[0] = 0ull;
  uint32_t nx[W];
#pragma unroll
  for (int r = 0; r < W; ++r) nx[r] = ld_pair(xb, t0 + r, C, t0 + r < t1);
  __nv_bfloat16* yt = yb + (long long)t0 * C;
  auto block = [&](auto edge, int t) {
    uint32_t cur[W];
#pragma unroll
    for (int r = 0; r < W; ++r) cur[r] = nx[r];
    ld_rows(nx, xb, t + W, C, 1, t + 2 * W <= t1, [&](int r) { return t + W + r < t1; });
#pragma unroll
    for (int r = 0; r < W; ++r) {
      win[r] = pair_f32x2(cur[r]);
      uint64_t s0 = b2, s1 = 0ull;
#pragma unroll
      for (int j = 0; j < W; j += 2) {
        if (!edge.value || j <= r) s0 = fma_f32x2(win[(r - j + W) % W], wf[j], s0);
        if (!edge.value || j + 1 <= r) s1 = fma_f32x2(win[(r - j - 1 + W) % W], wf[j + 1], s1);
      }
      float lo, hi;
      unpack_f32x2(add_f32x2(s0, s1), lo, hi);
      if (t + r < t1) *reinterpret_cast<uint32_t*>(yt) = pack_bf16(lo, hi);
      yt += C;
    }
  };
  int t = t0;
  if (t == 0) {
    block(std::true_type{}, 0);
    t = W;
  }
  for (; t < t1; t += W) block(std::false_type{}, t);
}

template <int W>
__global__ void __launch_bounds__(128) shortconv_ring_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                                 const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dx,
                                                                 float* __restrict__ part, int B, int T, int C, int span, int spans) {
  const int c = blockIdx.y * 64 + 2 * threadIdx.x;
  const int unit = blockIdx.x * 4 + threadIdx.y;
  if (c >= C || unit >= B * spans) return;
  const int b = unit / spans, t0 = (unit % spans) * span, t1 = min(T, t0 + span);
  const long long off = (long long)b * T * C + c;
  const __nv_bfloat16 *xb = x + off, *gb = dy + off;
  __nv_bfloat16* ob = dx + off;
  uint64_t wf[W], win[W], acc[W], accb = 0ull;
  shortconv_weights<W>(wf, w, c);
#pragma unroll
  for (int j = 0; j < W; ++j) acc[j] = 0ull;
  // step p of the walk is time t1 - 1 - p; slot r of the ring holds the step with p % W == r
#pragma unroll
  for (int j = 1; j < W; ++j) win[W - j] = pair_f32x2(ld_pair(gb, t1 - 1 + j, C, t1 - 1 + j < T));
  win[0] = 0ull;
  uint32_t ng[W], nx[W];
#pragma unroll
  for (int r = 0; r < W; ++r) {
    ng[r] = ld_pair(gb, t1 - 1 - r, C, t1 - 1 - r >= t0);
    nx[r] = ld_pair(xb, t1 - 1 - r, C, t1 - 1 - r >= t0);
  }
  for (int t = t1 - 1; t >= t0; t -= W) {
    uint32_t cg[W], cx[W];
#pragma unroll
    for (int r = 0; r < W; ++r) {
      cg[r] = ng[r];
      cx[r] = nx[r];
      ng[r] = ld_pair(gb, t - W - r, C, t - W - r >= t0);
      nx[r] = ld_pair(xb, t - W - r, C, t - W - r >= t0);
    }
#pragma unroll
    for (int r = 0; r < W; ++r) {
      win[r] = pair_f32x2(cg[r]);
      const uint64_t xv = pair_f32x2(cx[r]);            // zero before t0: those steps add nothing
      accb = add_f32x2(accb, win[r]);
      uint64_t s0 = 0ull, s1 = 0ull;
#pragma unroll
      for (int j = 0; j < W; j += 2) {
        const uint64_t g0 = win[(r - j + W) % W], g1 = win[(r - j - 1 + W) % W];
        s0 = fma_f32x2(g0, wf[j], s0);
        s1 = fma_f32x2(g1, wf[j + 1], s1);
        acc[j] = fma_f32x2(xv, g0, acc[j]);
        acc[j + 1] = fma_f32x2(xv, g1, acc[j + 1]);
      }
      float lo, hi;
      unpack_f32x2(add_f32x2(s0, s1), lo, hi);
      if (t - r >= t0) *reinterpret_cast<uint32_t*>(ob + (long long)(t - r) * C) = pack_bf16(lo, hi);
    }
  }
  float* pb = part + (long long)unit * (W + 1) * C + c;
#pragma unroll
  for (int j = 0; j <= W; ++j) {
    float lo, hi;
    unpack_f32x2(j < W ? acc[j < W ? j : 0] : accb, lo, hi);
    *reinterpret_cast<float2*>(pb + (long long)j * C) = make_float2(lo, hi);
  }
  if (t1 + W - 1 > T && (not_finite_f32x2(acc[0]) || not_finite_f32x2(accb) || shortconv_weights_bad<W>(wf)))
    shortconv_bwd_again<W>(xb, w + (long long)c * W, gb, ob, pb, t0, t1, T, C);
}

// A gradient in the type it is wanted in: fp32 sums, rounded once (as two casts behind the kernel would, without their launches)
__device__ __forceinline__ void put_grad(float* p, float v) { *p = v; }
__device__ __forceinline__ void put_grad(__nv_bfloat16* p, float v) { *p = __float2bfloat16(v); }

// dw[c, j] = sum over the slices of part[slice][j][c], db[c] from row `taps`. grid (ceil(C / 32), taps + 1), block (32, 16)
template <typename G>
__global__ void __launch_bounds__(512) shortconv_sum_kernel(const float* __restrict__ part, G* __restrict__ dw, G* __restrict__ db,
                                                            int slices, int C, int taps) {
  __shared__ float red[16][33];
  const int c = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y;
  float s = 0.f;
  if (c < C) {
#pragma unroll 4
    for (int i = threadIdx.y; i < slices; i += 16) s += part[((long long)i * (taps + 1) + j) * C + c];
  }
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < C) {
    float tot = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) tot += red[k][threadIdx.x];
    if (j < taps) put_grad(dw + (long long)c * taps + j, tot);
    else if (db) put_grad(db + c, tot);
  }
}

// ShortConv of T new positions behind the last `tail` ones of a stream, which the layer keeps: u[b, t] from the tail and the new inputs, and tail and
// inputs side by side as the next tail's source, in one launch, for short blocks (see shortconv_stream_long). RING: the order of the sums of the
// register-ring kernels (even and odd taps apart), otherwise that of the general one, so that the bits do not depend on how a sequence is cut.
// A block is 64 channel pairs of one position. grid (B * T, ceil(C / 128))
template <bool RING>
__global__ void __launch_bounds__(64) shortconv_stream_kernel(const __nv_bfloat16* __restrict__ tail, long long tail_stride,
                                                              const __nv_bfloat16* __restrict__ n, const __nv_bfloat16* __restrict__ w,
                                                              const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ xin,
                                                              __nv_bfloat16* __restrict__ u, int tails, int T, int C, int W) {
  const int c = (blockIdx.y * 64 + threadIdx.x) * 2, t = blockIdx.x % T, b = blockIdx.x / T;
  if (c >= C) return;
  const __nv_bfloat16 *tb = tail + b * tail_stride + c, *nb = n + (long long)b * T * C + c;
  shortconv_stream_pair<RING>([&](int i) {                             // position i of tail and inputs
    return *reinterpret_cast<const uint32_t*>(i < tails ? tb + (long long)i * C : nb + (long long)(i - tails) * C);
  }, w, bias, xin + (long long)b * (tails + T) * C + c, u + ((long long)b * T + t) * C + c, tails, t, c, C, W);
}

// ---- any other window of up to 128 taps, 16 taps and 16 time steps at a time, a channel pair per lane: the 31 inputs that such a block meets wait in
// registers (a ring of 32 slots, unrolled twice, so that their names are fixed), the 16 that the next one adds are under way meanwhile, and 256 packed
// multiply-adds work on 16 independent sums.
// B 8, T 2048, C 1024, W 64 (1.07 G multiply-adds each: 30 us at the chip's fp32 rate): output 72 us, input gradient 69,
// weight gradient 77 + 10 for the joint; one tap of one position at a time they took 268, 270 and 1047. The multiply-adds are 45 % of the instructions (the
// others load, unpack and go round), half of the issue slots are taken. W 32 139 for 865 us in all, W 5 81 for 402, W 128 402 for 2927; 2 x 1655 x 256,
// W 64: 29 for 96. Loads with a test and a 64-bit multiplication each, and weights stored 32 lanes to a bank, cost half as much again (342 us at W 64).
constexpr int SC_TILE = 16;
constexpr int SC_WARPS = 8;
constexpr int SC_WLD = 66;                               // floats of a tap's 64 weights: channel by channel stores meet two to a bank

// One output of the block kernel below as it is meant, for weights that are not finite: no product with what lies outside the sequence.
template <bool DX>
__device__ __noinline__ void shortconv_rows(const __nv_bfloat16* ib, const __nv_bfloat16* wc, uint64_t b2, __nv_bfloat16* ob, int s0, int T, int C, int W) {
  for (int s = s0; s < min(T, s0 + SC_TILE); ++s) {
    float a0, a1;
    unpack_f32x2(b2, a0, a1);
    for (int j = 0; j < min(W, s + 1); ++j) {
      const uint32_t v = ld_pair(ib, DX ? T - 1 - s + j : s - j, C, true);
      a0 = fmaf(bf16_lo(v), __bfloat162float(wc[j]), a0);
      a1 = fmaf(bf16_hi(v), __bfloat162float(wc[W + j]), a1);
    }
    *reinterpret_cast<uint32_t*>(ob + (long long)(DX ? T - 1 - s : s) * C) = pack_bf16(a0, a1);
  }
}

// Sequences of up to N steps (2, or SC_FEW), 16 / N of them in flight, forward and input gradient: step s is time s or T - 1 - s, all of a sequence's
// outputs from its registers, and no other products than those of the sums, which run over j in order as below. A warp takes sequence after sequence, its
// weights in registers; bound by memory (4096 sequences of two steps, 1024 channels, W 5: 34 MB in 8.3 us). A block of 16 taps by 16 steps is made whatever
// the sequence fills of it. us, output / all gradients, in such blocks -> so: W 5, 4096 x 2 x 1024 92 / 361 -> 8 / 25, 1024 x 4 x 1024 27 / 79 -> 8 / 23,
// 512 x 8 x 1024 16.5 / 45 -> 8 / 21; W 64 298 / 1143 -> 12 / 52, 80 / 361 -> 17 / 50, 43 / 189 -> 21 / 49. (From nine steps on the blocks: 512 x 9 x 1024,
// W 5, 16.5 / 46.) grid (any, ceil(C / 64)), block (32, SC_WARPS)
constexpr int SC_FEW = 8;
template <bool DX, int N>
__global__ void __launch_bounds__(32 * SC_WARPS) shortconv_few_kernel(const __nv_bfloat16* __restrict__ in, const __nv_bfloat16* __restrict__ w,
                                                                      const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ out, int B, int T,
                                                                      int C, int W) {
  const int c = blockIdx.y * 64 + 2 * threadIdx.x, taps = min(W, T);
  if (c >= C) return;
  uint64_t wv[N];
#pragma unroll
  for (int j = 0; j < N; ++j)
    wv[j] = j < taps ? pack_f32x2(__bfloat162float(w[(long long)c * W + j]), __bfloat162float(w[(long long)(c + 1) * W + j])) : 0ull;
  const uint64_t b2 = !DX && bias ? pack_f32x2(__bfloat162float(bias[c]), __bfloat162float(bias[c + 1])) : 0ull;
#pragma unroll (16 / N)
  for (int b = blockIdx.x * SC_WARPS + threadIdx.y; b < B; b += gridDim.x * SC_WARPS) {
    const __nv_bfloat16* ib = in + (long long)b * T * C + c;
    __nv_bfloat16* ob = out + (long long)b * T * C + c;
    uint32_t q[N];
#pragma unroll
    for (int s = 0; s < N; ++s) q[s] = ld_pair(ib, DX ? T - 1 - s : s, C, s < T);
#pragma unroll
    for (int s = 0; s < N; ++s)
      if (s < T) {
        uint64_t a = b2;
#pragma unroll
        for (int j = 0; j <= s; ++j)
          if (j < taps) a = fma_f32x2(pair_f32x2(q[s - j]), wv[j], a);
        float lo, hi;
        unpack_f32x2(a, lo, hi);
        *reinterpret_cast<uint32_t*>(ob + (long long)(DX ? T - 1 - s : s) * C) = pack_bf16(lo, hi);
      }
  }
}
// and the weight gradient, as shortconv_dw_kernel leaves it. grid (ceil(slices / 4), ceil(C / 64)), block (32, 4)
template <int N>
__global__ void __launch_bounds__(128) shortconv_few_dw_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                                                               float* __restrict__ part, int B, int T, int C, int W, int seqs, int slices) {
  const int c = blockIdx.y * 64 + 2 * threadIdx.x, unit = blockIdx.x * 4 + threadIdx.y;
  if (c >= C || unit >= slices) return;
  uint64_t acc[N], accb = 0ull;
#pragma unroll
  for (int j = 0; j < N; ++j) acc[j] = 0ull;
  const int b1 = min(B, (unit + 1) * seqs);
#pragma unroll (16 / N)
  for (int b = unit * seqs; b < b1; ++b) {
    const __nv_bfloat16 *xb = x + (long long)b * T * C + c, *gb = dy + (long long)b * T * C + c;
    uint32_t xq[N], gq[N];
#pragma unroll
    for (int t = 0; t < N; ++t) {
      xq[t] = ld_pair(xb, t, C, t < T);
      gq[t] = ld_pair(gb, t, C, t < T);
    }
#pragma unroll
    for (int t = 0; t < N; ++t)
      if (t < T) {
        const uint64_t g = pair_f32x2(gq[t]);
        accb = add_f32x2(accb, g);
#pragma unroll
        for (int j = 0; j <= t; ++j) acc[j] = fma_f32x2(pair_f32x2(xq[t - j]), g, acc[j]);
      }
  }
  float* pb = part + (long long)unit * (W + 1) * C + c;
  auto put = [&](int j, uint64_t v) {
    float lo, hi;
    unpack_f32x2(v, lo, hi);
    *reinterpret_cast<float2*>(pb + (long long)j * C) = make_float2(lo, hi);
  };
#pragma unroll
  for (int j = 0; j < N; ++j)
    if (j < W) put(j, acc[j]);
  for (int j = N; j < W; ++j) put(j, 0ull);
  put(W, accb);
}

// Forward (y[t] = bias + sum_j x[t - j] w[j]) and, walked from late to early, the input gradient (dx[t] = sum_j dy[t + j] w[j]); step s is time s or
// T - 1 - s. The sum of an output runs over j in order, as in shortconv_stream_kernel. What lies outside the sequence is zero, which finite weights leave
// so. taps: those that a sequence meets, min(W, T). grid (ceil(B * tiles / SC_WARPS), ceil(C / 64)), block (32, SC_WARPS), dynamic shared memory: the
// weights, taps by SC_WLD floats.
template <bool DX>
__global__ void __launch_bounds__(32 * SC_WARPS, 2) shortconv_tile_kernel(const __nv_bfloat16* __restrict__ in, const __nv_bfloat16* __restrict__ w,
                                                                          const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ out,
                                                                          int B, int T, int C, int W, int taps, int tiles) {
  extern __shared__ __align__(16) float sw[];
  const int lane = threadIdx.x, warp = threadIdx.y, c0 = blockIdx.y * 64;
  float z = 0.f;
  for (int j = lane; j < taps; j += 32) {                   // consecutive lanes read consecutive weights of a channel
#pragma unroll
    for (int i = 0; i < 64 / SC_WARPS; ++i) {
      const int cl = warp + i * SC_WARPS;
      const float f = c0 + cl < C ? __bfloat162float(w[(long long)(c0 + cl) * W + j]) : 0.f;
      sw[j * SC_WLD + cl] = f;
      z = fmaf(f, 0.f, z);
    }
  }
  const bool bad = __syncthreads_or(z != 0.f);
  const int c = c0 + 2 * lane;
  const long long unit = (long long)blockIdx.x * SC_WARPS + warp;
  if (c >= C || unit >= (long long)B * tiles) return;
  const long long off = unit / tiles * T * C + c;
  const int s0 = (int)(unit % tiles) * SC_TILE;
  const __nv_bfloat16* ib = in + off;
  __nv_bfloat16* ob = out + off;
  const uint64_t b2 = !DX && bias ? pack_f32x2(__bfloat162float(bias[c]), __bfloat162float(bias[c + 1])) : 0ull;
  if (bad) {
    shortconv_rows<DX>(ib, w + (long long)c * W, b2, ob, s0, T, C, W);
    return;
  }
  // steps s, s - 1, ..., s - 15
  auto get = [&](uint32_t (&q)[SC_TILE], int s) {
    ld_rows(q, ib, DX ? T - 1 - s : s, C, DX ? 1 : -1, s < T && s >= SC_TILE - 1, [&](int i) { return s - i < T && s - i >= 0; });
  };
  uint64_t win[2 * SC_TILE], acc[SC_TILE];               // step s0 + p is in slot p mod 32
  {
    uint32_t q[2][SC_TILE];
    get(q[0], s0 + SC_TILE - 1);
    get(q[1], s0 - 1);
#pragma unroll
    for (int i = 0; i < SC_TILE; ++i) {
      win[SC_TILE - 1 - i] = pair_f32x2(q[0][i]);
      win[2 * SC_TILE - 1 - i] = pair_f32x2(q[1][i]);
    }
  }
#pragma unroll
  for (int r = 0; r < SC_TILE; ++r) acc[r] = b2;
  auto block = [&](auto half, auto whole, int j0) {
    constexpr int H = decltype(half)::value * SC_TILE;
    uint32_t nx[SC_TILE];
    if (j0 + SC_TILE < taps) {
      get(nx, s0 - j0 - SC_TILE);
    } else {
#pragma unroll
      for (int i = 0; i < SC_TILE; ++i) nx[i] = 0u;
    }
#pragma unroll
    for (int jj = 0; jj < SC_TILE; ++jj) {
      if (!whole.value && j0 + jj >= taps) break;        // an input that is not finite would make NaN of a tap of zero
      const uint64_t wv = *reinterpret_cast<const uint64_t*>(sw + (j0 + jj) * SC_WLD + 2 * lane);
#pragma unroll
      for (int r = 0; r < SC_TILE; ++r) acc[r] = fma_f32x2(win[(r - jj - H) & 31], wv, acc[r]);
    }
#pragma unroll
    for (int i = 0; i < SC_TILE; ++i) win[(-H - SC_TILE - i) & 31] = pair_f32x2(nx[i]);
  };
  using Even = std::integral_constant<int, 0>;
  using Odd = std::integral_constant<int, 1>;
  const int full = taps / (2 * SC_TILE) * (2 * SC_TILE);
  for (int j0 = 0; j0 < full; j0 += 2 * SC_TILE) {
    block(Even{}, std::true_type{}, j0);
    block(Odd{}, std::true_type{}, j0 + SC_TILE);
  }
  if (full < taps) block(Even{}, std::false_type{}, full);
  if (full + SC_TILE < taps) block(Odd{}, std::false_type{}, full + SC_TILE);
  __nv_bfloat16* o = ob + (long long)(DX ? T - 1 - s0 : s0) * C;
  const long long step = DX ? -(long long)C : C;
#pragma unroll
  for (int r = 0; r < SC_TILE; ++r, o += step) {
    float lo, hi;
    unpack_f32x2(acc[r], lo, hi);
    if (s0 + r < T) *reinterpret_cast<uint32_t*>(o) = pack_bf16(lo, hi);
  }
}

// The sums of 16 taps over a span of one sequence as they are meant, where those of shortconv_dw_kernel came out not finite: zeros stand in there for
// what lies outside the span and the sequence.
__device__ __noinline__ void shortconv_dw_again(const __nv_bfloat16* x, const __nv_bfloat16* dy, float* pb, int b0, int b1, int t0, int t1, int T, int C, int W,
                                                int j0) {
  for (int ch = 0; ch < 2; ++ch)
    for (int j = j0; j < min(W, j0 + SC_TILE); ++j) {
      float s = 0.f;
      for (int b = b0; b < b1; ++b)
        for (int t = max(t0, j); t < t1; ++t)
          s = fmaf(__bfloat162float(x[((long long)b * T + t - j) * C + ch]), __bfloat162float(dy[((long long)b * T + t) * C + ch]), s);
      pb[(long long)j * C + ch] = s;
    }
}

// part[slice][j][c] = sum over the slice's steps of dy[t, c] x[t - j, c], part[slice][W][c] that of dy. A warp takes 64 channels, 16 taps and a slice: a span of
// one sequence, or with many sequences all of `seqs`. grid (ceil(slices / 4), ceil(C / 64), ceil(W / 16)), block (32, 4)
__global__ void __launch_bounds__(128, 3) shortconv_dw_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                                                              float* __restrict__ part, int B, int T, int C, int W, int span, int spans, int seqs, int slices) {
  const int c = blockIdx.y * 64 + 2 * threadIdx.x, j0 = blockIdx.z * SC_TILE, unit = blockIdx.x * 4 + threadIdx.y;
  if (c >= C || unit >= slices) return;
  const int b0 = unit / spans * seqs, b1 = min(B, b0 + seqs), t0 = unit % spans * span, t1 = min(T, t0 + span);
  uint64_t acc[SC_TILE], accb = 0ull;
#pragma unroll
  for (int j = 0; j < SC_TILE; ++j) acc[j] = 0ull;
  for (int b = j0 < T ? b0 : b1; b < b1; ++b) {          // (taps longer than the sequence: zero)
    const __nv_bfloat16 *xb = x + (long long)b * T * C + c, *gb = dy + (long long)b * T * C + c;
    uint64_t win[2 * SC_TILE];                           // input t0 - j0 + p is in slot p mod 32
    uint32_t nx[SC_TILE], ng[SC_TILE];
    auto get_x = [&](int t) {
      ld_rows(nx, xb, t - j0, C, 1, t >= j0 && t + SC_TILE <= t1, [&](int r) { return t - j0 + r >= 0 && t + r < t1; });
    };
    auto get_g = [&](int t) { ld_rows(ng, gb, t, C, 1, t + SC_TILE <= t1, [&](int r) { return t + r < t1; }); };
    get_x(t0 - SC_TILE);
#pragma unroll
    for (int r = 0; r < SC_TILE; ++r) win[SC_TILE + r] = pair_f32x2(nx[r]);
    get_x(t0);
    get_g(t0);
    auto block = [&](auto half, int t) {
      constexpr int H = decltype(half)::value * SC_TILE;
      uint32_t cg[SC_TILE];
#pragma unroll
      for (int r = 0; r < SC_TILE; ++r) {
        win[r + H] = pair_f32x2(nx[r]);
        cg[r] = ng[r];
      }
      get_x(t + SC_TILE);
      get_g(t + SC_TILE);
#pragma unroll
      for (int r = 0; r < SC_TILE; ++r) {
        const uint64_t g = pair_f32x2(cg[r]);
        accb = add_f32x2(accb, g);
#pragma unroll
        for (int j = 0; j < SC_TILE; ++j) acc[j] = fma_f32x2(win[(r - j + H) & 31], g, acc[j]);
      }
    };
    for (int t = t0; t < t1; t += 2 * SC_TILE) {
      block(std::integral_constant<int, 0>{}, t);
      if (t + SC_TILE < t1) block(std::integral_constant<int, 1>{}, t + SC_TILE);
    }
  }
  float* pb = part + (long long)unit * (W + 1) * C + c;
  uint64_t z = 0ull;
#pragma unroll
  for (int j = 0; j < SC_TILE; ++j) {
    float lo, hi;
    unpack_f32x2(acc[j], lo, hi);
    if (j0 + j < W) *reinterpret_cast<float2*>(pb + (long long)(j0 + j) * C) = make_float2(lo, hi);
    z = fma_f32x2(acc[j], 0ull, z);
  }
  if (j0 == 0) {
    float lo, hi;
    unpack_f32x2(accb, lo, hi);
    *reinterpret_cast<float2*>(pb + (long long)W * C) = make_float2(lo, hi);
  }
  if (not_finite_f32x2(z)) shortconv_dw_again(x + c, dy + c, pb, b0, b1, t0, t1, T, C, W, j0);
}

template <bool DX>
int launch_shortconv_tile(const __nv_bfloat16* in, const __nv_bfloat16* w, const __nv_bfloat16* bias, __nv_bfloat16* out, int B, int T, int C, int W,
                          cudaStream_t s) {
  const int tiles = (T + SC_TILE - 1) / SC_TILE, taps = std::min(W, T);
  if (T <= SC_FEW) {
    const long long groups = (C + 63) / 64, all = ((long long)B + SC_WARPS - 1) / SC_WARPS, room = std::max(1ll, 148 * 8 / groups);
    const dim3 g((unsigned)std::min(all, room), (unsigned)groups), blk(32, SC_WARPS);
    if (T <= 2) shortconv_few_kernel<DX, 2><<<g, blk, 0, s>>>(in, w, bias, out, B, T, C, W);
    else shortconv_few_kernel<DX, SC_FEW><<<g, blk, 0, s>>>(in, w, bias, out, B, T, C, W);
    ELFA_CUDA(cudaGetLastError());
    ::elfa::count_launches(1);
    return ELFA_OK;
  }
  const dim3 grid((unsigned)(((long long)B * tiles + SC_WARPS - 1) / SC_WARPS), (C + 63) / 64), block(32, SC_WARPS);
  shortconv_tile_kernel<DX><<<grid, block, (size_t)taps * SC_WLD * sizeof(float), s>>>(in, w, bias, out, B, T, C, W, taps, tiles);
  ELFA_CUDA(cudaGetLastError());
  ::elfa::count_launches(1);
  return ELFA_OK;
}

// The slices of shortconv_dw_kernel: no sum longer than SC_CHAIN steps (its error grows with its length: in one wave of warps, up to 2048 steps, it was twice
// that of sums of 512), in whole waves of its warps (12 of them per SM). The scratch that this takes: a slice per 256 steps or more, (W + 1) C floats each:
// 21 MB at B 8, T 2048, C 1024, W 64, 34 MB at W 128; of long inputs as many bytes as x has at W 127, half of them at W 63.
constexpr int SC_CHAIN = 256;
struct ShortConvSlices {
  int span, spans, seqs, slices;
};
ShortConvSlices shortconv_slices(int B, int T, int C, int W) {
  const long long per = (long long)((C + 63) / 64) * ((W + SC_TILE - 1) / SC_TILE), wave = 12ll * 148;        // warps of a slice; of the chip
  const long long least = ((long long)B * T + SC_CHAIN - 1) / SC_CHAIN, want = std::max(1ll, (least * per + wave - 1) / wave * wave / per);
  const int tiles = (T + SC_TILE - 1) / SC_TILE, cut = (int)std::min<long long>(tiles, std::max<long long>((T + SC_CHAIN - 1) / SC_CHAIN, want / B));
  ShortConvSlices q;
  q.span = (tiles + cut - 1) / cut * SC_TILE;
  q.spans = (T + q.span - 1) / q.span;
  q.seqs = (int)std::min(std::max(1ll, (B + want - 1) / want), (long long)std::max(1, SC_CHAIN / T));
  q.slices = (B + q.seqs - 1) / q.seqs * q.spans;
  return q;
}

template <int D>
int launch_efla_fwd(const void* k, const void* v, const float* beta, const float* state0, void* o, float* state_out, int B,
                    int T, int H, cudaStream_t s) {
  efla_scan_fwd_kernel<D><<<dim3(B * H, D / 32), 32 * EFLA_W, 0, s>>>(static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v), beta, state0,
                                              static_cast<__nv_bfloat16*>(o), state_out, T, H);
  ELFA_CUDA(cudaGetLastError());
  ::elfa::count_launches(1);
  return ELFA_OK;
}

}  // namespace
}  // namespace elfa

using namespace elfa;

// k, v, o: [B, T, H, d] bf16; beta: 1 float; state0 (optional) / state_out: [B, H, d, d] fp32.
ELFA_API int elfa_efla_scan_fwd(const void* k, const void* v, const float* beta, const float* state0, void* o, float* state_out,
                                int B, int T, int H, int d, void* stream) {
  ELFA_REQUIRE(k && v && beta && o && B > 0 && T > 0 && H > 0, "efla_scan_fwd: bad arguments");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (d) {
    case 32: return launch_efla_fwd<32>(k, v, beta, state0, o, state_out, B, T, H, s);
    case 64: return launch_efla_fwd<64>(k, v, beta, state0, o, state_out, B, T, H, s);
    case 96: return launch_efla_fwd<96>(k, v, beta, state0, o, state_out, B, T, H, s);
    case 128: return launch_efla_fwd<128>(k, v, beta, state0, o, state_out, B, T, H, s);
    default: set_last_error("efla_scan_fwd: head dimension must be 32, 64, 96 or 128"); return ELFA_ERR_UNSUPPORTED;
  }
}

// Time steps a warp of the register-ring kernels walks: long spans amortise the seam, short ones keep the SMs busy on small inputs.
static int shortconv_span(int B, int T, int C) {
  const long long warps64 = (long long)B * ((T + 63) / 64) * ((C + 63) / 64);
  return warps64 >= 148 * 8 ? 64 : (warps64 >= 148 * 4 ? 32 : 16);
}
static bool shortconv_ring(int W) { return W == 4 || W == 8 || W == 16; }

// Slices of the weight-gradient scratch of elfa_shortconv_bwd_as (slices * (W + 1) * C floats).
ELFA_API int elfa_shortconv_bwd_slices(int B, int T, int C, int W) {
  if (B <= 0 || T <= 0 || C <= 0 || W <= 0) return 0;
  if (!shortconv_ring(W)) return shortconv_slices(B, T, C, W).slices;
  const int span = shortconv_span(B, T, C);
  return B * ((T + span - 1) / span);
}

ELFA_API int elfa_shortconv_fwd(const void* x, const void* w, const void* bias, void* y, int B, int T, int C, int W, void* stream) {
  ELFA_REQUIRE(x && w && y && B > 0 && T > 0 && C > 0 && W > 0, "shortconv_fwd: bad arguments");
  ELFA_REQUIRE(C % 2 == 0 && W <= 128, "shortconv_fwd: the channel count must be even and the window at most 128");
  if (shortconv_ring(W)) {
    const auto *X = static_cast<const __nv_bfloat16*>(x), *Wt = static_cast<const __nv_bfloat16*>(w), *Bi = static_cast<const __nv_bfloat16*>(bias);
    auto* Y = static_cast<__nv_bfloat16*>(y);
    // four taps: the seam is three rows, and more warps keep more loads in flight (B 4, T 4096, C 512: 20 -> 16 us, B 2, T 1531, C 1024: 12 -> 10)
    const int span = W == 4 ? 16 : shortconv_span(B, T, C), spans = (T + span - 1) / span;
    const dim3 g((unsigned)(((long long)B * spans + 3) / 4), (C + 63) / 64), blk(32, 4);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (W == 4) shortconv_ring_fwd_kernel<4><<<g, blk, 0, s>>>(X, Wt, Bi, Y, B, T, C, span, spans);
    else if (W == 8) shortconv_ring_fwd_kernel<8><<<g, blk, 0, s>>>(X, Wt, Bi, Y, B, T, C, span, spans);
    else shortconv_ring_fwd_kernel<16><<<g, blk, 0, s>>>(X, Wt, Bi, Y, B, T, C, span, spans);
    ELFA_CUDA(cudaGetLastError());
    ::elfa::count_launches(1);
    return ELFA_OK;
  }
  return launch_shortconv_tile<false>(static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), static_cast<const __nv_bfloat16*>(bias),
                                      static_cast<__nv_bfloat16*>(y), B, T, C, W, static_cast<cudaStream_t>(stream));
}

// Whether T positions behind a tail are long enough for the ordinary kernels: tail and inputs are copied side by side, the outputs of the tail's own
// positions are made and dropped, with several sequences the others are copied together. The one kernel reads 2 W weights per channel pair and
// position straight from [C, W], where every lane touches another line: long blocks cost it 5 (W 4), 9 (8), 30 (16), 24 (24), 114 (32) and 226 (64)
// microseconds per 10^6 values. Measured, one kernel / ordinary ones, microseconds: W 4, 1 sequence 2^20 values 6.9 / 6.5, 2^22 21 / 10, 4 sequences
// 2^22 21 / 26; W 8 2^20 11 / 7 and 11 / 11; W 16 2^17 6.6 / 6.4 and 6.6 / 8.2, 2^18 10.6 / 6.5 and 10.6 / 8.4, 2^22 125 / 13; W 24 2^18 10 / 12,
// 2^19 19 / 12 and 19 / 18; W 32 2^16 13 / 12 and 14 / 17, 2^17 21 / 12 and 21 / 17; W 48 2^17 17 / 13 and 17 / 19;
// W 64 2^15 17 / 14 and 19 / 22, 2^16 23 / 15 and 25 / 22, 2^20 245 / 17; W 100 2^16 23 / 17 and 23 / 23; W 128 2^16 41 / 20 and 41 / 25.
static bool shortconv_stream_long(int B, int T, int C, int W) {
  const long long values = (long long)B * T * C;
  if (W < 8) return B == 1 && values >= 1 << 21;
  if (W < 16) return values >= 1 << 20;
  return values >= 1 << (W == 16 ? 18 : (W < 32 ? 19 : (W < 64 ? 17 : 16)));
}

// `bytes` of each of B batches. One copy of rows wants them apart and a pitch below 2^31 bytes (a block of a million positions of 1024 values is
// past it); one tail shared by several sequences, and longer blocks, go one by one.
static cudaError_t copy_batches(void* dst, size_t dpitch, const void* src, size_t spitch, size_t bytes, int B, cudaStream_t s) {
  if (B > 1 && spitch >= bytes && dpitch < (1ull << 31) && spitch < (1ull << 31))
    return cudaMemcpy2DAsync(dst, dpitch, src, spitch, bytes, B, cudaMemcpyDeviceToDevice, s);
  for (int b = 0; b < B; ++b) {
    const cudaError_t e = cudaMemcpyAsync(static_cast<unsigned char*>(dst) + b * dpitch, static_cast<const unsigned char*>(src) + b * spitch, bytes,
                                          cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Positions of scratch (C values each) of elfa_shortconv_stream: all of tail and inputs in the long form, otherwise none.
ELFA_API int elfa_shortconv_stream_rows(int B, int tails, int T, int C, int W) {
  return B > 0 && tails > 0 && T > 0 && C > 0 && W > 0 && shortconv_stream_long(B, T, C, W) ? B * (tails + T) : 0;
}

// tail [B, tails, C] (batches tail_stride elements apart), n [B, T, C] -> u [B, T, C] = ShortConv of tail and n side by side, its last T positions,
// and xin [B, tails + T, C], the two side by side. full: scratch of elfa_shortconv_stream_rows() positions (null when 0); with one sequence u may
// be full + tails * C, where the long form leaves it anyway.
ELFA_API int elfa_shortconv_stream(const void* tail, long long tail_stride, const void* n, const void* w, const void* bias, void* xin, void* u,
                                   void* full, int B, int tails, int T, int C, int W, void* stream) {
  ELFA_REQUIRE(tail && n && w && xin && u && B > 0 && tails > 0 && T > 0 && (long long)B * (tails + (long long)T) < (1ll << 31) && C > 0 && W > 0,
               "shortconv_stream: bad arguments");
  ELFA_REQUIRE(C % 2 == 0 && tail_stride % 2 == 0 && W <= 128, "shortconv_stream: channels and batch stride must be even, the window at most 128");
  for (const void* q : {tail, n, static_cast<const void*>(xin), static_cast<const void*>(u), static_cast<const void*>(full)})
    ELFA_REQUIRE((reinterpret_cast<uintptr_t>(q) & 3) == 0, "shortconv_stream: operands must be 4-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (shortconv_stream_long(B, T, C, W)) {
    ELFA_REQUIRE(full, "shortconv_stream: this length needs the scratch buffer");
    const size_t row = (size_t)C * 2, all = (size_t)(tails + T) * row;
    auto* x = static_cast<unsigned char*>(xin);
    const auto* f = static_cast<const unsigned char*>(full) + tails * row;
    ELFA_CUDA(copy_batches(x, all, tail, (size_t)tail_stride * 2, tails * row, B, s));
    ELFA_CUDA(copy_batches(x + tails * row, all, n, T * row, T * row, B, s));
    const int rc = elfa_shortconv_fwd(xin, w, bias, full, B, tails + T, C, W, stream);
    if (rc == ELFA_OK && u != f) ELFA_CUDA(copy_batches(u, T * row, f, all, T * row, B, s));
    return rc;
  }
  auto kernel = shortconv_ring(W) ? shortconv_stream_kernel<true> : shortconv_stream_kernel<false>;
  const auto h = [](const void* p) { return static_cast<const __nv_bfloat16*>(p); };
  kernel<<<dim3((unsigned)(B * T), (C + 127) / 128), 64, 0, s>>>(h(tail), tail_stride, h(n), h(w), h(bias), static_cast<__nv_bfloat16*>(xin),
                                                               static_cast<__nv_bfloat16*>(u), tails, T, C, W);
  ELFA_CUDA(cudaGetLastError());
  ::elfa::count_launches(1);
  return ELFA_OK;
}

// dx bf16 [B,T,C]; dw [C,W] and db [C] (or null) in fp32, or in bf16 where `grads_bf16`; part: scratch of
// elfa_shortconv_bwd_slices() * (W + 1) * C floats.
ELFA_API int elfa_shortconv_bwd_as(const void* x, const void* w, const void* dy, void* dx, void* dw_, void* db_, float* part, int grads_bf16,
                                   int B, int T, int C, int W, void* stream) {
  float *dw = static_cast<float*>(dw_), *db = static_cast<float*>(db_);
  ELFA_REQUIRE(x && w && dy && dx && dw && B > 0 && T > 0 && C > 0 && W > 0, "shortconv_bwd: bad arguments");
  ELFA_REQUIRE(C % 2 == 0 && W <= 128, "shortconv_bwd: the channel count must be even and the window at most 128");
  ELFA_REQUIRE(part, "shortconv_bwd: the scratch buffer is missing");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const auto *X = static_cast<const __nv_bfloat16*>(x), *Wt = static_cast<const __nv_bfloat16*>(w), *G = static_cast<const __nv_bfloat16*>(dy);
  auto* DX = static_cast<__nv_bfloat16*>(dx);
  int slices;
  if (shortconv_ring(W)) {
    const int span = shortconv_span(B, T, C), spans = (T + span - 1) / span;
    const dim3 g((unsigned)(((long long)B * spans + 3) / 4), (C + 63) / 64), blk(32, 4);
    if (W == 4) shortconv_ring_bwd_kernel<4><<<g, blk, 0, s>>>(X, Wt, G, DX, part, B, T, C, span, spans);
    else if (W == 8) shortconv_ring_bwd_kernel<8><<<g, blk, 0, s>>>(X, Wt, G, DX, part, B, T, C, span, spans);
    else shortconv_ring_bwd_kernel<16><<<g, blk, 0, s>>>(X, Wt, G, DX, part, B, T, C, span, spans);
    slices = B * spans;
  } else {
    const int rc = launch_shortconv_tile<true>(G, Wt, nullptr, DX, B, T, C, W, s);
    if (rc != ELFA_OK) return rc;
    const ShortConvSlices q = shortconv_slices(B, T, C, W);
    const dim3 few((q.slices + 3) / 4, (C + 63) / 64);
    if (T <= 2)
      shortconv_few_dw_kernel<2><<<few, dim3(32, 4), 0, s>>>(X, G, part, B, T, C, W, q.seqs, q.slices);
    else if (T <= SC_FEW)
      shortconv_few_dw_kernel<SC_FEW><<<few, dim3(32, 4), 0, s>>>(X, G, part, B, T, C, W, q.seqs, q.slices);
    else
      shortconv_dw_kernel<<<dim3((q.slices + 3) / 4, (C + 63) / 64, (W + SC_TILE - 1) / SC_TILE), dim3(32, 4), 0, s>>>(X, G, part, B, T, C, W, q.span, q.spans,
                                                                                                                    q.seqs, q.slices);
    slices = q.slices;
  }
  ELFA_CUDA(cudaGetLastError());
  const dim3 gs((C + 31) / 32, W + 1), bs(32, 16);
  if (grads_bf16) shortconv_sum_kernel<<<gs, bs, 0, s>>>(part, static_cast<__nv_bfloat16*>(dw_), static_cast<__nv_bfloat16*>(db_), slices, C, W);
  else shortconv_sum_kernel<<<gs, bs, 0, s>>>(part, dw, db, slices, C, W);
  ELFA_CUDA(cudaGetLastError());
  ::elfa::count_launches(2);
  return ELFA_OK;
}
