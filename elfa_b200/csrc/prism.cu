// PRISM iterative refinement, forward and backward, one kernel each.
//
// reference: src/model/prism.zig:318-421 (host loops over tokens, groups and iterations) and
// :488-871 (backward); kernels/cuda/include/kernels.h declares prism_forward_cuda but no source defines it.
//
//   r_0 = v - u                                   per group g of d channels
//   delta_l = gelu(p_l * r_l),  r_{l+1} = r_l - delta_l,  l = 0 .. L-1      (p_l [B,T,d] is shared by all groups)
//   y = u + sum_l delta_l
//
// One thread owns one (token, channel-in-group) pair and walks over the G groups, so the gradient of
// p_l (a sum over groups) is accumulated in registers: no atomics, deterministic. Consecutive
// threads touch consecutive channels: every access is coalesced. The backward recomputes r_l.
#include <algorithm>

#include "elfa_native.h"
#include "prism_step.cuh"

namespace elfa {
namespace {

struct PrismPtrs {
  const __nv_bfloat16* p[PRISM_MAX_L];   // [tokens, d] each
  float* dp[PRISM_MAX_L];                // [tokens, d] fp32 each (backward)
};

__global__ void __launch_bounds__(256) prism_fwd_kernel(const __nv_bfloat16* __restrict__ u, const __nv_bfloat16* __restrict__ v,
                                                        PrismPtrs pp, __nv_bfloat16* __restrict__ y, long long tokens, int G, int d,
                                                        int L) {
  const long long n = tokens * d;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const long long t = i / d;
    const int c = (int)(i - t * d);
    float pl[PRISM_MAX_L];
    for (int l = 0; l < L; ++l) pl[l] = __bfloat162float(pp.p[l][t * d + c]);
    const long long base = t * (long long)G * d + c;
    for (int g = 0; g < G; ++g) {
      const float uu = __bfloat162float(u[base + (long long)g * d]);
      float r = __bfloat162float(v[base + (long long)g * d]) - uu;
      float refined = 0.f;
      for (int l = 0; l < L; ++l) {
        const float delta = gelu_tanh(pl[l] * r);
        r -= delta;
        refined += delta;
      }
      y[base + (long long)g * d] = __float2bfloat16(uu + refined);
    }
  }
}

__global__ void __launch_bounds__(256) prism_bwd_kernel(const __nv_bfloat16* __restrict__ u, const __nv_bfloat16* __restrict__ v,
                                                        PrismPtrs pp, const __nv_bfloat16* __restrict__ dy,
                                                        __nv_bfloat16* __restrict__ du, __nv_bfloat16* __restrict__ dv, long long tokens,
                                                        int G, int d, int L) {
  const long long n = tokens * d;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const long long t = i / d;
    const int c = (int)(i - t * d);
    float pl[PRISM_MAX_L], dpl[PRISM_MAX_L];
    for (int l = 0; l < L; ++l) {
      pl[l] = __bfloat162float(pp.p[l][t * d + c]);
      dpl[l] = 0.f;
    }
    const long long base = t * (long long)G * d + c;
    for (int g = 0; g < G; ++g) {
      const long long idx = base + (long long)g * d;
      const float uu = __bfloat162float(u[idx]);
      const float go = __bfloat162float(dy[idx]);
      float rl[PRISM_MAX_L];
      float r = __bfloat162float(v[idx]) - uu;
      for (int l = 0; l < L; ++l) {      // forward again: r_l
        rl[l] = r;
        r -= gelu_tanh(pl[l] * r);
      }
      float dr = 0.f;                    // gradient with respect to r_{l+1}
      for (int l = L - 1; l >= 0; --l) {
        const float z = pl[l] * rl[l];
        const float dz = (go - dr) * dgelu_tanh(z);
        dpl[l] += dz * rl[l];
        dr += dz * pl[l];
      }
      du[idx] = __float2bfloat16(go - dr);
      dv[idx] = __float2bfloat16(dr);
    }
    for (int l = 0; l < L; ++l) pp.dp[l][t * d + c] = dpl[l];
  }
}

bool prism_aligned(const void* a, const void* b) { return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0; }

int prism_grid(long long n) {
  long long b = (n + 255) / 256;
  return (int)(b < 148 * 8 ? b : 148 * 8);
}

// ---- gates from their logits -------------------------------------------------------------------------
// The layer's own form: p_l = sigmoid(z_l) with the bf16 logits z_l [tokens, d] at z + l d (row pitch ldz), formed in fp32 inside the
// kernel; backward returns the gradient of the logits (bf16). A thread owns VEC channels of a token (16- or 8-byte accesses) and
// walks over the groups with UG groups' loads in flight. gelu(x) = x sigmoid(2 u) with u the argument of the tanh form: one
// exponential and one reciprocal (tanh.approx has 2^-11), and the derivative reuses the sigmoid. They are __expf and __fdividef; results, gradients
// and the carried fp32 state are as far from 64 bits as with PyTorch's functions (state: 5.5e-8 to 8.2e-7 relative against 6.0e-8 to 8.2e-7). Bound by the special
// functions (two per element and iteration) and memory about equally: 16384 tokens x 1024 channels, two iterations: 40 us forward (100 MB),
// 47 us backward (168 MB). With fp32 gates the layer ran PyTorch's elementwise kernels before: 2.85 ms forward and backward, 0.79 with these.
template <int VEC> struct PrismVec;
template <> struct PrismVec<8> { using T = uint4; };
template <> struct PrismVec<4> { using T = uint2; };

template <int VEC>
__device__ __forceinline__ void prism_unpack(float (&f)[VEC], const typename PrismVec<VEC>::T& v) {
  const uint32_t* p = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
  for (int i = 0; i < VEC / 2; ++i) {
    f[2 * i] = bf16_lo(p[i]);
    f[2 * i + 1] = bf16_hi(p[i]);
  }
}
template <int VEC>
__device__ __forceinline__ typename PrismVec<VEC>::T prism_pack(const float (&f)[VEC]) {
  typename PrismVec<VEC>::T v;
  uint32_t* p = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
  for (int i = 0; i < VEC / 2; ++i) p[i] = pack_bf16(f[2 * i], f[2 * i + 1]);
  return v;
}

template <int L, int VEC>
__global__ void __launch_bounds__(256) prism_gated_fwd_kernel(const __nv_bfloat16* __restrict__ u, const __nv_bfloat16* __restrict__ v,
                                                              const __nv_bfloat16* __restrict__ z, long long ldz,
                                                              __nv_bfloat16* __restrict__ y, long long tokens, int G, int d, int parts) {
  using V = typename PrismVec<VEC>::T;
  constexpr int UG = 4;
  const int per = d / VEC, each = ((G + parts - 1) / parts + UG - 1) / UG * UG;           // groups of a thread
  const long long n = tokens * per * parts;
  for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
    const long long i = j % (tokens * per), t = i / per;
    const int c = (int)(i - t * per) * VEC, from = (int)(j / (tokens * per)) * each, to = min(G, from + each);
    float p[L][VEC];
#pragma unroll
    for (int l = 0; l < L; ++l) {
      prism_unpack<VEC>(p[l], *reinterpret_cast<const V*>(z + t * ldz + (long long)l * d + c));
#pragma unroll
      for (int x = 0; x < VEC; ++x) p[l][x] = prism_sigmoid(p[l][x]);
    }
    const long long base = t * (long long)G * d + c;
    for (int g0 = from; g0 < to; g0 += UG) {
      V uq[UG], vq[UG];
#pragma unroll
      for (int k = 0; k < UG; ++k)
        if (g0 + k < to) {
          uq[k] = *reinterpret_cast<const V*>(u + base + (long long)(g0 + k) * d);
          vq[k] = *reinterpret_cast<const V*>(v + base + (long long)(g0 + k) * d);
        }
#pragma unroll
      for (int k = 0; k < UG; ++k)
        if (g0 + k < to) {
          float uu[VEC], r[VEC];
          prism_unpack<VEC>(uu, uq[k]);
          prism_unpack<VEC>(r, vq[k]);
#pragma unroll
          for (int x = 0; x < VEC; ++x) {
            float res = r[x] - uu[x], refined = 0.f;
#pragma unroll
            for (int l = 0; l < L; ++l) {
              const float delta = prism_delta(p[l][x], res);
              res -= delta;
              refined += delta;
            }
            uu[x] += refined;
          }
          *reinterpret_cast<V*>(y + base + (long long)(g0 + k) * d) = prism_pack<VEC>(uu);
        }
    }
  }
}

template <int L, int VEC>
__global__ void __launch_bounds__(256) prism_gated_bwd_kernel(const __nv_bfloat16* __restrict__ u, const __nv_bfloat16* __restrict__ v,
                                                              const __nv_bfloat16* __restrict__ z, long long ldz,
                                                              const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ du,
                                                              __nv_bfloat16* __restrict__ dv, __nv_bfloat16* __restrict__ dz,
                                                              long long tokens, int G, int d) {
  using V = typename PrismVec<VEC>::T;
  constexpr int UG = 2;
  const int per = d / VEC;
  const long long n = tokens * per;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / per;
    const int c = (int)(i - t * per) * VEC;
    float p[L][VEC], dp[L][VEC];
#pragma unroll
    for (int l = 0; l < L; ++l) {
      prism_unpack<VEC>(p[l], *reinterpret_cast<const V*>(z + t * ldz + (long long)l * d + c));
#pragma unroll
      for (int x = 0; x < VEC; ++x) {
        p[l][x] = prism_sigmoid(p[l][x]);
        dp[l][x] = 0.f;
      }
    }
    const long long base = t * (long long)G * d + c;
    for (int g0 = 0; g0 < G; g0 += UG) {
      V uq[UG], vq[UG], gq[UG];
#pragma unroll
      for (int k = 0; k < UG; ++k)
        if (g0 + k < G) {
          const long long idx = base + (long long)(g0 + k) * d;
          uq[k] = *reinterpret_cast<const V*>(u + idx);
          vq[k] = *reinterpret_cast<const V*>(v + idx);
          gq[k] = *reinterpret_cast<const V*>(dy + idx);
        }
#pragma unroll
      for (int k = 0; k < UG; ++k)
        if (g0 + k < G) {
          float uu[VEC], r[VEC], go[VEC];
          prism_unpack<VEC>(uu, uq[k]);
          prism_unpack<VEC>(r, vq[k]);
          prism_unpack<VEC>(go, gq[k]);
#pragma unroll
          for (int x = 0; x < VEC; ++x) {
            float rl[L], sg[L], res = r[x] - uu[x];
#pragma unroll
            for (int l = 0; l < L; ++l) {
              rl[l] = res;
              const float a = p[l][x] * res;
              sg[l] = prism_gelu_gate(a);
              res -= a * sg[l];
            }
            float dr = 0.f;                // gradient with respect to r_{l+1}
#pragma unroll
            for (int l = L - 1; l >= 0; --l) {
              const float a = p[l][x] * rl[l];
              // gelu'(a) = s + a s (1 - s) 2u'(a)
              const float da = (go[x] - dr) * fmaf(a * sg[l] * (1.f - sg[l]), 1.5957691216057308f * fmaf(0.134145f * a, a, 1.f), sg[l]);
              dp[l][x] += da * rl[l];
              dr += da * p[l][x];
            }
            uu[x] = go[x] - dr;
            r[x] = dr;
          }
          const long long idx = base + (long long)(g0 + k) * d;
          *reinterpret_cast<V*>(du + idx) = prism_pack<VEC>(uu);
          *reinterpret_cast<V*>(dv + idx) = prism_pack<VEC>(r);
        }
    }
#pragma unroll
    for (int l = 0; l < L; ++l) {
#pragma unroll
      for (int x = 0; x < VEC; ++x) dp[l][x] *= p[l][x] * (1.f - p[l][x]);
      *reinterpret_cast<V*>(dz + t * ldz + (long long)l * d + c) = prism_pack<VEC>(dp[l]);
    }
  }
}

template <int L, int VEC>
int launch_prism_gated(const void* u, const void* v, const void* z, long long ldz, const void* dy, void* out0, void* dv, void* dz,
                       long long tokens, int G, int d, cudaStream_t s) {
  const long long blocks = (tokens * (d / VEC) + 255) / 256;
  const int grid = (int)(blocks < 148 * 16 ? blocks : 148 * 16);
  const auto* U = static_cast<const __nv_bfloat16*>(u);
  const auto* X = static_cast<const __nv_bfloat16*>(v);
  const auto* Z = static_cast<const __nv_bfloat16*>(z);
  auto* O = static_cast<__nv_bfloat16*>(out0);
  if (dy)
    prism_gated_bwd_kernel<L, VEC><<<grid, 256, 0, s>>>(U, X, Z, ldz, static_cast<const __nv_bfloat16*>(dy), O,
                                                        static_cast<__nv_bfloat16*>(dv), static_cast<__nv_bfloat16*>(dz), tokens, G, d);
  else {
    // few tokens: the groups are spread over threads too, four each (the gates are formed again for every four). 128 tokens, 16 groups of 64, two iterations:
    // one thread per token and vector for all groups 16 us (four blocks), spread 6; from two blocks per SM on the gates would cost more than it gains.
    const int quads = (G + 3) / 4;
    int parts = 1;
    while (parts < quads && blocks * parts < 2 * 148) parts *= 2;
    parts = parts < quads ? parts : quads;
    const long long all = (tokens * (d / VEC) * parts + 255) / 256;
    prism_gated_fwd_kernel<L, VEC><<<(int)(all < 148 * 16 ? all : 148 * 16), 256, 0, s>>>(U, X, Z, ldz, O, tokens, G, d, parts);
  }
  ELFA_CUDA(cudaGetLastError());
  count_launches(1);
  return ELFA_OK;
}

int dispatch_prism_gated(const void* u, const void* v, const void* z, long long ldz, const void* dy, void* out0, void* dv, void* dz,
                         long long tokens, int G, int d, int L, cudaStream_t s) {
  switch (L) {     // eight channels per thread while the gates and their gradients fit the registers
    case 1: return launch_prism_gated<1, 8>(u, v, z, ldz, dy, out0, dv, dz, tokens, G, d, s);
    case 2: return launch_prism_gated<2, 8>(u, v, z, ldz, dy, out0, dv, dz, tokens, G, d, s);
    case 3: return launch_prism_gated<3, 8>(u, v, z, ldz, dy, out0, dv, dz, tokens, G, d, s);
    case 4: return launch_prism_gated<4, 4>(u, v, z, ldz, dy, out0, dv, dz, tokens, G, d, s);
    case 5: return launch_prism_gated<5, 4>(u, v, z, ldz, dy, out0, dv, dz, tokens, G, d, s);
    case 6: return launch_prism_gated<6, 4>(u, v, z, ldz, dy, out0, dv, dz, tokens, G, d, s);
    case 7: return launch_prism_gated<7, 4>(u, v, z, ldz, dy, out0, dv, dz, tokens, G, d, s);
    default: return launch_prism_gated<8, 4>(u, v, z, ldz, dy, out0, dv, dz, tokens, G, d, s);
  }
}

// ---- weight gradients of the gates ----------------------------------------------------------------------
// out_l [D, d] = sum over the slices of parts [slice][row][L d], columns l d .. l d + d - 1, in slice order: the same bits on every call. A
// thread owns one element. mode: 0 bf16 store, 1 fp32 store, 2 fp32 add, 3 bf16 add, -1 not wanted.
struct PrismSumOut {
  void* out[PRISM_MAX_L];
  long long ld[PRISM_MAX_L];
  int mode[PRISM_MAX_L];
};

__global__ void __launch_bounds__(256) prism_weight_sum_kernel(const float* __restrict__ parts, int splits, long long split_stride, int D,
                                                               int d, int L, const PrismSumOut o) {
  const int cols = L * d;
  const long long n = (long long)D * cols;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int row = (int)(i / cols), col = (int)(i % cols), l = col / d;
    const int mode = o.mode[l];
    if (mode < 0) continue;
    float s = 0.f;
#pragma unroll 8
    for (int k = 0; k < splits; ++k) s += parts[k * split_stride + i];
    const long long at = row * o.ld[l] + (col - l * d);
    if (mode == 1 || mode == 2) {
      float* p = static_cast<float*>(o.out[l]) + at;
      *p = mode == 2 ? *p + s : s;
    } else {
      __nv_bfloat16* p = static_cast<__nv_bfloat16*>(o.out[l]) + at;
      *p = __float2bfloat16(mode == 3 ? __bfloat162float(*p) + s : s);
    }
  }
}

// ---- fast-weight state carry ---------------------------------------------------------------------------
// Per (batch, group), state S [D, D] fp32 over the tokens t and iterations l (reference: src/model/prism.zig:318-421):
//   k = z_k / |z_k|, b = sigmoid(mean z_b), delta_l as in the refinement
//   l = 0: S <- forget S + b (delta - forget S k) k^T        l > 0: S <- S + b delta k^T
// The rows of S never meet, so a quad of threads owns a row (D / 4 columns each, in registers for the whole block of tokens; the dot
// product is two shuffles) and one CTA of 4 D threads owns a (batch, group). Keys, gates and deltas of a tile of tokens are
// formed in parallel in shared memory first, so the serial part of a token is about D / 2 + L D / 4 multiply-adds per thread. Tiles of up to 64 tokens,
// four items of a warp or thread in flight: with tiles of eight, one item at a time and a division per iteration the preparation of a block of 64 tokens took
// twice as long as its walk. (B 2, 16 groups of 64, two iterations, 64 tokens: 33 us, with tiles of eight 51.) Tiles below 16 have no four items: one, and four
// iterations of its loads in flight (one token of 16 groups of 64, eight iterations: 6.5 us, four items 10.5). Where the states are several to an SM a tile
// takes its part of the shared memory (2048 of 32, eight iterations, 64 tokens: 352 us; half of an SM's whatever their number 830, tiles of eight 468).
template <int D, int U>
__global__ void __launch_bounds__(4 * D) prism_state_kernel(const __nv_bfloat16* __restrict__ u, const __nv_bfloat16* __restrict__ v,
                                                            const __nv_bfloat16* __restrict__ z, long long ldz, int off_b, int off_k,
                                                            const float* __restrict__ state, float* __restrict__ out, int T, int G, int L,
                                                            float forget, int tile) {
  extern __shared__ __align__(16) float ps_smem[];
  const PrismTile<D> sm(ps_smem, tile, L);
  const PrismSource in{u, v, z, ldz, off_b, off_k, T, G, L};
  const int bg = blockIdx.x, row = threadIdx.x >> 2, part = threadIdx.x & 3;
  float S[D / 4];
  prism_state_load<D>(S, state + ((long long)bg * D + row) * D, part);
  for (int t0 = 0; t0 < T; t0 += tile) {
    const int n = min(tile, T - t0);
    if (t0) __syncthreads();                    // the previous tokens have been consumed
    prism_state_prepare<D, 4 * D, U, U == 1 ? 4 : 1>(in, sm, bg, t0, n, threadIdx.x, [] { __syncthreads(); });
    prism_state_rows<D>(S, sm, n, L, row, part, forget);
  }
  prism_state_store<D>(S, out + ((long long)bg * D + row) * D, part);
}

constexpr int PS_SHARED = 110 * 1024;           // most that a tile takes: half of an SM's
template <int D, int U>
int launch_prism_state_as(const void* u, const void* v, const void* z, long long ldz, int off_b, int off_k, const float* state, float* out,
                          int B, int T, int G, int L, float forget, int tile, int bytes, cudaStream_t s) {
  ELFA_CUDA((allow_shared<prism_state_kernel<D, U>>(PS_SHARED)));
  prism_state_kernel<D, U><<<B * G, 4 * D, bytes, s>>>(static_cast<const __nv_bfloat16*>(u), static_cast<const __nv_bfloat16*>(v),
                                                       static_cast<const __nv_bfloat16*>(z), ldz, off_b, off_k, state, out, T, G, L, forget, tile);
  ELFA_CUDA(cudaGetLastError());
  count_launches(1);
  return ELFA_OK;
}
template <int D>
int launch_prism_state(const void* u, const void* v, const void* z, long long ldz, int off_b, int off_k, const float* state, float* out,
                       int B, int T, int G, int L, float forget, cudaStream_t s) {
  // tokens of a tile, a multiple of four (its parts start on 16 bytes): up to 64, as the CTAs that an SM will have, by the registers at most 1024 threads,
  // leave room for, at least eight
  const int token = (2 * D + 1) * L * (int)sizeof(float);
  const long long ctas = std::min<long long>(std::max(2, 1024 / (4 * D)), std::max<long long>(2, ((long long)B * G + 147) / 148));
  const int room = std::min(PS_SHARED, (int)(220 * 1024 / ctas)), least = std::min(8, PS_SHARED / token / 4 * 4);
  const int most = std::max(least, std::min(64, room / token / 4 * 4)), tile = std::min(most, std::max(4, (T + 3) / 4 * 4));
  return tile < 16 ? launch_prism_state_as<D, 1>(u, v, z, ldz, off_b, off_k, state, out, B, T, G, L, forget, tile, tile * token, s)
                   : launch_prism_state_as<D, 4>(u, v, z, ldz, off_b, off_k, state, out, B, T, G, L, forget, tile, tile * token, s);
}

}  // namespace
}  // namespace elfa

using namespace elfa;

// u, v, y: [tokens, G * d] bf16; p: host array of L device pointers to [tokens, d] bf16 (already sigmoid-ed).
ELFA_API int elfa_prism_fwd(const void* u, const void* v, const unsigned long long* p, void* y, long long tokens, int G, int d, int L,
                            void* stream) {
  ELFA_REQUIRE(u && v && p && y && tokens > 0 && G > 0 && d > 0 && L >= 1 && L <= PRISM_MAX_L, "prism_fwd: bad arguments");
  PrismPtrs pp{};
  for (int l = 0; l < L; ++l) pp.p[l] = reinterpret_cast<const __nv_bfloat16*>(p[l]);
  prism_fwd_kernel<<<prism_grid(tokens * d), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(u), static_cast<const __nv_bfloat16*>(v), pp, static_cast<__nv_bfloat16*>(y), tokens, G, d, L);
  ELFA_CUDA(cudaGetLastError());
  count_launches(1);
  return ELFA_OK;
}

// du, dv: [tokens, G * d] bf16; dp: host array of L device pointers to [tokens, d] fp32.
ELFA_API int elfa_prism_bwd(const void* u, const void* v, const unsigned long long* p, const void* dy, void* du, void* dv,
                            const unsigned long long* dp, long long tokens, int G, int d, int L, void* stream) {
  ELFA_REQUIRE(u && v && p && dy && du && dv && dp && tokens > 0 && G > 0 && d > 0 && L >= 1 && L <= PRISM_MAX_L,
               "prism_bwd: bad arguments");
  PrismPtrs pp{};
  for (int l = 0; l < L; ++l) {
    pp.p[l] = reinterpret_cast<const __nv_bfloat16*>(p[l]);
    pp.dp[l] = reinterpret_cast<float*>(dp[l]);
  }
  prism_bwd_kernel<<<prism_grid(tokens * d), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(u), static_cast<const __nv_bfloat16*>(v), pp, static_cast<const __nv_bfloat16*>(dy),
      static_cast<__nv_bfloat16*>(du), static_cast<__nv_bfloat16*>(dv), tokens, G, d, L);
  ELFA_CUDA(cudaGetLastError());
  count_launches(1);
  return ELFA_OK;
}

// The layer's form: z = logits of the L gates, [tokens, L * d] bf16 with row pitch ldz. y: [tokens, G * d] bf16. Pointers 16-byte aligned,
// d and ldz multiples of 8.
ELFA_API int elfa_prism_gated_fwd(const void* u, const void* v, const void* z, long long ldz, void* y, long long tokens, int G, int d, int L,
                                  void* stream) {
  ELFA_REQUIRE(u && v && z && y && tokens > 0 && G > 0 && d > 0 && L >= 1 && L <= PRISM_MAX_L, "prism_gated_fwd: bad arguments");
  ELFA_REQUIRE(d % 8 == 0 && ldz % 8 == 0 && prism_aligned(u, v) && prism_aligned(z, y), "prism_gated_fwd: 8-element alignment");
  return dispatch_prism_gated(u, v, z, ldz, nullptr, y, nullptr, nullptr, tokens, G, d, L, static_cast<cudaStream_t>(stream));
}

// du, dv: [tokens, G * d] bf16 (du without the part that comes through the logits); dz: [tokens, L * d] bf16 with row pitch ldz.
ELFA_API int elfa_prism_gated_bwd(const void* u, const void* v, const void* z, long long ldz, const void* dy, void* du, void* dv, void* dz,
                                  long long tokens, int G, int d, int L, void* stream) {
  ELFA_REQUIRE(u && v && z && dy && du && dv && dz && tokens > 0 && G > 0 && d > 0 && L >= 1 && L <= PRISM_MAX_L,
               "prism_gated_bwd: bad arguments");
  ELFA_REQUIRE(d % 8 == 0 && ldz % 8 == 0 && prism_aligned(u, v) && prism_aligned(z, dy) && prism_aligned(du, dv) && prism_aligned(dz, dz),
               "prism_gated_bwd: 8-element alignment");
  return dispatch_prism_gated(u, v, z, ldz, dy, du, dv, dz, tokens, G, d, L, static_cast<cudaStream_t>(stream));
}

// parts: what elfa_gemm_bf16_parts left, split_stride elements from slice to slice. outs: L triples (pointer, row pitch, mode; see
// prism_weight_sum_kernel), host memory.
ELFA_API int elfa_prism_weight_sum(const float* parts, int splits, long long split_stride, int D, int d, int L, const unsigned long long* outs,
                                   void* stream) {
  ELFA_REQUIRE(parts && outs && splits > 0 && D > 0 && d > 0 && L >= 1 && L <= PRISM_MAX_L, "prism_weight_sum: bad arguments");
  PrismSumOut o{};
  for (int l = 0; l < L; ++l) {
    o.out[l] = reinterpret_cast<void*>(outs[3 * l]);
    o.ld[l] = (long long)outs[3 * l + 1];
    o.mode[l] = (int)(long long)outs[3 * l + 2];
    ELFA_REQUIRE(o.mode[l] >= -1 && o.mode[l] <= 3 && (o.mode[l] < 0 || o.out[l]), "prism_weight_sum: bad output");
  }
  const long long blocks = ((long long)D * L * d + 255) / 256;
  prism_weight_sum_kernel<<<(int)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(parts, splits, split_stride, D,
                                                                                                               d, L, o);
  ELFA_CUDA(cudaGetLastError());
  count_launches(1);
  return ELFA_OK;
}

// Carries the fast-weight state [B, G, d, d] fp32 over T tokens. u, v: [B, T, G * d] bf16; z: [B * T, ..] bf16 with row pitch ldz holding the
// logits of the L gates at column 0, of the betas at off_b and the unnormalised keys at off_k (L * d columns each).
ELFA_API int elfa_prism_state(const void* u, const void* v, const void* z, long long ldz, int off_b, int off_k, const float* state, float* out,
                              int B, int T, int G, int d, int L, float forget, void* stream) {
  ELFA_REQUIRE(u && v && z && state && out && B > 0 && T > 0 && G > 0 && L >= 1 && L <= PRISM_MAX_L, "prism_state: bad arguments");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (d) {
    case 32: return launch_prism_state<32>(u, v, z, ldz, off_b, off_k, state, out, B, T, G, L, forget, s);
    case 64: return launch_prism_state<64>(u, v, z, ldz, off_b, off_k, state, out, B, T, G, L, forget, s);
    case 96: return launch_prism_state<96>(u, v, z, ldz, off_b, off_k, state, out, B, T, G, L, forget, s);
    case 128: return launch_prism_state<128>(u, v, z, ldz, off_b, off_k, state, out, B, T, G, L, forget, s);
    default: set_last_error("prism_state: group size must be 32, 64, 96 or 128"); return ELFA_ERR_UNSUPPORTED;
  }
}
