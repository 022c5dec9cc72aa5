// Attention of a few new positions against a key / value cache (incremental decoding), with the cache's growth in the same pass.
//
// q [s, B, H, hd], the new keys / values [s, B, Hkv, hd] (slices of the fused projection output) and the cache [t, B, Hkv, hd] give
// out [s, B, H * hd] and the cache of t + s rows. Scores, softmax and the sum over the values are fp32. A CTA owns one (batch, key
// head) and a slice of the positions: it copies its rows into the new cache while they pass through, scores them against all
// rep * s query rows that share the key head (H / Hkv = rep heads read a key once) and leaves an unnormalised partial result; a second
// small launch combines the slices (fixed order). Bound by latency at small t and by the
// read and write of the cache at large t. B 4, 16 heads of 64 on 4 key heads, t 512: 4.9 + 4.1 us; concatenation, head repetition and fp32 einsum
// in PyTorch: about 15 launches.
//
// reference: src/eval/evaluator.zig:419-470 (generation runs the whole context again for every token).
#include <type_traits>

#include "common.cuh"
#include "elfa_native.h"

namespace elfa {
namespace {

constexpr int DEC_MAX_SLICE = 256;

struct DecodeParams {
  const __nv_bfloat16 *q, *knew, *vnew, *kold, *vold;
  __nv_bfloat16 *kout, *vout, *out;
  float *part, *stat;                  // [slices][B * Hkv * R][hd], [slices][B * Hkv * R][2] (max, sum)
  long long ss, sb;                    // strides of q / knew / vnew over positions and batch
  int t, s, B, H, Hkv, slice, slices;
  float scale;
};

// R >= s * rep query rows per key head (the surplus rows repeat the last one and are not written)
template <int HD, int R>
__global__ void __launch_bounds__(128) attn_decode_kernel(const DecodeParams p) {
  constexpr int LPK = HD / 8, KPW = 32 / LPK, UN = 4;       // lanes per key, keys per warp and pass, passes in flight
  constexpr int CP = HD / 2, NG = 128 / CP;                 // value columns are taken in pairs; key groups of the second pass
  __shared__ float sc[R][DEC_MAX_SLICE];
  __shared__ float red[NG][R][HD];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.x / p.Hkv, hk = blockIdx.x % p.Hkv, rep = p.H / p.Hkv, rows = p.s * rep, total = p.t + p.s;
  const int k0 = blockIdx.y * p.slice, n = min(p.slice, total - k0);
  const long long crow = (long long)p.B * p.Hkv * HD, coff = ((long long)b * p.Hkv + hk) * HD;
  const __nv_bfloat16* kn = p.knew + b * p.sb + (long long)hk * HD;
  const __nv_bfloat16* vn = p.vnew + b * p.sb + (long long)hk * HD;

  pdl_wait();
  pdl_next();
  float qr[R][8];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int rr = min(r, rows - 1), qi = rr / rep, h = hk * rep + rr % rep;
    const uint4 v = *reinterpret_cast<const uint4*>(p.q + qi * p.ss + b * p.sb + (long long)h * HD + (lane % LPK) * 8);
    const uint32_t* pv = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      qr[r][2 * j] = bf16_lo(pv[j]);
      qr[r][2 * j + 1] = bf16_hi(pv[j]);
    }
  }
  for (int kb = warp * KPW * UN; kb < n; kb += 4 * KPW * UN) {
    uint4 kq[UN];
#pragma unroll
    for (int x = 0; x < UN; ++x) {
      const int key = kb + x * KPW + lane / LPK, at = k0 + key;
      kq[x] = make_uint4(0, 0, 0, 0);
      if (key < n)
        kq[x] = at < p.t ? *reinterpret_cast<const uint4*>(p.kold + at * crow + coff + (lane % LPK) * 8)
                         : *reinterpret_cast<const uint4*>(kn + (at - p.t) * p.ss + (lane % LPK) * 8);
    }
#pragma unroll
    for (int x = 0; x < UN; ++x) {
      const int key = kb + x * KPW + lane / LPK, at = k0 + key;
      if (key < n) *reinterpret_cast<uint4*>(p.kout + at * crow + coff + (lane % LPK) * 8) = kq[x];
      const uint32_t* pk = reinterpret_cast<const uint32_t*>(&kq[x]);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float a = 0.f, c = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          a += qr[r][2 * j] * bf16_lo(pk[j]);
          c += qr[r][2 * j + 1] * bf16_hi(pk[j]);
        }
        a += c;
#pragma unroll
        for (int o = LPK / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (key < n && lane % LPK == 0) sc[r][key] = a * p.scale;
      }
    }
  }
  __syncthreads();
  for (int r = warp; r < R; r += 4) {
    // which keys are hidden follows from positions, never from the scores: fmaxf passes over NaN, so a slice whose visible scores are all
    // NaN keeps -inf as its maximum and must still hand its NaN on
    const int seen = min(n, p.t + r / rep + 1 - k0);
    float mx = -INFINITY;
    for (int i = lane; i < seen; i += 32) mx = fmaxf(mx, sc[r][i]);
    mx = warp_max(mx);
    const float ref = mx == -INFINITY ? 0.f : mx;
    float sum = 0.f;
    for (int i = lane; i < seen; i += 32) {
      const float e = expf(sc[r][i] - ref);
      sc[r][i] = e;
      sum += e;
    }
    sum = warp_sum(sum);
    if (lane == 0 && r < rows) {
      float* st = p.stat + (((long long)blockIdx.y * gridDim.x + blockIdx.x) * rows + r) * 2;
      st[0] = mx;
      st[1] = sum;
    }
  }
  __syncthreads();
  const int grp = threadIdx.x / CP, cp = threadIdx.x % CP;
  float acc[R][2];
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r][0] = acc[r][1] = 0.f;
  constexpr int UV = 8;
  // CHECK: the slice holds keys that lie behind a row's position t + r / rep; they must not reach its sum even when their value is not finite
  auto values = [&](auto check) {
    for (int kb = grp; kb < n; kb += NG * UV) {
      uint32_t vq[UV];
#pragma unroll
      for (int x = 0; x < UV; ++x) {
        const int key = kb + x * NG, at = k0 + key;
        vq[x] = 0u;
        if (key < n)
          vq[x] = at < p.t ? *reinterpret_cast<const uint32_t*>(p.vold + at * crow + coff + cp * 2)
                           : *reinterpret_cast<const uint32_t*>(vn + (at - p.t) * p.ss + cp * 2);
      }
#pragma unroll
      for (int x = 0; x < UV; ++x) {
        const int key = kb + x * NG;
        if (key >= n) continue;
        *reinterpret_cast<uint32_t*>(p.vout + (k0 + key) * crow + coff + cp * 2) = vq[x];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float w = sc[r][key];
          if (check.value && k0 + key > p.t + r / rep) continue;
          acc[r][0] += w * bf16_lo(vq[x]);
          acc[r][1] += w * bf16_hi(vq[x]);
        }
      }
    }
  };
  if (k0 + n - 1 <= p.t) values(std::false_type{});
  else values(std::true_type{});
#pragma unroll
  for (int r = 0; r < R; ++r) *reinterpret_cast<float2*>(&red[grp][r][cp * 2]) = make_float2(acc[r][0], acc[r][1]);
  __syncthreads();
  for (int i = threadIdx.x; i < rows * HD; i += 128) {
    const int r = i / HD, c = i % HD;
    float a = 0.f;
#pragma unroll
    for (int g = 0; g < NG; ++g) a += red[g][r][c];
    p.part[(((long long)blockIdx.y * gridDim.x + blockIdx.x) * rows + r) * HD + c] = a;
  }
}

// grid B * Hkv * rows, block hd: out = sum_i part_i exp(m_i - M) / sum_i l_i exp(m_i - M). The weights of up to 256 slices are formed side by side,
// one per thread, and the partial results are fetched eight at a time: one slice after the other they took 9.7 us at B 1, t 4096
// (129 slices), 9.1 this way; with 17 slices (B 4, t 512) 4.5 and 4.1.
__global__ void attn_decode_combine_kernel(const DecodeParams p, int hd) {
  pdl_wait();
  pdl_next();
  __shared__ float sw[256], red[2][8];
  const int rep = p.H / p.Hkv, rows = p.s * rep, bhk = blockIdx.x / rows, r = blockIdx.x % rows, c = threadIdx.x;
  const int warp = c >> 5, warps = hd >> 5;
  const long long step = (long long)p.B * p.Hkv * rows;
  const float2* stat = reinterpret_cast<const float2*>(p.stat) + blockIdx.x;
  const int b = bhk / p.Hkv, h = (bhk % p.Hkv) * rep + r % rep;
  __nv_bfloat16* out = p.out + (((long long)(r / rep) * p.B + b) * p.H + h) * hd + c;
  if (p.slices == 1) {
    *out = __float2bfloat16(p.part[(long long)blockIdx.x * hd + c] / stat[0].y);
    return;
  }
  float M = -INFINITY;
  for (int i = c; i < p.slices; i += hd) M = fmaxf(M, stat[i * step].x);
  M = warp_max(M);
  if ((c & 31) == 0) red[0][warp] = M;
  __syncthreads();
  for (int i = 0; i < warps; ++i) M = fmaxf(M, red[0][i]);
  float num = 0.f, den = 0.f;
  for (int base = 0; base < p.slices; base += 256) {
    const int n = min(256, p.slices - base);
    if (base) __syncthreads();
    for (int i = c; i < n; i += hd) {
      const float2 st = stat[(base + i) * step];
      // nothing but hidden keys (or scores of -inf): adds nothing; a slice of NaN scores has -inf for its maximum too, but a NaN sum
      const float w = st.x == -INFINITY && st.y == 0.f ? 0.f : expf(st.x - M);
      sw[i] = w;
      den += w * st.y;
    }
    __syncthreads();
    const float* part = p.part + (base * step + blockIdx.x) * hd + c;
    const long long stride = step * hd;
    int i = 0;
    for (; i + 8 <= n; i += 8, part += 8 * stride) {
      float v[8];
#pragma unroll
      for (int x = 0; x < 8; ++x) v[x] = __ldg(part + x * stride);
#pragma unroll
      for (int x = 0; x < 8; ++x) num += sw[i + x] * v[x];
    }
    float v[7];
#pragma unroll
    for (int x = 0; x < 7; ++x) v[x] = i + x < n ? __ldg(part + x * stride) : 0.f;
#pragma unroll
    for (int x = 0; x < 7; ++x)
      if (i + x < n) num += sw[i + x] * v[x];
  }
  den = warp_sum(den);
  if ((c & 31) == 0) red[1][warp] = den;
  __syncthreads();
  den = 0.f;
  for (int i = 0; i < warps; ++i) den += red[1][i];
  *out = __float2bfloat16(num / den);
}

template <int HD>
int launch_decode(const DecodeParams& p, cudaStream_t st) {
  const int rows = p.s * (p.H / p.Hkv);
  const dim3 grid(p.B * p.Hkv, p.slices);
  auto kernel = rows <= 1 ? attn_decode_kernel<HD, 1> : (rows <= 2 ? attn_decode_kernel<HD, 2> : (rows <= 4 ? attn_decode_kernel<HD, 4> : attn_decode_kernel<HD, 8>));
  ELFA_CUDA(launch_chain(kernel, grid, dim3(128), 0, st, 1, p));
  ELFA_CUDA(cudaGetLastError());
  ELFA_CUDA(launch_chain(attn_decode_combine_kernel, dim3(p.B * p.Hkv * rows), dim3(HD), 0, st, 1, p, HD));
  ELFA_CUDA(cudaGetLastError());
  ::elfa::count_launches(2);
  return ELFA_OK;
}

// Positions per CTA: about two CTAs per SM, 32 to DEC_MAX_SLICE positions each.
int decode_slice(int total, int heads) {
  const int want = (2 * 148 + heads - 1) / heads;
  int slice = ((total + want - 1) / want + 31) / 32 * 32;
  return slice < 32 ? 32 : (slice > DEC_MAX_SLICE ? DEC_MAX_SLICE : slice);
}

}  // namespace
}  // namespace elfa

using namespace elfa;

// Slices the positions are split into (sizes the scratch of elfa_attention_decode: slices * B * s * H * (hd + 2) floats).
ELFA_API int elfa_attention_decode_slices(int total, int B, int Hkv) {
  if (total <= 0 || B <= 0 || Hkv <= 0) return 0;
  const int slice = decode_slice(total, B * Hkv);
  return (total + slice - 1) / slice;
}

// q / knew / vnew: bf16, element (position i, batch b, head h, column c) at i * ss + b * sb + h * hd + c, 16-byte aligned rows; kold / vold:
// [t, B, Hkv, hd] and kout / vout: [t + s, B, Hkv, hd] contiguous; out: [s, B, H * hd]. hd 32, 64, 128 or 256, s * H / Hkv <= 8.
ELFA_API int elfa_attention_decode(const void* q, const void* knew, const void* vnew, long long ss, long long sb, const void* kold,
                                   const void* vold, void* kout, void* vout, void* out, float* scratch, int t, int s, int B, int H, int Hkv,
                                   int hd, float scale, void* stream) {
  ELFA_REQUIRE(q && knew && vnew && kold && vold && kout && vout && out && scratch, "attention_decode: null pointer");
  ELFA_REQUIRE(t > 0 && s > 0 && B > 0 && Hkv > 0 && H > 0 && H % Hkv == 0 && s * (H / Hkv) <= 8, "attention_decode: bad sizes");
  ELFA_REQUIRE(ss % 8 == 0 && sb % 8 == 0, "attention_decode: row strides must be multiples of 8");
  uintptr_t bits = 0;
  for (const void* ptr : {q, knew, vnew, kold, vold, static_cast<const void*>(kout), static_cast<const void*>(vout)}) bits |= reinterpret_cast<uintptr_t>(ptr);
  ELFA_REQUIRE((bits & 15) == 0, "attention_decode: operands must be 16-byte aligned");
  DecodeParams p{};
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.knew = static_cast<const __nv_bfloat16*>(knew);
  p.vnew = static_cast<const __nv_bfloat16*>(vnew);
  p.kold = static_cast<const __nv_bfloat16*>(kold);
  p.vold = static_cast<const __nv_bfloat16*>(vold);
  p.kout = static_cast<__nv_bfloat16*>(kout);
  p.vout = static_cast<__nv_bfloat16*>(vout);
  p.out = static_cast<__nv_bfloat16*>(out);
  p.ss = ss; p.sb = sb;
  p.t = t; p.s = s; p.B = B; p.H = H; p.Hkv = Hkv;
  p.slice = decode_slice(t + s, B * Hkv);
  p.slices = (t + s + p.slice - 1) / p.slice;
  ELFA_REQUIRE(p.slices <= 65535, "attention_decode: the cache is too long");
  p.scale = scale;
  p.part = scratch;
  p.stat = scratch + (long long)p.slices * B * s * H * hd;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (hd) {
    case 32: return launch_decode<32>(p, st);
    case 64: return launch_decode<64>(p, st);
    case 128: return launch_decode<128>(p, st);
    case 256: return launch_decode<256>(p, st);
    default: set_last_error("attention_decode: head dimension must be 32, 64, 128 or 256"); return ELFA_ERR_UNSUPPORTED;
  }
}
