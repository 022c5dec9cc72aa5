// Gates, refinement and fast-weight state of PRISM (prism.cu): what decode.cu runs inside a whole decoding step too.
#pragma once
#include "common.cuh"

namespace elfa {

constexpr int PRISM_MAX_L = 8;

__device__ __forceinline__ float prism_sigmoid(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }
// -> sigmoid(2u) of the tanh-form GELU at x
__device__ __forceinline__ float prism_gelu_gate(float x) {
  return prism_sigmoid(1.5957691216057308f * x * fmaf(0.044715f * x, x, 1.f));
}

__device__ __forceinline__ float prism_delta(float p, float res) {
  const float a = p * res;
  return a * prism_gelu_gate(a);
}

struct PrismSource {
  const __nv_bfloat16 *u, *v, *z;
  long long ldz;
  int off_b, off_k, T, G, L;
};
// Shared memory of a tile: keys and deltas [tokens][L][D], b [tokens][L]
template <int D>
struct PrismTile {
  float *k, *d, *b;
  __device__ PrismTile(float* at, int tokens, int L) : k(at), d(at + tokens * L * D), b(at + 2 * tokens * L * D) {}
};

template <int D>
__device__ __forceinline__ void prism_state_load(float (&S)[D / 4], const float* sp, int part) {
#pragma unroll
  for (int m = 0; m < D / 16; ++m)
#pragma unroll
    for (int x = 0; x < 4; ++x) S[4 * m + x] = sp[m * 16 + part * 4 + x];
}
template <int D>
__device__ __forceinline__ void prism_state_store(const float (&S)[D / 4], float* op, int part) {
#pragma unroll
  for (int m = 0; m < D / 16; ++m)
#pragma unroll
    for (int x = 0; x < 4; ++x) op[m * 16 + part * 4 + x] = S[4 * m + x];
}

// keys, gates and deltas of tokens t0 .. t0 + n - 1 of (batch, group) bg by NT threads (tid), U items of a warp or thread at a time so that their loads are
// in flight together, and of a delta's iterations LU; ends with a barrier
template <int D, int NT, int U, int LU, typename Sync>
__device__ __forceinline__ void prism_state_prepare(const PrismSource& in, const PrismTile<D>& sm, int bg, int t0, int n, int tid, Sync together) {
  const int b = bg / in.G, g = bg % in.G, warp = tid >> 5, lane = tid & 31, L = in.L, items = n * L;
  const long long ldz = in.ldz, first = (long long)b * in.T + t0;
#pragma unroll 1
  for (int i0 = warp; i0 < items; i0 += NT / 32 * U) {
    __nv_bfloat16 kz[U][D / 32], bz[U][D / 32];
#pragma unroll
    for (int y = 0; y < U; ++y) {
      const int i = min(i0 + y * (NT / 32), items - 1), tt = i / L;
      const __nv_bfloat16* zr = in.z + (first + tt) * ldz + (i - tt * L) * D + lane;
#pragma unroll
      for (int m = 0; m < D / 32; ++m) {
        kz[y][m] = zr[in.off_k + m * 32];
        bz[y][m] = zr[in.off_b + m * 32];
      }
    }
#pragma unroll
    for (int y = 0; y < U; ++y) {
      const int i = i0 + y * (NT / 32);
      if (i >= items) break;
      float kx[D / 32], ss = 0.f, sum = 0.f;
#pragma unroll
      for (int m = 0; m < D / 32; ++m) {
        kx[m] = __bfloat162float(kz[y][m]);
        ss += kx[m] * kx[m];
        sum += __bfloat162float(bz[y][m]);
      }
      ss = sqrtf(warp_sum(ss));
      sum = warp_sum(sum);
      const float inv = ss < 1e-12f ? 1.f : 1.f / ss;
#pragma unroll
      for (int m = 0; m < D / 32; ++m) sm.k[i * D + m * 32 + lane] = kx[m] * inv;
      if (lane == 0) sm.b[i] = prism_sigmoid(sum / (float)D);
    }
  }
#pragma unroll 1
  for (int i0 = NT - 1 - tid; i0 < n * D; i0 += NT * U) {   // beside the keys, from the last warp on
    float r[U];
    long long row[U];
#pragma unroll
    for (int y = 0; y < U; ++y) {
      const int i = min(i0 + y * NT, n * D - 1), c = i % D;
      row[y] = first + i / D;
      const long long at = (row[y] * in.G + g) * D + c;
      r[y] = __bfloat162float(in.v[at]) - __bfloat162float(in.u[at]);
    }
#pragma unroll LU
    for (int l = 0; l < L; ++l) {
      __nv_bfloat16 z[U];
#pragma unroll
      for (int y = 0; y < U; ++y) z[y] = in.z[row[y] * ldz + l * D + (i0 + y * NT) % D];
#pragma unroll
      for (int y = 0; y < U; ++y) {
        const float delta = prism_delta(prism_sigmoid(__bfloat162float(z[y])), r[y]);
        r[y] -= delta;
        const int i = i0 + y * NT;
        if (i < n * D) sm.d[(i / D * L + l) * D + i % D] = delta;
      }
    }
  }
  together();
}

// one row of the state, a quad of threads, over the n tokens of a tile
template <int D>
__device__ __forceinline__ void prism_state_rows(float (&S)[D / 4], const PrismTile<D>& sm, int n, int L, int row, int part, float forget) {
  auto add = [&](int i, float coef) {
    const float4* kr = reinterpret_cast<const float4*>(sm.k + i * D);
#pragma unroll
    for (int m = 0; m < D / 16; ++m) {
      const float4 kk = kr[m * 4 + part];
      S[4 * m] += coef * kk.x;
      S[4 * m + 1] += coef * kk.y;
      S[4 * m + 2] += coef * kk.z;
      S[4 * m + 3] += coef * kk.w;
    }
  };
#pragma unroll 1
  for (int t = 0, i = 0; t < n; ++t) {
    const float4* kr = reinterpret_cast<const float4*>(sm.k + i * D);
    float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
#pragma unroll
    for (int m = 0; m < D / 16; ++m) {
      const float4 kk = kr[m * 4 + part];
      p0 += kk.x * S[4 * m];
      p1 += kk.y * S[4 * m + 1];
      p2 += kk.z * S[4 * m + 2];
      p3 += kk.w * S[4 * m + 3];
    }
    float p = (p0 + p1) + (p2 + p3);
    p += __shfl_xor_sync(0xffffffffu, p, 1);
    p += __shfl_xor_sync(0xffffffffu, p, 2);
    const float coef = sm.b[i] * sm.d[i * D + row] - sm.b[i] * forget * p;
#pragma unroll
    for (int m = 0; m < D / 4; ++m) S[m] *= forget;
    add(i, coef);
    ++i;
#pragma unroll 1
    for (int l = 1; l < L; ++l, ++i) add(i, sm.b[i] * sm.d[i * D + row]);
  }
}

}  // namespace elfa
