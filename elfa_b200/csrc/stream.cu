// Streaming calls (a prompt, then a few tokens per call, without a gradient) of both model families, issued from here: every kernel of all
// layers from one call, over one workspace. The kernels and the order of their roundings are those of the layer-by-layer route in Python.
// What this removes is host time: a decoding step of 4 layers (B 4, width 1024) is about 30 launches and took 1.1 ms to issue op by op from
// Python (autograd call, output tensors and argument conversion of each) for 0.3 ms of kernels.
//
// reference: src/model/model.zig:415-454 (streaming with carried states), src/eval/evaluator.zig:419-470.
#include <math.h>

#include "common.cuh"
#include "decode.cuh"
#include "elfa_native.h"

namespace elfa {
namespace {

typedef __nv_bfloat16 bf16;

// Workspace: pieces of 256-byte multiples. With base == nullptr only the size is counted.
struct Pieces {
  unsigned char* base;
  size_t used = 0;
  template <typename T>
  T* take(long long n) {
    T* p = reinterpret_cast<T*>(base + used);
    used += ((size_t)n * sizeof(T) + 255) / 256 * 256;
    return p;
  }
};

int linear(const void* x, const void* w, void* y, long long rows, int in, int out, unsigned flags, void* s) {      // w [in, out]
  return elfa_gemm_bf16(x, w, y, (int)rows, out, in, in, out, out, 0, 1, nullptr, nullptr, 0, nullptr, 0, 1.f, flags, 0, 0, s);
}
int logits(const void* x, const void* w, void* y, long long rows, int in, int out, void* s) {                      // w [out, in]
  return elfa_gemm_bf16(x, w, y, (int)rows, out, in, in, in, out, 0, 0, nullptr, nullptr, 0, nullptr, 0, 1.f, 0, 0, 0, s);
}
int copy2d(void* dst, size_t dpitch, const void* src, size_t spitch, size_t width, size_t height, cudaStream_t s) {
  ELFA_CUDA(cudaMemcpy2DAsync(dst, dpitch, src, spitch, width, height, cudaMemcpyDeviceToDevice, s));
  return ELFA_OK;
}

// out [D, n * d] = n matrices [D, d] side by side, 16 bytes per thread
struct ConcatArgs {
  const uint4* src[24];
};
__global__ void __launch_bounds__(256) concat_cols_kernel(const ConcatArgs a, uint4* __restrict__ out, int D, int n, int dv) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)D * n * dv) return;
  const int c = (int)(i % dv), m = (int)(i / dv % n);
  out[i] = a.src[m][i / ((long long)dv * n) * dv + c];
}

// f = act(n W_up) W_down
int mlp(const bf16* n, const void* up, const void* down, bf16* h, bf16* g, bf16* f, long long rows, int D, int F, int act, void* s) {
  int rc = linear(n, up, h, rows, D, act == ACT_SWIGLU ? 2 * F : F, act == ACT_GELU ? ELFA_EPI_GELU : 0, s);
  if (rc == ELFA_OK && act == ACT_SWIGLU) rc = elfa_swiglu(h, nullptr, g, rows, F, s);
  if (rc == ELFA_OK && act > 0) rc = elfa_elementwise(act, h, nullptr, g, rows * F, 1.f, s);
  if (rc == ELFA_OK) rc = linear(act == ACT_GELU ? h : g, down, f, rows, F, D, 0, s);
  return rc;
}

struct GptDims {
  long long S, B, D, H, Hkv, hd, F, V, layers, pos0, t, act, kind, has_pos;
};
struct GptWork {
  bf16 *x[2], *n, *f, *qkv, *o, *h, *g;
  float* scratch;
};
size_t gpt_work(const GptDims& m, unsigned char* base, GptWork* w) {
  Pieces p{base};
  const long long rows = m.S * m.B;
  w->x[0] = p.take<bf16>(rows * m.D);
  w->x[1] = p.take<bf16>(rows * m.D);
  w->n = p.take<bf16>(rows * m.D);
  w->f = p.take<bf16>(rows * m.D);
  w->qkv = p.take<bf16>(rows * (m.H + 2 * m.Hkv) * m.hd);
  w->o = p.take<bf16>(rows * m.H * m.hd);
  w->h = p.take<bf16>(rows * m.F * (m.act == ACT_SWIGLU ? 2 : 1));
  w->g = p.take<bf16>(m.act == ACT_GELU ? 0 : rows * m.F);
  const long long part = m.t > 0 ? (long long)elfa_attention_decode_slices((int)(m.t + m.S), (int)m.B, (int)m.Hkv) * (m.hd + 2) : 1;
  w->scratch = p.take<float>(rows * m.H * part);      // partial results of the cached attention, or the row log-sum-exp
  return p.used;
}

size_t efla_work(const EflaDims& m, unsigned char* base, EflaWork* w, int segments, bool step) {
  Pieces p{base};
  const long long rows = m.B * m.T, hd = m.H * m.d, chunks = (m.T + 31) / 32;
  w->x[0] = p.take<bf16>(rows * m.D);
  w->x[1] = p.take<bf16>(rows * m.D);
  w->r = p.take<bf16>(rows * m.D);
  w->n = p.take<bf16>(rows * m.D);
  w->k = p.take<bf16>(rows * hd);
  w->v = p.take<bf16>(rows * hd);
  w->o = p.take<bf16>(rows * hd);
  w->e = p.take<bf16>(rows * m.D);
  const long long positions = m.prism && m.tail ? elfa_shortconv_stream_rows((int)m.B, (int)m.tail, (int)m.T, (int)m.D, (int)m.W) : 0;
  w->full = p.take<bf16>(positions * m.D);
  w->u = positions && m.B == 1 ? w->full + m.tail * m.D : p.take<bf16>(m.prism ? rows * m.D : 0);
  w->z = p.take<bf16>(m.prism ? rows * 3 * m.L * m.d : 0);
  w->wc = p.take<bf16>(m.prism ? m.D * 3 * m.L * m.d : 0);
  w->q = p.take<bf16>(m.prism ? rows * m.D : 0);
  w->h = p.take<bf16>(rows * m.F);
  w->g = p.take<bf16>(m.act == ACT_GELU ? 0 : rows * m.F);
  w->f = p.take<bf16>(rows * m.D);
  w->nmat = p.take<bf16>(step ? 0 : m.B * m.H * chunks * 3 * 32 * 32);
  w->coef = p.take<float>(step ? 0 : m.B * m.H * chunks * 4 * 32);
  w->segw = p.take<float>(!step && segments > 1 ? 3 * segments * m.B * m.H * m.d * m.d : 0);
  w->arrived = p.take<unsigned int>(DECODE_COUNTERS);
  return p.used;
}

int kib(size_t bytes) { return (int)((bytes + 1023) / 1024); }

}  // namespace
}  // namespace elfa

using namespace elfa;

#define STREAM_CALL(expr)             \
  do {                                \
    const int rc_ = (expr);           \
    if (rc_ != ELFA_OK) return rc_;   \
  } while (0)

// dims: GptDims in order. Workspace in KiB.
ELFA_API int elfa_gpt_stream_work(const long long* dims) {
  if (!dims) return 0;
  GptWork w;
  return kib(gpt_work(*reinterpret_cast<const GptDims*>(dims), nullptr, &w));
}

// One streaming call of the softmax-attention family: ids [S, B] of positions pos0 .. of sequences whose caches hold t positions (0: a
// prompt). p: ids, token table [V, D], position table or 0, final norm weight and bias (or 0), head [V, D], logits out [S, B, V], workspace; then per
// layer: norm weight and bias, w_qkv, w_o, second norm's two, up, down, key and value cache [t, B, Hkv, hd] (or 0), the grown caches [t + S, ...].
// Weights are [in, out], contiguous, bf16.
ELFA_API int elfa_gpt_stream(const unsigned long long* p, const long long* dims, float eps, void* stream) {
  ELFA_REQUIRE(p && dims, "gpt_stream: null argument");
  const GptDims& m = *reinterpret_cast<const GptDims*>(dims);
  ELFA_REQUIRE(m.S > 0 && m.B > 0 && m.D > 0 && m.layers > 0 && m.t >= 0 && m.S * m.B < (1ll << 31), "gpt_stream: bad sizes");
  auto at = [&](int i) { return reinterpret_cast<void*>(p[i]); };
  GptWork w;
  gpt_work(m, static_cast<unsigned char*>(at(7)), &w);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int rows = (int)(m.S * m.B), D = (int)m.D, S = (int)m.S, B = (int)m.B, H = (int)m.H, Hkv = (int)m.Hkv, hd = (int)m.hd, kind = (int)m.kind;
  const long long sb = (m.H + 2 * m.Hkv) * m.hd, ss = sb * m.B;
  const float scale = (float)(1.0 / sqrt((double)m.hd));
  STREAM_CALL(elfa_embedding_fwd(static_cast<const long long*>(at(0)), at(1), m.has_pos ? at(2) : nullptr, w.x[0], rows, D, S, B, (int)m.pos0, 0, (int)m.V,
                                 (int)m.V, stream));
  // Decoding: the chain of small launches overlaps their starts, and a product's first weights are on their way before its rows are there. The
  // weights and caches that the chain reads early were written before the ordinary launch above.
  const PdlScope chain(m.t > 0);
  int cur = 0;
  for (int l = 0; l < m.layers; ++l) {
    const int q = 8 + 12 * l;
    if (l == 0) {
      STREAM_CALL(elfa_norm_fwd(w.x[0], nullptr, at(q), at(q + 1), w.n, nullptr, nullptr, nullptr, rows, D, eps, kind, stream));
    } else {
      STREAM_CALL(elfa_norm_fwd(w.x[cur], w.f, at(q), at(q + 1), w.n, w.x[cur ^ 1], nullptr, nullptr, rows, D, eps, kind, stream));
      cur ^= 1;
    }
    STREAM_CALL(linear(w.n, at(q + 2), w.qkv, rows, D, (int)sb, 0, stream));
    const bf16 *k = w.qkv + m.H * m.hd, *v = k + m.Hkv * m.hd;
    if (m.t > 0) {
      STREAM_CALL(elfa_attention_decode(w.qkv, k, v, ss, sb, at(q + 8), at(q + 9), at(q + 10), at(q + 11), w.o, w.scratch, (int)m.t, S, B, H, Hkv, hd, scale,
                                        stream));
    } else {
      const size_t width = (size_t)m.Hkv * m.hd * 2;
      STREAM_CALL(copy2d(at(q + 10), width, k, sb * 2, width, rows, s));
      STREAM_CALL(copy2d(at(q + 11), width, v, sb * 2, width, rows, s));
      STREAM_CALL(elfa_attention_fwd_ex(w.qkv, ss, sb, w.o, m.H * m.hd * m.B, m.H * m.hd, w.scratch, S, B, H, Hkv, hd, scale, 1, nullptr, stream));
    }
    STREAM_CALL(linear(w.o, at(q + 3), w.f, rows, H * hd, D, 0, stream));
    STREAM_CALL(elfa_norm_fwd(w.x[cur], w.f, at(q + 4), at(q + 5), w.n, w.x[cur ^ 1], nullptr, nullptr, rows, D, eps, kind, stream));
    cur ^= 1;
    STREAM_CALL(mlp(w.n, at(q + 6), at(q + 7), w.h, w.g, w.f, rows, D, (int)m.F, (int)m.act, stream));
  }
  STREAM_CALL(elfa_norm_fwd(w.x[cur], w.f, at(3), at(4), w.n, w.x[cur ^ 1], nullptr, nullptr, rows, D, eps, kind, stream));
  return logits(w.n, at(5), at(6), rows, D, (int)m.V, stream);
}

// dims: EflaDims in order. Workspace in KiB.
ELFA_API int elfa_efla_stream_work(const long long* dims, int step_tokens) {
  if (!dims) return 0;
  const EflaDims& m = *reinterpret_cast<const EflaDims*>(dims);
  EflaWork w;
  return kib(efla_work(m, nullptr, &w, elfa_efla_segments((int)m.B, (int)m.T, (int)m.H, (int)m.d), m.T <= step_tokens));
}

// One streaming call of the EFLA family: ids [B, T], T <= step_tokens in the token-by-token form. p: ids, token table [V, D], final norm weight
// and bias (or 0), head [V, D], logits out [B, T, V], workspace; then per layer 19 + 3 L: first norm's weight and bias, w_k, w_v, w_o, beta
// (fp32), ShortConv weight [D, W] and bias, second norm's two, up, down, EFLA state in and out, PRISM state in and out, ShortConv tail
// [B, tail, D] and its batch stride in elements, ShortConv input out [B, tail + T, D], and the 3 L gate weights [D, d] (w_p, w_beta, w_k).
// forget: one per layer. Without PRISM the fields that belong to it are 0 and L is 0.
ELFA_API int elfa_efla_stream(const unsigned long long* p, const long long* dims, const float* forget, float eps, int step_tokens, void* stream) {
  ELFA_REQUIRE(p && dims && forget, "efla_stream: null argument");
  const EflaDims& m = *reinterpret_cast<const EflaDims*>(dims);
  ELFA_REQUIRE(m.B > 0 && m.T > 0 && m.D > 0 && m.layers > 0 && m.L >= 0 && m.L <= 8 && m.tail >= 0 && m.B * m.T < (1ll << 31), "efla_stream: bad sizes");
  ELFA_REQUIRE(m.act != ACT_SWIGLU, "efla_stream: the block's MLP is not gated");       // (its buffers are F wide)
  auto at = [&](int i) { return reinterpret_cast<void*>(p[i]); };
  const int segments = elfa_efla_segments((int)m.B, (int)m.T, (int)m.H, (int)m.d);
  const bool step = m.T <= step_tokens;
  EflaWork w;
  efla_work(m, static_cast<unsigned char*>(at(6)), &w, segments, step);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int rows = (int)(m.B * m.T), D = (int)m.D, B = (int)m.B, T = (int)m.T, H = (int)m.H, d = (int)m.d, L = (int)m.L, kind = (int)m.kind, G = D / d;
  const int hd = H * d, per = 19 + 3 * L;
  if (step && efla_decode_fits(m)) {
    const int rc = efla_decode(p, m, w, forget, eps, s);
    if (rc == ELFA_OK) {
      const PdlScope head(true);
      return logits(w.n, at(4), at(5), rows, D, (int)m.V, stream);
    }
    if (rc != ELFA_ERR_UNSUPPORTED) return rc;
  }
  STREAM_CALL(elfa_embedding_fwd(static_cast<const long long*>(at(0)), at(1), nullptr, w.x[0], rows, D, T, 1, 0, 0, (int)m.V, (int)m.V, stream));
  const PdlScope chain(m.B * m.T <= 8);        // decoding, as above
  int cur = 0;
  for (int l = 0; l < m.layers; ++l) {
    const int q = 7 + per * l;
    bf16* xin = m.prism ? static_cast<bf16*>(at(q + 18)) : nullptr;
    bf16* n = m.prism && !m.tail ? xin : w.n;
    STREAM_CALL(elfa_norm_fwd(w.x[cur], nullptr, at(q), at(q + 1), n, nullptr, nullptr, nullptr, rows, D, eps, kind, stream));
    STREAM_CALL(linear(n, at(q + 2), w.k, rows, D, hd, 0, stream));
    STREAM_CALL(linear(n, at(q + 3), w.v, rows, D, hd, 0, stream));
    const float* beta = static_cast<const float*>(at(q + 5));
    const float* s0 = static_cast<const float*>(at(q + 12));
    float* s1 = static_cast<float*>(at(q + 13));
    if (step) STREAM_CALL(elfa_efla_scan_fwd(w.k, w.v, beta, s0, w.o, s1, B, T, H, d, stream));
    else STREAM_CALL(elfa_efla_chunk_fwd_cut(w.k, w.v, beta, s0, w.o, s1, nullptr, w.nmat, w.coef, segments > 1 ? w.segw : nullptr, segments, B, T, H, d, stream));
    STREAM_CALL(linear(w.o, at(q + 4), w.e, rows, hd, D, 0, stream));
    const bf16* y = w.e;
    if (m.prism) {
      if (m.tail)
        STREAM_CALL(elfa_shortconv_stream(at(q + 16), (long long)p[q + 17], n, at(q + 6), at(q + 7), xin, w.u, w.full, B, (int)m.tail, T, D, (int)m.W,
                                          stream));
      else
        STREAM_CALL(elfa_shortconv_fwd(xin, at(q + 6), at(q + 7), w.u, B, T, D, (int)m.W, stream));
      ConcatArgs a{};
      for (int i = 0; i < 3 * L; ++i) a.src[i] = static_cast<const uint4*>(at(q + 19 + i));
      const long long vecs = (long long)D * 3 * L * (d / 8);
      concat_cols_kernel<<<(unsigned)((vecs + 255) / 256), 256, 0, s>>>(a, reinterpret_cast<uint4*>(w.wc), D, 3 * L, d / 8);
      ELFA_CUDA(cudaGetLastError());
      ::elfa::count_launches(1);
      {       // its matrix was put together by the launch above: nothing of it may be asked for early
        const PdlScope whole(false);
        STREAM_CALL(linear(w.u, w.wc, w.z, rows, D, 3 * L * d, 0, stream));
      }
      STREAM_CALL(elfa_prism_gated_fwd(w.u, w.e, w.z, 3 * L * d, w.q, rows, G, d, L, stream));
      STREAM_CALL(elfa_prism_state(w.u, w.e, w.z, 3 * L * d, L * d, 2 * L * d, static_cast<const float*>(at(q + 14)), static_cast<float*>(at(q + 15)), B, T, G, d,
                                   L, forget[l], stream));
      y = w.q;
    }
    // r = q + x (fused into the norm), then x = r + MLP
    STREAM_CALL(elfa_norm_fwd(y, w.x[cur], at(q + 8), at(q + 9), w.n, w.r, nullptr, nullptr, rows, D, eps, kind, stream));
    STREAM_CALL(mlp(w.n, at(q + 10), at(q + 11), w.h, w.g, w.f, rows, D, (int)m.F, (int)m.act, stream));
    STREAM_CALL(elfa_elementwise(2, w.r, w.f, w.x[cur ^ 1], (long long)rows * D, 1.f, stream));
    cur ^= 1;
  }
  STREAM_CALL(elfa_norm_fwd(w.x[cur], nullptr, at(2), at(3), w.n, nullptr, nullptr, nullptr, rows, D, eps, kind, stream));
  return logits(w.n, at(4), at(5), rows, D, (int)m.V, stream);
}
