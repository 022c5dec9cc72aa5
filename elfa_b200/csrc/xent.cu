// Fused softmax cross-entropy: one pass for the row statistics, one pass that turns the logits
// into their gradient in place, so the [tokens, vocab] probabilities are never materialised.
// Supports label smoothing, an ignore index (-100) and a vocabulary-parallel split in which every
// rank holds a [tokens, vocab/N] slice: the statistics of the slices are combined between the two
// passes.
//
// reference: src/kernels/nn_kernels.zig:269-318 (loss with label smoothing, f64 sum-exp),
// kernels/cuda/elementwise.cu:159-300 (forward / backward kernels, out-of-range target flag; the
// reference gradient carries no 1/N and no upstream gradient - both are folded into `grad_scale` here).
#include "common.cuh"
#include "elfa_native.h"
#include "mma_sync.cuh"

namespace elfa {
namespace {

constexpr int XENT_THREADS = 512;

struct RowStat {  // per row and per vocabulary slice
  float max, sumexp, target_logit, sumx;
};

__device__ __forceinline__ void online_combine(float& m, float& s, float m2, float s2) {
  const float nm = fmaxf(m, m2);
  if (nm == -INFINITY) return;  // both sides empty
  s = s * __expf(m - nm) + s2 * __expf(m2 - nm);
  m = nm;
}

// Sums relative to the (base 2) maxima of 2 FROM lanes, joined: the maximum first, so each lane takes one exponential and not two per step.
template <int FROM>
__device__ __forceinline__ void join_sums2(float& m, float& s) {
  float top = m;
#pragma unroll
  for (int o = FROM; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
  s *= fast_exp2(m - (top == -INFINITY ? 0.f : top));        // nothing but empty sums: zero, as they are
#pragma unroll
  for (int o = FROM; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  m = top;
}

struct StatPeers {      // vocabulary-parallel exchange: every rank's [slices][rows] statistics table (peer-addressable)
  unsigned long long p[8];
  int world, slice, rows;
};

// stats[row] = (max, sum exp(x - max), x[target] if the target is in this slice else 0, sum x).
// With `peers.world > 0` the four numbers are also stored into slot [slice][row] of every rank's table (16-byte peer
// stores over NVLink): the exchange of the vocabulary-parallel loss happens inside this kernel instead of a library
// all-gather (reference call site: src/distributed/tensor_parallel.zig:77-129 gather, then consume).
__global__ void __launch_bounds__(XENT_THREADS) xent_stats_kernel(const __nv_bfloat16* __restrict__ logits, long long ld,
                                                                  const long long* __restrict__ targets, RowStat* __restrict__ stats,
                                                                  int V, int vocab_lo, int vocab_total, unsigned int* status,
                                                                  const StatPeers peers) {
  __shared__ float sm[3][XENT_THREADS / 32];
  const int row = blockIdx.x;
  const __nv_bfloat16* x = logits + (long long)row * ld;
  const int nvec = V / 8;
  float m = -INFINITY, s = 0.f, sx = 0.f;
  for (int v = threadIdx.x; v < nvec; v += XENT_THREADS) {
    const uint4 q = reinterpret_cast<const uint4*>(x)[v];
    const uint32_t* pq = reinterpret_cast<const uint32_t*>(&q);
    float f[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) { f[2 * j] = bf16_lo(pq[j]); f[2 * j + 1] = bf16_hi(pq[j]); }
    float lm = f[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) lm = fmaxf(lm, f[j]);
    const float nm = fmaxf(m, lm);
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) { acc += __expf(f[j] - nm); sx += f[j]; }
    s = s * __expf(m - nm) + acc;
    m = nm;
  }
  for (int c = nvec * 8 + threadIdx.x; c < V; c += XENT_THREADS) {
    const float f = __bfloat162float(x[c]);
    online_combine(m, s, f, 1.f);
    sx += f;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
    online_combine(m, s, m2, s2);
    sx += __shfl_xor_sync(0xffffffffu, sx, o);
  }
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { sm[0][wid] = m; sm[1][wid] = s; sm[2][wid] = sx; }
  __syncthreads();
  if (threadIdx.x == 0) {
    float M = sm[0][0], S = sm[1][0], SX = sm[2][0];
    for (int i = 1; i < XENT_THREADS / 32; ++i) { online_combine(M, S, sm[0][i], sm[1][i]); SX += sm[2][i]; }
    const long long t = targets[row];
    float tl = 0.f;
    if (t >= vocab_lo && t < vocab_lo + V) tl = __bfloat162float(x[t - vocab_lo]);
    else if (t != -100 && (t < 0 || t >= vocab_total)) atomicOr(status, (unsigned)ELFA_ST_BAD_TARGET);
    const RowStat rs{M, S, tl, SX};
    if (stats) stats[row] = rs;
    for (int i = 0; i < peers.world; ++i) {
      const int r = (peers.slice + i) % peers.world;      // own table first, then the peers, staggered by rank
      reinterpret_cast<RowStat*>(peers.p[r])[(long long)peers.slice * peers.rows + row] = rs;
    }
  }
}

// Combines `nslices` statistics per row (slice k of row r at stats[k * rows + r]) into the loss and
// rewrites the local logits slice as d loss / d logits * grad_scale.
__global__ void __launch_bounds__(XENT_THREADS) xent_grad_kernel(__nv_bfloat16* __restrict__ logits, long long ld,
                                                                 __nv_bfloat16* __restrict__ dlogits, long long ldd,
                                                                 const long long* __restrict__ targets, const RowStat* __restrict__ stats,
                                                                 int nslices, int rows, float* __restrict__ loss_out, int V, int vocab_lo,
                                                                 int vocab_total, float smoothing, const float* __restrict__ grad_scale_ptr,
                                                                 float grad_scale) {
  const int row = blockIdx.x;
  float M = -INFINITY, S = 0.f, TL = 0.f, SX = 0.f;
  for (int k = 0; k < nslices; ++k) {
    const RowStat st = stats[(long long)k * rows + row];
    online_combine(M, S, st.max, st.sumexp);
    TL += st.target_logit;
    SX += st.sumx;
  }
  const float lse = M + __logf(S);
  const long long t = targets[row];
  const bool valid = t >= 0 && t < vocab_total;
  if (threadIdx.x == 0 && loss_out) {
    float loss = 0.f;
    if (valid) loss = -((1.f - smoothing) * (TL - lse) + (smoothing / (float)vocab_total) * (SX - (float)vocab_total * lse));
    loss_out[row] = loss;
  }
  if (!dlogits) return;
  float gs = grad_scale_ptr ? grad_scale * (*grad_scale_ptr) : grad_scale;
  if (!valid) gs = 0.f;
  const float uni = smoothing / (float)vocab_total;
  const __nv_bfloat16* x = logits + (long long)row * ld;
  __nv_bfloat16* dx = dlogits + (long long)row * ldd;
  const int tcol = (int)(t - vocab_lo);  // may be outside [0, V)
  const int nvec = V / 8;
  for (int v = threadIdx.x; v < nvec; v += XENT_THREADS) {
    const uint4 q = reinterpret_cast<const uint4*>(x)[v];
    const uint32_t* pq = reinterpret_cast<const uint32_t*>(&q);
    float f[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) { f[2 * j] = bf16_lo(pq[j]); f[2 * j + 1] = bf16_hi(pq[j]); }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float p = __expf(f[j] - lse) - uni;
      if (v * 8 + j == tcol) p -= (1.f - smoothing);
      f[j] = p * gs;
    }
    reinterpret_cast<uint4*>(dx)[v] = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
  }
  for (int c = nvec * 8 + threadIdx.x; c < V; c += XENT_THREADS) {
    float p = __expf(__bfloat162float(x[c]) - lse) - uni;
    if (c == tcol) p -= (1.f - smoothing);
    dx[c] = __float2bfloat16(p * gs);
  }
}

// Loss and gradient of whole rows in one pass: the row waits in shared memory between the statistics and the gradient (every thread
// copies in and reads back its own 16-byte vectors, so the copies need no barrier), and the logits are read from memory once and written
// once - the two-kernel form reads them twice. At V = 32000 a row takes 64 KB: three rows per SM, one loading while the others
// compute; more than 32768 columns would leave two. 8192 x 32000: 181 us (1.05 GB, 5.8 TB/s; the exponentials alone take 116), with two
// exponentials per step of the joints (40 per thread beside its 125) 203, as two kernels about 300.
constexpr int XENT_ROW_MAX = 8 * 8 * XENT_THREADS;

// The row of xent_row_kernel when its maximum leaves base 2 (|x| log2(e) past the largest float: rows of the type's lowest value, for one; or
// infinite logits): in natural units, everything relative to the maximum.
template <int NT>
__device__ __noinline__ void xent_row_huge(__nv_bfloat16* x, const uint4* xrow, int nvec, int V, bool valid, float tl, int tv, int tj,
                                           float smoothing, float grad_scale, float* loss, float (*red)[NT / 32]) {
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float m = -INFINITY;
  for (int i = threadIdx.x; i < nvec * 8; i += NT) m = fmaxf(m, __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(xrow)[i]));
  m = warp_max(m);
  __syncthreads();
  if (lane == 0) red[0][wid] = m;
  __syncthreads();
  for (int i = 0; i < NT / 32; ++i) m = fmaxf(m, red[0][i]);
  float s = 0.f, sx = 0.f;
  for (int i = threadIdx.x; i < nvec * 8; i += NT) {
    const float f = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(xrow)[i]) - m;
    s += expf(f);
    sx += f / (float)V;                    // the plain sum would overflow
  }
  s = warp_sum(s);
  sx = warp_sum(sx);
  if (lane == 0) { red[1][wid] = s; red[2][wid] = sx; }
  __syncthreads();
  s = sx = 0.f;
  for (int i = 0; i < NT / 32; ++i) { s += red[1][i]; sx += red[2][i]; }
  if (threadIdx.x == 0) {
    float l = (1.f - smoothing) * (tl - m - logf(s));
    if (smoothing != 0.f) l += smoothing * (sx - logf(s));
    *loss = valid ? -l : 0.f;
  }
  const float gs = valid ? grad_scale : 0.f, off = -gs * (smoothing / (float)V), tg = gs * (1.f - smoothing);
  for (int i = threadIdx.x; i < nvec * 8; i += NT) {
    const float f = expf(__bfloat162float(reinterpret_cast<const __nv_bfloat16*>(xrow)[i]) - m) / s * gs + off;
    x[i] = __float2bfloat16(f - (valid && i == tv * 8 + tj ? tg : 0.f));
  }
}

template <int NT>
__global__ void __launch_bounds__(NT, NT < 64 ? 32 : 3 * XENT_THREADS / NT) xent_row_kernel(__nv_bfloat16* __restrict__ logits, long long ld,
                                                                   const long long* __restrict__ targets, float* __restrict__ loss_out, int V,
                                                                   float smoothing, float grad_scale, unsigned int* status) {
  extern __shared__ __align__(16) uint4 xrow[];
  __shared__ float sm[3][NT / 32];
  const int row = blockIdx.x, nvec = V / 8, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __nv_bfloat16* x = logits + (long long)row * ld;
  for (int v = threadIdx.x; v < nvec; v += NT) cp_async16(smem_u32(xrow + v), x + v * 8, true);
  cp_async_commit();
  const long long t = targets[row];
  const float tl = t >= 0 && t < V ? __bfloat162float(x[t]) : 0.f;                 // read before any thread overwrites the row
  cp_async_wait<0>();
  // in base 2 throughout: exp(x - m) = 2^(x log2(e) - m2) is one fused multiply-add and one special-function instruction
  constexpr float L2E = 1.4426950408889634f;
  __nv_bfloat162 mp = __halves2bfloat162(__ushort_as_bfloat16(0xff80), __ushort_as_bfloat16(0xff80));     // -inf
#pragma unroll 2
  for (int v = threadIdx.x; v < nvec; v += NT) {
    const uint4 q = xrow[v];
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&q);
    mp = __hmax2(mp, __hmax2(__hmax2(p[0], p[1]), __hmax2(p[2], p[3])));
  }
  float m2 = fmaxf(__low2float(mp), __high2float(mp)) * L2E, s = 0.f, sx = 0.f;
  const float nm2 = m2 == -INFINITY ? 0.f : -m2;
#pragma unroll 2
  for (int v = threadIdx.x; v < nvec; v += NT) {
    const uint4 q = xrow[v];
    const uint32_t* p = reinterpret_cast<const uint32_t*>(&q);
    float e[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) e[j] = fast_exp2(fmaf(bf16_lo(p[j]), L2E, nm2)) + fast_exp2(fmaf(bf16_hi(p[j]), L2E, nm2));
    s += (e[0] + e[1]) + (e[2] + e[3]);
    if (smoothing != 0.f) {
#pragma unroll
      for (int j = 0; j < 4; ++j) sx += bf16_lo(p[j]) + bf16_hi(p[j]);
    }
  }
  join_sums2<16>(m2, s);
  if (smoothing != 0.f) sx = warp_sum(sx);
  if (lane == 0) { sm[0][wid] = m2; sm[1][wid] = s; sm[2][wid] = sx; }
  __syncthreads();
  // every warp joins the warps' sums for itself, a lane (or several, with the same) per sum
  constexpr int NW = NT / 32;
  float M2 = sm[0][lane & (NW - 1)], S = sm[1][lane & (NW - 1)], SX = 0.f;
  join_sums2<NW / 2>(M2, S);
  if (smoothing != 0.f) {
#pragma unroll
    for (int i = 0; i < NT / 32; ++i) SX += sm[2][i];
  }
  const float ls = log2f(S), lse2 = M2 + ls;
  const bool valid = t >= 0 && t < V;
  if (threadIdx.x == 0 && !valid && t != -100) atomicOr(status, (unsigned)ELFA_ST_BAD_TARGET);
  if (fabsf(M2) == INFINITY) {             // (a thread whose own maximum overflows downwards rightly adds nothing to a larger one)
    xent_row_huge<NT>(x, xrow, nvec, V, valid, tl, valid ? (int)(t >> 3) : -1, (int)(t & 7), smoothing, grad_scale, loss_out + row, sm);
    return;
  }
  if (threadIdx.x == NT - 1) {     // the thread with the fewest vectors
    // the loss in natural units, from the maximum as it is: M2 carries the rounding of M log2(e), and a result in base 2 would be rounded at
    // 1.44 times its size (up to 1.5 times the error against 64 bits). M is a bf16 number, so M2 ln(2) rounds to it.
    constexpr float LN2 = 0.6931471805599453f;
    const float M = __bfloat162float(__float2bfloat16(M2 * LN2)), l = (ls - fmaf(M, L2E, -M2)) * LN2;
    float loss = (1.f - smoothing) * ((tl - M) - l);
    if (smoothing != 0.f) loss += (smoothing / (float)V) * (SX - (float)V * (M + l));
    loss_out[row] = valid ? -loss : 0.f;
  }
  const float gs = valid ? grad_scale : 0.f, off = -gs * (smoothing / (float)V), tg = gs * (1.f - smoothing);
  const int tv = valid ? (int)(t >> 3) : -1, tj = (int)(t & 7);
#pragma unroll 2
  for (int v = threadIdx.x; v < nvec; v += NT) {
    const uint4 q = xrow[v];
    const uint32_t* p = reinterpret_cast<const uint32_t*>(&q);
    float f[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      f[2 * j] = fmaf(fast_exp2(fmaf(bf16_lo(p[j]), L2E, -lse2)), gs, off);
      f[2 * j + 1] = fmaf(fast_exp2(fmaf(bf16_hi(p[j]), L2E, -lse2)), gs, off);
    }
    if (v == tv) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j == tj) f[j] -= tg;
    }
    reinterpret_cast<uint4*>(x)[v] = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
  }
}

template <int NT>
int launch_xent_row(void* logits, long long ld, const long long* targets, float* loss_out, int rows, int V, float smoothing, float grad_scale,
                    unsigned int* st, cudaStream_t s) {
  ELFA_CUDA(cudaFuncSetAttribute(xent_row_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, XENT_ROW_MAX * 2));
  xent_row_kernel<NT><<<rows, NT, V * 2, s>>>(static_cast<__nv_bfloat16*>(logits), ld, targets, loss_out, V, smoothing, grad_scale, st);
  ELFA_CUDA(cudaGetLastError());
  ::elfa::count_launches(1);
  return ELFA_OK;
}

}  // namespace
}  // namespace elfa

using namespace elfa;

// Pass 1. stats: rows * 4 floats (this rank's slice).
ELFA_API int elfa_xent_stats(const void* logits, long long ld, const long long* targets, float* stats, int rows, int V, int vocab_lo,
                             int vocab_total, void* stream) {
  ELFA_REQUIRE(logits && targets && stats && rows > 0 && V > 0, "xent_stats: bad arguments");
  ELFA_REQUIRE(ld % 8 == 0, "xent_stats: row pitch must be a multiple of 8");
  unsigned int* st = status_word();
  ELFA_REQUIRE(st != nullptr, "xent: no status word");
  xent_stats_kernel<<<rows, XENT_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(logits), ld, targets, reinterpret_cast<RowStat*>(stats), V, vocab_lo, vocab_total, st, StatPeers{});
  ELFA_CUDA(cudaGetLastError());
  ::elfa::count_launches(1);
  return ELFA_OK;
}

// Pass 1 of the vocabulary-parallel loss with the exchange inside the kernel: this rank's statistics go to slot [slice] of
// every rank's table (peer_tables: `world` device addresses of [world][rows][4] fp32 tables in peer-addressable memory).
// A barrier over the group (elfa_symm_barrier) must follow before any rank runs pass 2 on its table.
ELFA_API int elfa_xent_stats_push(const void* logits, long long ld, const long long* targets, const unsigned long long* peer_tables,
                                  int slice, int world, int rows, int V, int vocab_lo, int vocab_total, void* stream) {
  ELFA_REQUIRE(logits && targets && peer_tables && rows > 0 && V > 0, "xent_stats_push: bad arguments");
  ELFA_REQUIRE(world >= 1 && world <= 8 && slice >= 0 && slice < world, "xent_stats_push: bad slice / world");
  ELFA_REQUIRE(ld % 8 == 0, "xent_stats_push: row pitch must be a multiple of 8");
  unsigned int* st = status_word();
  ELFA_REQUIRE(st != nullptr, "xent: no status word");
  StatPeers sp{};
  for (int i = 0; i < world; ++i) {
    ELFA_REQUIRE((peer_tables[i] & 15) == 0, "xent_stats_push: tables must be 16-byte aligned");
    sp.p[i] = peer_tables[i];
  }
  sp.world = world; sp.slice = slice; sp.rows = rows;
  xent_stats_kernel<<<rows, XENT_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(logits), ld, targets, nullptr, V, vocab_lo, vocab_total, st, sp);
  ELFA_CUDA(cudaGetLastError());
  ::elfa::count_launches(1);
  return ELFA_OK;
}

// Pass 2. stats: nslices * rows * 4 floats (slice-major). dlogits may alias logits (in place) or be
// null (loss only). loss_out: rows floats (per-token loss) or null. The gradient is multiplied by
// grad_scale and, if grad_scale_ptr is not null, by the device scalar it points to.
ELFA_API int elfa_xent_grad(void* logits, long long ld, void* dlogits, long long ldd, const long long* targets, const float* stats,
                            int nslices, float* loss_out, int rows, int V, int vocab_lo, int vocab_total, float smoothing,
                            const float* grad_scale_ptr, float grad_scale, void* stream) {
  ELFA_REQUIRE(logits && targets && stats && rows > 0 && V > 0 && nslices > 0, "xent_grad: bad arguments");
  ELFA_REQUIRE(ld % 8 == 0 && (!dlogits || ldd % 8 == 0), "xent_grad: row pitch must be a multiple of 8");
  xent_grad_kernel<<<rows, XENT_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<__nv_bfloat16*>(logits), ld, static_cast<__nv_bfloat16*>(dlogits), ldd, targets,
      reinterpret_cast<const RowStat*>(stats), nslices, rows, loss_out, V, vocab_lo, vocab_total, smoothing, grad_scale_ptr, grad_scale);
  ELFA_CUDA(cudaGetLastError());
  ::elfa::count_launches(1);
  return ELFA_OK;
}

// Widest row of elfa_xent_row.
ELFA_API int elfa_xent_row_max(void) { return XENT_ROW_MAX; }

// Both passes in one for whole rows (no vocabulary split): the logits become d loss / d logits * grad_scale in place, loss_out gets the
// per-token loss. V a multiple of 8 and at most elfa_xent_row_max(), rows on 16-byte boundaries.
// Threads per row: what a thread does once (the joints, the logarithm, two barriers) should be little beside its share of the row, and rows in different
// phases should share an SM. 16384 rows, us, 32 / 64 / 128 / 256 / 512 threads: V 256 17 / 20 / 27 / 45 / 89; 1000 27 / 29 / 35 / 51 / 94; 2048 36 / 34 / 45
// / 61 / 101; 4096 55 / 51 / 60 / 78 / 123; 8000 119 / 94 / 95 / 108 / 160; 12000 198 / 143 / 135 / 136 / 183; 16384 305 / 216 / 192 / 167 / 218. 4096 rows:
// 8192 42 / 34 / 34 / 35 / 47; 24000 160 / 114 / 90 / 74 / 80; 32000 266 / 162 / 125 / 98 / 94. Few rows leave the SMs room, and a call takes what one row
// takes: up to two rows to an SM as for a row four times as wide, up to eight twice (16 rows: 1000 5.4 / 4.1 / 4.1 / 4.1 / 4.1, 4096 6.2 / 6.2 / 4.1 / 4.1 /
// 4.1, 8192 10.2 / 6.2 / 6.2 / 5.1 / 5.0; 600 rows: 1000 6.2 / 5.3 / 4.1 / 4.2 / 6.2, 4096 8.2 / 6.2 / 6.2 / 6.2 / 8.2, 8192 12.3 / 8.2 / 8.2 / 8.2 / 10.2).
ELFA_API int elfa_xent_row(void* logits, long long ld, const long long* targets, float* loss_out, int rows, int V, float smoothing,
                           float grad_scale, void* stream) {
  ELFA_REQUIRE(logits && targets && loss_out && rows > 0 && V > 0, "xent_row: bad arguments");
  ELFA_REQUIRE(V % 8 == 0 && ld % 8 == 0 && V <= XENT_ROW_MAX && (reinterpret_cast<uintptr_t>(logits) & 15) == 0,
               "xent_row: V must be a multiple of 8 and at most 32768, rows 16-byte aligned");
  unsigned int* st = status_word();
  ELFA_REQUIRE(st != nullptr, "xent: no status word");
  auto* s = static_cast<cudaStream_t>(stream);
  const int w = rows <= 300 ? 4 * V : (rows <= 1200 ? 2 * V : V);
  if (w <= 1024) return launch_xent_row<32>(logits, ld, targets, loss_out, rows, V, smoothing, grad_scale, st, s);
  if (w <= 4096) return launch_xent_row<64>(logits, ld, targets, loss_out, rows, V, smoothing, grad_scale, st, s);
  if (w <= 8192) return launch_xent_row<128>(logits, ld, targets, loss_out, rows, V, smoothing, grad_scale, st, s);
  if (V <= 24576) return launch_xent_row<256>(logits, ld, targets, loss_out, rows, V, smoothing, grad_scale, st, s);
  return launch_xent_row<512>(logits, ld, targets, loss_out, rows, V, smoothing, grad_scale, st, s);
}
