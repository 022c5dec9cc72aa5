// A decoding step (up to eight rows) of the EFLA family, all layers in one cooperative kernel.
//
// As a chain of launches a step was 14 small kernels per layer, each of which waits for the one ahead, fetches its first operands, and drains: 5 to 6 us
// apiece, whatever the overlap of their starts. Here a layer is five phases with a grid barrier between (1.2 to 1.4 us on 264 CTAs, two per SM), and what is
// small and elementwise - norms, residual sums, activations, PRISM's refinement - is done again by every CTA on the rows that it needs while it copies them to
// shared memory:
//   norm, w_k and w_v, ShortConv | scan, gate logits | w_o | refinement, norm, w_up | activation, w_down, PRISM's state
// Scan and state belong to the CTAs that have no tile of their phase's product, where those are enough for them. A phase's weights do not depend on the
// phases before it: the blocks that fit are copied to shared memory between the arrival at the barrier and the wait, and each CTA asks for its part of the
// next layer's into L2 there. The phases go through one copy of the code, in loops rather than unrolled: a warp that meets straight-line code for the first
// time takes about eight cycles per instruction. Two layers, 1024 wide, B 2: a step 67 us (and 17 for the logits); prompt of 64 tokens and four steps 1131 us
// with the chain, 740 to 770 with this. Wide products and many rows are the chain's (efla_decode_better).
//
// The launch is cooperative, and its CTAs start together: it waits until all of them have room, two to an SM, whatever else runs, where the chain's small
// launches go into what is free. Steps of 4 layers, 1024 wide, B 2, microseconds with chain / this, alone 498 / 334, and beside another stream of the same
// priority, with that stream's passes per second: products of 4096^3 (8900 alone) 1826 / 576, 8732 / 7093; of 8192^3 (1280) 4638 / 1509, 1285 / 755; one
// elementwise pass after the other over 0.5 GB (6170) 6846 / 486, 6128 / 3978; prompts of 4 x 2048 tokens (133 / 170), whose states' kernel holds 64 SMs for
// a millisecond, 556 / 1209, 116 / 142. A kernel that holds 20 SMs for 200 ms keeps a step waiting for 200 ms. Four threads that decode on a stream each:
// 3084 / 2949 steps a second. What a step waits for must not itself wait for the step (a kernel that spins for a peer which needs this step's result). On a
// stream with a part of the SMs the chain is taken.
//
// The softmax family has no such kernel: cached attention and the joint of its slices are two more phases, each about as long as the launch it would
// replace (a layer of the same width, B 4, 512 positions: 35 us in one kernel, 42 as eight launches whose starts overlap, whole calls 3 to 7 % slower).
//
// Arithmetic, orders of sums and roundings are those of the kernels of the layer-by-layer route, piece by piece from the same functions, so the bits are
// the same. The slices of a product are CTAs of a cluster of eight.
//
// reference: src/model/model.zig:415-454 (streaming with carried states), src/eval/evaluator.zig:419-470.
#include "decode.cuh"

#include <string.h>

#include <algorithm>
#include <atomic>

#include "efla_step.cuh"
#include "elementwise.cuh"
#include "elfa_native.h"
#include "gemm_skinny.cuh"
#include "mma_sync.cuh"
#include "norm.cuh"
#include "prism_step.cuh"

namespace elfa {
namespace {

typedef __nv_bfloat16 bf16;

constexpr int CL = 8, NT = 256;                        // CTAs of a cluster, threads of a CTA; two CTAs run on an SM
// Shared memory: the sums of the warps, for at least PART_ROWS rows, which between products are the phases' own scratch; a ring of weight blocks, in
// flight or to be multiplied; the rows of A
constexpr int PITCH = 132;                             // of the sums: [warp][row of A][column]
constexpr int PART_ROWS = 4, BLOCK_ROWS = 128, HALF_BLOCK = BLOCK_ROWS * 128;
constexpr int SHARED = 115712 - 512;                   // half of an SM's, but for what the kernels declare
constexpr int part_bytes(int M) { return 8 * (M > PART_ROWS ? M : PART_ROWS) * PITCH * 4; }
constexpr int EFLA_TOKENS = 8;                         // rows of a call, so tokens of one sequence

// How one product is cut (skinny_plan) and dealt out: `tiles` of one matrix, `total` of all that are multiplied side by side; a cluster takes
// `per` = CL / shares tiles at a time (inv = 256 / shares, rounded up), `used` clusters have one, and it is done after `rounds`.
struct Cut {
  int N, K, tiles, total, shares, ks, narrow, per, inv, used, rounds;
};

struct Team {                                          // a thread's place, and its CTA's
  int tid, warp, lane, g, q;
  int cta, ctas, rank, cluster, clusters;
  int lda, rows;                                       // row pitch of the rows in shared memory; rows that the sums have room for
  bf16* a;
  float* part;
  unsigned char* ring;
  int halves;                                          // half blocks (64 columns) that the ring holds: 4 or 2
  unsigned int *arrived, target, *status;
  int* dead;
};

__device__ __forceinline__ uint4 ld_l2(const void* p) { return __ldcg(reinterpret_cast<const uint4*>(p)); }
// (bar.sync wants a warp's threads at once, and its callers come from loops that some of them leave early)
__device__ __forceinline__ void named_sync(int id, int threads) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// Grid barrier in two halves; all CTAs of a cooperative launch run at once. A wait that runs out is recorded, and none of the later ones waits again:
// the results are lost then, but no index depends on data.
__device__ __forceinline__ void grid_arrive(Team& c) {
  __syncthreads();
  c.target += c.ctas;
  if (c.tid == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(c.arrived) : "memory");
}
__device__ __forceinline__ void grid_wait(const Team& c) {
  if (c.tid == 0 && !*c.dead) {
    const long long t0 = clock64();
    for (;;) {
      unsigned int v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(c.arrived) : "memory");
      if ((int)(v - c.target) >= 0) break;
      if (clock64() - t0 > kWaitCycles) {
        *c.dead = 1;
        atomicOr(c.status, (unsigned)ELFA_ST_FLAG_TIMEOUT);
        break;
      }
    }
  }
  __syncthreads();
}

__device__ __forceinline__ Team make_team(unsigned char* smem, int* dead, int M, int lda, int halves, unsigned int* arrived, unsigned int* status) {
  Team c;
  c.tid = threadIdx.x;
  c.warp = c.tid >> 5;
  c.lane = c.tid & 31;
  c.g = c.lane >> 2;
  c.q = c.lane & 3;
  c.cta = blockIdx.x;
  c.ctas = gridDim.x;
  c.rank = c.cta % CL;
  c.cluster = c.cta / CL;
  c.clusters = c.ctas / CL;
  c.lda = lda;
  c.rows = max(M, PART_ROWS);
  c.part = reinterpret_cast<float*>(smem);
  c.ring = smem + part_bytes(M);
  c.halves = halves;
  c.a = reinterpret_cast<bf16*>(c.ring + halves * HALF_BLOCK);
  c.arrived = arrived;
  c.target = 0;
  c.status = status;
  c.dead = dead;
  if (c.tid == 0) *dead = 0;
  __syncthreads();
  return c;
}

// ------------------------------------------------------------------------------------------------ products
// Weights of a product: the addresses of matrices [K, ld] that lie side by side, each `tiles` tiles wide (two products of the same shape), or, where
// `split`, one product's columns in pieces of ld.
struct Weights {
  const unsigned long long* w;
  int ld;
  bool split;
};
template <int HD>
__device__ __forceinline__ const bf16* column(const Weights& m, const Cut& u, int tile, int col) {
  if (col >= u.N) return nullptr;
  const int i = m.split ? col / HD : tile >= u.tiles;
  return reinterpret_cast<const bf16*>(m.w[i]) + (m.split ? col - i * HD : col);
}

struct Place {
  int tile, n0, share, k0, k1;                         // n0: first column in its matrix; rows k0 .. k1 - 1 of the contraction
  bool on;
};
__device__ __forceinline__ Place place(const Team& c, const Cut& u, int round) {
  const int at = c.rank * u.inv >> 8;                  // c.rank / u.shares
  Place p;
  p.share = c.rank - at * u.shares;
  p.tile = (round * u.per + at) * c.clusters + c.cluster;
  p.on = at < u.per && p.tile < u.total;
  p.n0 = (p.tile >= u.tiles ? p.tile - u.tiles : p.tile) * (u.narrow ? 64 : 128);
  p.k0 = p.share * u.ks;
  p.k1 = min(u.K, p.k0 + u.ks);
  return p;
}
__device__ __forceinline__ int slice_of(const Team& c, const Cut& u) { return (c.rank - (c.rank * u.inv >> 8) * u.shares) * u.ks; }

// Block b of a tile: 128 rows of the contraction, 64 columns each (128 bytes a row, in two halves where the tile is wide), its 16-byte pieces exchanged
// by the row's number so that ldmatrix meets no bank twice. What lies outside becomes zero. Always one group of copies.
__device__ __forceinline__ int stages(const Team& c, const Cut& u) { return u.narrow ? c.halves : c.halves >> 1; }
template <int HD>
__device__ __forceinline__ void load_block(const Team& c, const Cut& u, const Weights& m, const Place& p, int b) {
  const int k = p.k0 + b * BLOCK_ROWS;
  if (p.on && k < p.k1) {
    const int stage = b & (stages(c, u) - 1), ch = c.tid & 7, r0 = c.tid >> 3;
#pragma unroll 1
    for (int h = 0; h < (u.narrow ? 1 : 2); ++h) {
      const bf16* at = column<HD>(m, u, p.tile, p.n0 + h * 64 + ch * 8);
      const int rows = at ? p.k1 - k : 0;
      if (!at) at = reinterpret_cast<const bf16*>(m.w[0]);
      at += (long long)(k + r0) * m.ld;                // (not read past the matrix: see `rows`)
      uint32_t dst = smem_u32(c.ring) + (u.narrow ? stage : 2 * stage + h) * HALF_BLOCK + r0 * 128 + ((ch ^ (r0 & 7)) << 4);
#pragma unroll
      for (int i = 0; i < BLOCK_ROWS / 32; ++i) {
        const bool in = r0 + 32 * i < rows;
        cp_async16(dst + i * 4096, in ? at + (long long)i * 32 * m.ld : reinterpret_cast<const bf16*>(m.w[0]), in);
      }
    }
  }
  cp_async_commit();
}
// as many blocks of the CTA's tile of a round as the ring holds
template <int HD>
__device__ __forceinline__ void load_first(const Team& c, const Cut& u, const Weights& m, int round = 0) {
  const Place p = place(c, u, round);
#pragma unroll 1
  for (int b = 0; b < stages(c, u); ++b) load_block<HD>(c, u, m, p, b);
}
// One thread asks for this CTA's part of n matrices [K, ld] into L2, up to 24 MB of each
__device__ __forceinline__ void ask_l2(const Team& c, const unsigned long long* w, int n, int K, int ld) {
  if (c.tid != 32) return;
  const unsigned int all = (unsigned int)min((long long)K * ld * 2, 24ll << 20), part = (all / c.ctas + 127) / 128 * 128, from = part * c.cta;
  if (from >= all) return;
  const unsigned int bytes = min(part, all - from) & ~15u;
#pragma unroll 1
  for (int i = 0; i < n; ++i)
    if (bytes) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(w[i] + from), "r"(bytes) : "memory");
}

// the warps' parts of M rows (of `rows` that there is room for), added up over those of warp 0
__device__ __forceinline__ void add_warps(float* sum, int rows, int M, int halves, int tid) {
  const int sh = 3 + halves;                           // 16 halves groups of four columns
#pragma unroll 1
  for (int i = tid; i < M << sh; i += 256) {
    const int at = (i >> sh) * PITCH + (i & ((1 << sh) - 1)) * 4;
    float4 s = *reinterpret_cast<const float4*>(sum + at);
#pragma unroll
    for (int w = 1; w < 8; ++w) {
      const float4 v = *reinterpret_cast<const float4*>(sum + w * rows * PITCH + at);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    *reinterpret_cast<float4*>(sum + at) = s;
  }
}
// the sums of `shares` CTAs of the cluster, from rank `first` on, added up in rank order, two columns per thread: put(row, column, values) for the
// `share`-th part of the outputs. All loads of a thread are in flight together: another CTA's shared memory is some 250 cycles away.
template <typename Put>
__device__ __forceinline__ void add_shares(const float* sum, int M, int halves, int first, int share, int shares, int tid, Put put) {
  const int sh = 4 + halves;
#pragma unroll 1
  for (int i = share + tid * shares; i < M << sh; i += 256 * shares) {
    const int m = i >> sh, c = (i & ((1 << sh) - 1)) * 2;
    const uint32_t at = smem_u32(sum + m * PITCH + c);
    float2 x[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) x[r] = ld_cluster_f2(shares > 1 ? map_to_cta(at, first + min(r, shares - 1)) : at);
    float f[2] = {};
#pragma unroll
    for (int r = 0; r < 8; ++r) {                      // (chosen behind the sum: no branches between the loads)
      f[0] = r < shares ? f[0] + x[r].x : f[0];
      f[1] = r < shares ? f[1] + x[r].y : f[1];
    }
    put(m, c, f);
  }
}

// The tiles of a product, its first blocks under way. Row m of A from column `koff` on lies at c.a + m * c.lda; outputs: C of the first `tiles` tiles and
// C2 of the others, [M, N]. The order of the sums is that of skinny_nn_kernel: warp w takes rows 16 w .. of every 128, the warps add up in order, then
// the slices; the fragments come out of shared memory by ldmatrix instead of byte permutations, which leaves a third of the instructions.
template <int HD>
__device__ __forceinline__ void product(const Team& c, const Cut& u, const Weights& m, int koff, int M, bf16* C, bf16* C2, bool gelu) {
  const int halves = u.narrow ? 1 : 2, ahead = stages(c, u);
#pragma unroll 1
  for (int round = 0; round < u.rounds; ++round) {
    const Place p = place(c, u, round);
    if (p.on) {
      float acc[8][4];
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[j][x] = 0.f;
      const int row = c.warp * 16 + (c.lane & 7) + (c.lane >> 4) * 8, ch = c.lane >> 3 & 1;
      const bf16* a = c.a + c.g * c.lda - koff + 2 * c.q + c.warp * 16;
#pragma unroll 1
      for (int b = 0; p.k0 + b * BLOCK_ROWS < p.k1; ++b) {
        if (ahead == 4) cp_async_wait<3>();
        else if (ahead == 2) cp_async_wait<1>();
        else cp_async_wait<0>();
        __syncthreads();
        const int k = p.k0 + b * BLOCK_ROWS;
        if (k + c.warp * 16 < p.k1) {
          uint32_t x0 = 0, x1 = 0;                     // A[g][2 q ..] and A[g][2 q + 8 ..]; K is a multiple of 8
          if (c.g < M) {
            x0 = *reinterpret_cast<const uint32_t*>(a + k);
            if (k + c.warp * 16 + 8 < p.k1) x1 = *reinterpret_cast<const uint32_t*>(a + k + 8);
          }
          const uint32_t src = smem_u32(c.ring) + (b & (ahead - 1)) * halves * HALF_BLOCK + row * 128;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (h == halves) break;
#pragma unroll
            for (int j = 0; j < 4; ++j) {              // 16 columns: fragment rows g and g + 8
              uint32_t f[4];
              ldsm4_t(f, src + h * HALF_BLOCK + (((2 * j + ch) ^ (row & 7)) << 4));
              mma_bf16(acc[4 * h + j], f, x0, x1);
            }
          }
        }
        if (p.k0 + (b + ahead) * BLOCK_ROWS < p.k1) {
          __syncthreads();
          load_block<HD>(c, u, m, p, b + ahead);
        } else {
          cp_async_commit();
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (h == halves) break;
        float* dst = c.part + (c.warp * c.rows + 2 * c.q) * PITCH + h * 64 + c.g;
        if (2 * c.q < c.rows) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            dst[16 * j] = acc[4 * h + j][0];
            dst[16 * j + 8] = acc[4 * h + j][2];
            if (2 * c.q + 1 < c.rows) {
              dst[16 * j + PITCH] = acc[4 * h + j][1];
              dst[16 * j + 8 + PITCH] = acc[4 * h + j][3];
            }
          }
        }
      }
    }
    __syncthreads();
    if (round + 1 < u.rounds) load_first<HD>(c, u, m, round + 1);
    if (p.on) add_warps(c.part, c.rows, M, halves, c.tid);
    if (u.shares > 1) cluster_sync_all();
    else __syncthreads();
    if (p.on) {
      bf16* out = p.tile >= u.tiles ? C2 : C;
      add_shares(c.part, M, halves, c.rank - p.share, p.share, u.shares, c.tid, [&](int row, int col, float (&f)[2]) {
        if (gelu) {
          f[0] = gelu_tanh(f[0]);
          f[1] = gelu_tanh(f[1]);
        }
        if (p.n0 + col < u.N) *reinterpret_cast<uint32_t*>(out + (long long)row * u.N + p.n0 + col) = pack_bf16(f[0], f[1]);
      });
    }
    if (round + 1 < u.rounds) {
      if (u.shares > 1) cluster_sync_all();
      else __syncthreads();
    }
  }
}
// Other work beside a product, `items` equal pieces: it belongs to the CTAs of the clusters that have no tile, where those take no more rounds than all CTAs
// would, and otherwise to all of them, ahead of the product, those without a tile first. Two layers, eight rows, us, all on the CTAs without a tile / so:
// 2048 wide, 16 heads of 128, w_down leaves eight CTAs for 128 states, 450 / 245; 1024 wide, 8 heads of 128, no PRISM, no product beside the scan, 147 / 95.
// (-> the CTA has a part; its number and how many there are)
__device__ __forceinline__ bool side_work(const Team& c, const Cut& u, int items, int& at, int& n) {
  const int free = c.ctas - u.used * CL;
  n = free > 0 && (items + free - 1) / free <= (items + c.ctas - 1) / c.ctas ? free : c.ctas;
  at = c.cta - u.used * CL;
  if (at < 0) at += c.ctas;
  return at < n;
}

// ------------------------------------------------------------------------------------------------ rows
// Threads are dealt out evenly to the rows, a power of two each: f(row, i) for the vectors i < n of every row
template <typename F>
__device__ __forceinline__ void each_vector(const Team& c, int M, int n, F f) {
  const int sh = M > 4 ? 5 : (M > 2 ? 6 : (M > 1 ? 7 : 8)), row = c.tid >> sh;
  if (row < M)
#pragma unroll 2
    for (int i = c.tid & ((1 << sh) - 1); i < n; i += 1 << sh) f(row, i);
}
// the rows in shared memory normalised in place; TPR threads of a row as elfa_norm_fwd takes them. Loops, not straight-line code: nothing here is in
// the instruction caches when a phase gets to it.
template <int TPR>
__device__ __forceinline__ void norm_in_place(const Team& c, int M, int D, const bf16* w, const bf16* b, float eps, bool rms, float (*red)[NT / 32]) {
#pragma unroll 1
  for (int r0 = 0; r0 < M; r0 += NT / TPR) {
    const int t = c.tid % TPR, row = r0 + c.tid / TPR, nvec = row < M ? D / 8 : 0;
    uint4* xr = reinterpret_cast<uint4*>(c.a + row * c.lda);
    float s1 = 0.f, s2 = 0.f, mean, rstd;
#pragma unroll 1
    for (int i = t; i < nvec; i += TPR) norm_sums(xr[i], s1, s2);
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if (TPR > 32) {
      if (r0) __syncthreads();                         // the sums of the rows before have been read
      if (c.lane == 0) {
        red[0][c.warp] = s1;
        red[1][c.warp] = s2;
      }
      __syncthreads();
      s1 = s2 = 0.f;
#pragma unroll
      for (int i = 0; i < TPR / 32; ++i) {
        s1 += red[0][c.tid / TPR * (TPR / 32) + i];
        s2 += red[1][c.tid / TPR * (TPR / 32) + i];
      }
    }
    if (rms) norm_moments<true>(s1, s2, D, eps, mean, rstd);
    else norm_moments<false>(s1, s2, D, eps, mean, rstd);
#pragma unroll 1
    for (int i = t; i < nvec; i += TPR)
      xr[i] = norm_scale(xr[i], mean, rstd, *(reinterpret_cast<const uint4*>(w) + i), b ? *(reinterpret_cast<const uint4*>(b) + i) : make_uint4(0, 0, 0, 0));
  }
}
// Rows of D values, load(row, vector) each, normalised into shared memory; CTA 0 leaves what was loaded at `keep`. The weights are on their way while the
// rows are put together.
template <typename Load>
__device__ __forceinline__ void norm_rows(const Team& c, int M, int D, const bf16* w, const bf16* b, float eps, int kind, bf16* keep, Load load) {
  __shared__ float red[2][NT / 32];
  const bool rms = kind == 1;
  if (rms) b = nullptr;
  if (c.tid * 64 < D) {                                // a line per thread
    asm volatile("prefetch.global.L1 [%0];" ::"l"(w + c.tid * 64));
    if (b) asm volatile("prefetch.global.L1 [%0];" ::"l"(b + c.tid * 64));
  }
  each_vector(c, M, D / 8, [&](int r, int vi) {
    const uint4 x = load(r, vi);
    *reinterpret_cast<uint4*>(c.a + r * c.lda + vi * 8) = x;
    if (c.cta == 0) *reinterpret_cast<uint4*>(keep + (long long)r * D + vi * 8) = x;
  });
  __syncthreads();
  if (D <= 2048) norm_in_place<32>(c, M, D, w, b, eps, rms, red);
  else norm_in_place<64>(c, M, D, w, b, eps, rms, red);
  __syncthreads();
}
// columns k0 .. of the rows of src [M, K]
__device__ __forceinline__ void put_slice(const Team& c, int M, const Cut& u, const bf16* src) {
  const int k0 = slice_of(c, u), nvec = (min(u.K, k0 + u.ks) - k0) / 8;
  each_vector(c, M, nvec, [&](int row, int vi) {
    *reinterpret_cast<uint4*>(c.a + row * c.lda + vi * 8) = ld_l2(src + (long long)row * u.K + k0 + vi * 8);
  });
  __syncthreads();
}
__device__ __forceinline__ float activate(int act, float x) {
  switch (act) {
    case OP_SILU: return apply<OP_SILU>(x, 0.f, 1.f);
    case OP_RELU: return apply<OP_RELU>(x, 0.f, 1.f);
    case OP_GELU_ERF: return apply<OP_GELU_ERF>(x, 0.f, 1.f);
    default: return x;
  }
}
// the same of the MLP's activation, from h as the up-projection left it (GELU is in it already)
__device__ __forceinline__ void put_activation(const Team& c, int M, const Cut& u, const bf16* h, int act) {
  if (act == ACT_GELU) {
    put_slice(c, M, u, h);
    return;
  }
  const int k0 = slice_of(c, u), nvec = (min(u.K, k0 + u.ks) - k0) / 8;
  each_vector(c, M, nvec, [&](int row, int vi) {
    const uint4 hq = ld_l2(h + (long long)row * u.K + k0 + vi * 8);
    const uint32_t* ph = reinterpret_cast<const uint32_t*>(&hq);
    uint4 o;
    uint32_t* po = reinterpret_cast<uint32_t*>(&o);
#pragma unroll 1
    for (int j = 0; j < 4; ++j) po[j] = pack_bf16(activate(act, bf16_lo(ph[j])), activate(act, bf16_hi(ph[j])));
    *reinterpret_cast<uint4*>(c.a + row * c.lda + vi * 8) = o;
  });
  __syncthreads();
}

// ------------------------------------------------------------------------------------------------ EFLA
constexpr int EFLA_LAYERS = 8;

struct EflaLayerArgs {                                 // as in the list of elfa_efla_stream, the gates' 3 L weights at the end
  const bf16 *n1w, *n1b, *wk, *wv, *wo;
  const float* beta;
  const bf16 *cw, *cb, *n2w, *n2b, *up, *down;
  const float* s0;
  float* s1;
  const float* p0;
  float* p1;
  const bf16* tail;
  long long tail_stride;
  bf16* xin;
  unsigned long long gate[3 * PRISM_MAX_L];
};
struct EflaDecode {
  EflaLayerArgs layer[EFLA_LAYERS];
  EflaWork w;
  const long long* ids;
  const bf16 *tok, *nw, *nb;
  unsigned int *arrived, *status;
  Cut cut[5];                                          // w_k and w_v, gates, w_o, up, down
  int layers, B, T, D, H, V, L, W, tails, act, kind, prism, ring, lda, halves, cur;
  float eps, forget[EFLA_LAYERS];
};
static_assert(sizeof(EflaDecode) <= 4096, "kernel parameters");

// eight channels of the refined output of a row: prism_gated_fwd_kernel
__device__ __forceinline__ uint4 refined(const bf16* u, const bf16* v, const bf16* z, long long at, long long zat, int d, int L) {
  const uint4 uq = ld_l2(u + at), vq = ld_l2(v + at);
  const uint32_t *pu = reinterpret_cast<const uint32_t*>(&uq), *pv = reinterpret_cast<const uint32_t*>(&vq);
  float res[8], add[8];
#pragma unroll
  for (int x = 0; x < 8; ++x) {
    res[x] = (x & 1 ? bf16_hi(pv[x / 2]) - bf16_hi(pu[x / 2]) : bf16_lo(pv[x / 2]) - bf16_lo(pu[x / 2]));
    add[x] = 0.f;
  }
#pragma unroll 1
  for (int l = 0; l < L; ++l) {
    const uint4 zq = ld_l2(z + zat + (long long)l * d);
    const uint32_t* pz = reinterpret_cast<const uint32_t*>(&zq);
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const float delta = prism_delta(prism_sigmoid(x & 1 ? bf16_hi(pz[x / 2]) : bf16_lo(pz[x / 2])), res[x]);
      res[x] -= delta;
      add[x] += delta;
    }
  }
  uint4 o;
  uint32_t* po = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
  for (int j = 0; j < 4; ++j) po[j] = pack_bf16(bf16_lo(pu[j]) + add[2 * j], bf16_hi(pu[j]) + add[2 * j + 1]);
  return o;
}

template <int HD>
__global__ void __launch_bounds__(NT, 2) efla_decode_kernel(const __grid_constant__ EflaDecode p) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int dead;
  const int M = p.B * p.T, D = p.D, G = D / HD, ldz = 3 * p.L * HD;
  Team c = make_team(smem, &dead, M, p.lda, p.halves, p.arrived, p.status);
  int cur = p.cur;
  bool pending = p.ids == nullptr;
  const auto sum = [&](int row, int vi) {              // r + f
    const long long at = (long long)row * D + vi * 8;
    return norm_add(ld_l2(p.w.r + at), ld_l2(p.w.f + at));
  };
  const auto first = [&](int row, int vi) {
    const long long id = p.ids[row];
    const bool in = id >= 0 && id < p.V;
    if (!in && vi == 0 && c.cta == 0) atomicOr(p.status, (unsigned)ELFA_ST_BAD_TARGET);
    return in ? __ldg(reinterpret_cast<const uint4*>(p.tok + id * D) + vi) : make_uint4(0, 0, 0, 0);
  };
  const auto rows = [&](const bf16* nw, const bf16* nb) {
    if (pending) cur ^= 1;
    const bool add = pending;
    pending = true;
    norm_rows(c, M, D, nw, nb, p.eps, p.kind, p.w.x[cur], [&](int row, int vi) { return add ? sum(row, vi) : first(row, vi); });
  };
  const auto weights = [&](int l, int ph) {
    const EflaLayerArgs& y = p.layer[l];
    const unsigned long long* w = ph == 1 ? y.gate : reinterpret_cast<const unsigned long long*>(ph == 0 ? &y.wk : (ph == 2 ? &y.wo : (ph == 3 ? &y.up : &y.down)));
    return Weights{w, ph == 1 ? HD : p.cut[ph].N, ph == 1};
  };
  const auto ask = [&](int l, int ph) {
    const Weights m = weights(l, ph);
    if (ph != 1 || p.prism) ask_l2(c, m.w, ph == 0 ? 2 : (ph == 1 ? 3 * p.L : 1), p.cut[ph].K, m.ld);
  };
  load_first<HD>(c, p.cut[0], weights(0, 0));
  for (int ph = 0; ph < 5; ++ph) ask(0, ph);
#pragma unroll 1
  for (int i = 0, l = 0, ph = 0; l < p.layers; ++i) {
    const EflaLayerArgs& y = p.layer[l];
    const Cut& u = p.cut[ph];
    const bool multiply = ph != 1 || p.prism;
    int at, n;                                         // the CTAs of what goes on beside a product
    if (ph == 1 && side_work(c, u, (p.B * p.H * (HD / 32) + 1) / 2, at, n)) {           // the scan, beside the gates' logits: 128 threads per 32 columns of a head
      typedef EflaStepScratch<HD, EFLA_TOKENS> Scratch;
      static_assert(2 * sizeof(Scratch) <= part_bytes(1), "scratch of the scan");
      const int group = c.tid / 128;
      Scratch& sm = reinterpret_cast<Scratch*>(c.part)[group];
#pragma unroll 1
      for (int j = at + group * n; j < p.B * p.H * (HD / 32); j += 2 * n) {
        efla_scan_block<HD, EFLA_TOKENS>(p.w.k, p.w.v, y.beta, y.s0, p.w.o, y.s1, p.T, p.H, j / (HD / 32), j % (HD / 32), sm, c.tid % 128,
                                         [&] { named_sync(3 + group, 128); });
        named_sync(3 + group, 128);
      }
      __syncthreads();
    }
    if (ph == 4 && p.prism && side_work(c, u, p.B * G, at, n)) {
      // PRISM's state, which nothing of this call reads: a CTA per (batch, group), 64 rows at a time
      const PrismTile<HD> sm(c.part, p.T, p.L);
      const PrismSource in{p.w.u, p.w.e, p.w.z, ldz, p.L * HD, 2 * p.L * HD, p.T, G, p.L};
      const int part = c.tid & 3;
#pragma unroll 1
      for (int bg = at; bg < p.B * G; bg += n) {
        float S[HD / 4];                               // the first rows are on their way while keys and deltas are formed
        int row = c.tid >> 2;
        if (row < HD) prism_state_load<HD>(S, y.p0 + ((long long)bg * HD + row) * HD, part);
        prism_state_prepare<HD, NT, 1, 1>(in, sm, bg, 0, p.T, c.tid, [] { __syncthreads(); });
#pragma unroll 1
        for (; row < HD; row += NT / 4) {
          if (row >= NT / 4) prism_state_load<HD>(S, y.p0 + ((long long)bg * HD + row) * HD, part);
          prism_state_rows<HD>(S, sm, p.T, p.L, row, part, p.forget[l]);
          prism_state_store<HD>(S, y.p1 + ((long long)bg * HD + row) * HD, part);
        }
        __syncthreads();
      }
    }
    if (ph == 0) {
      rows(y.n1w, y.n1b);
      if (p.prism)                                     // ShortConv: every CTA a few pairs of channels
#pragma unroll 1
        for (int j = c.cta + (NT - 1 - c.tid) * c.ctas; j < M * (D / 2); j += NT * c.ctas) {
          const int row = j / (D / 2), ch = j % (D / 2) * 2, t = row % p.T, b = row / p.T;
          const bf16* tb = y.tail + b * y.tail_stride + ch;
          const auto at = [&](int k) {
            return *reinterpret_cast<const uint32_t*>(k < p.tails ? tb + (long long)k * D : c.a + (b * p.T + k - p.tails) * c.lda + ch);
          };
          bf16 *xb = y.xin + (long long)b * (p.tails + p.T) * D + ch, *o = p.w.u + (long long)row * D + ch;      // (the tail is copied below)
          if (p.ring) shortconv_stream_pair<true, false>(at, y.cw, y.cb, xb, o, p.tails, t, ch, D, p.W);
          else shortconv_stream_pair<false, false>(at, y.cw, y.cb, xb, o, p.tails, t, ch, D, p.W);
        }
    } else if (ph == 3) {
      norm_rows(c, M, D, y.n2w, y.n2b, p.eps, p.kind, p.w.r, [&](int row, int vi) {    // r = q + x
        const long long at = (long long)row * D + vi * 8;
        const uint4 o = p.prism ? refined(p.w.u, p.w.e, p.w.z, at, (long long)row * ldz + vi * 8 % HD, HD, p.L) : ld_l2(p.w.e + at);
        return norm_add(o, ld_l2(p.w.x[cur] + at));
      });
    } else if (ph == 4) {
      if (c.cluster < u.used) put_activation(c, M, u, p.w.h, p.act);
    } else if (multiply && c.cluster < u.used) {
      put_slice(c, M, u, ph == 1 ? p.w.u : p.w.o);
    }
    if (multiply)
      product<HD>(c, u, weights(l, ph), ph == 0 || ph == 3 ? 0 : slice_of(c, u), M,
                  ph == 0 ? p.w.k : (ph == 1 ? p.w.z : (ph == 2 ? p.w.e : (ph == 3 ? p.w.h : p.w.f))), p.w.v,
                  ph == 3 && p.act == ACT_GELU);
    const int asked = ph, done = l;
    if (++ph == 5) {
      ph = 0;
      if (++l == p.layers) break;
    }
    grid_arrive(c);
    if (ph != 1 || p.prism) load_first<HD>(c, p.cut[ph], weights(l, ph));
    if (done + 1 < p.layers) ask(done + 1, asked);
    if (asked == 0 && p.prism) {                       // the tail goes to the next call's source as it is
      const int half = D / 2, n = p.tails * half;
#pragma unroll 1
      for (int b = 0; b < p.B; ++b)
#pragma unroll 2
        for (int j = c.cta * NT + c.tid; j < n; j += c.ctas * NT)
          reinterpret_cast<uint32_t*>(y.xin + (long long)b * (p.tails + p.T) * D)[j] = reinterpret_cast<const uint32_t*>(y.tail + b * y.tail_stride)[j];
    }
    grid_wait(c);
  }
  cluster_sync_all();                                  // nobody leaves while its sums are being read
  if (!p.nw) return;
  grid_arrive(c);
  pdl_next();
  if (c.cta) return;
  grid_wait(c);
  rows(p.nw, p.nb);
#pragma unroll 1
  for (int i = c.tid; i < M * (D / 8); i += NT)
    *reinterpret_cast<uint4*>(p.w.n + i * 8) = *reinterpret_cast<const uint4*>(c.a + i / (D / 8) * c.lda + i % (D / 8) * 8);
}

// ------------------------------------------------------------------------------------------------ launches
Cut cut_of(long long N, long long K, int side_by_side = 1) {
  const SkinnyPlan plan = skinny_plan((int)N, (int)K);
  Cut u{};
  u.N = (int)N;
  u.K = (int)K;
  u.tiles = plan.tiles((int)N);
  u.total = side_by_side * u.tiles;
  u.shares = plan.shares;
  u.ks = plan.ks((int)K);
  u.narrow = plan.narrow;
  u.per = CL / u.shares;
  u.inv = (256 + u.shares - 1) / u.shares;
  return u;
}
void deal_out(Cut* cuts, int n, int clusters) {
  for (int i = 0; i < n; ++i) {
    Cut& u = cuts[i];
    u.used = std::min(clusters, u.total);              // a cluster's first tile comes before another one's second
    u.rounds = (u.total + u.per * clusters - 1) / (u.per * clusters);
  }
}
// The product goes by gemm_skinny in the layer-by-layer route too, and its rows fit
bool skinny(int M, long long N, long long K) {
  return N % 8 == 0 && K % 8 == 0 && N < (1 << 24) && K < (1 << 24) && gemm_skinny_better(M, (int)N, (int)K);
}
int pitch_of(int D, const Cut* cuts, int n) {          // rows of shared memory start four banks apart
  int k = D;
  for (int i = 0; i < n; ++i) k = std::max(k, cuts[i].ks);
  return (k + 63) / 64 * 64 + 8;
}
int shared_bytes(int M, int lda, int halves) { return part_bytes(M) + halves * HALF_BLOCK + M * lda * 2; }
int ring_halves(int M, int lda) { return shared_bytes(M, lda, 4) <= SHARED ? 4 : 2; }

// Clusters that run at once with so much shared memory; 0: the kernel cannot be launched this way here. Asked once per device, kernel and size class.
template <auto Kernel>
int room(int bytes) {
  static std::atomic<int> known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev > 63) return 0;
  int v = known[dev].load(std::memory_order_acquire);
  if (v == 0) {
    int coop = 0, most = 0;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(CL);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = SHARED;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CL;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const bool ok = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop &&
                    cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SHARED) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&most, Kernel, &cfg) == cudaSuccess && most > 0;
    if (!ok) cudaGetLastError();
    v = ok ? most : -1;
    known[dev].store(v, std::memory_order_release);
  }
  return v > 0 && bytes <= SHARED ? v : 0;
}
template <auto Kernel, typename P>
int launch(P& p, int bytes, cudaStream_t s) {
  const int clusters = room<Kernel>(bytes);
  ELFA_REQUIRE(clusters > 0, "decode: the kernel does not fit this device");
  deal_out(p.cut, sizeof(p.cut) / sizeof(Cut), clusters);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(clusters * CL);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = SHARED;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CL;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeCooperative;
  at[1].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, Kernel, p);
  if (e == cudaErrorCooperativeLaunchTooLarge) {       // the stream has a part of the SMs only (a green context)
    cudaGetLastError();
    set_last_error("decode: the CTAs do not run at once on this stream");
    return ELFA_ERR_UNSUPPORTED;
  }
  ELFA_CUDA(e);
  ::elfa::count_launches(1);
  return ELFA_OK;
}

void efla_cuts(const EflaDims& m, Cut* cut) {
  cut[0] = cut_of(m.H * m.d, m.D, 2);
  cut[1] = m.prism ? cut_of(3 * m.L * m.d, m.D) : cut[0];
  if (!m.prism) cut[1].total = 0;                      // the scan alone
  cut[2] = cut_of(m.D, m.H * m.d);
  cut[3] = cut_of(m.F, m.D);
  cut[4] = cut_of(m.D, m.F);
}

// Whether a layer takes less time here than as a chain: what the launches cost, against what every CTA does again on the rows (M D values) and the half
// blocks of further rounds of tiles, where the chain's own grids take one. Microseconds, from 736 shapes (256 to 4096 wide, 1 to 8 rows, MLPs 2, 8 / 3
// and 4 times as wide, heads of 64 and 128, with PRISM and without): the slower form is taken at 41 of them, by up to 10 %. Two layers, chain / kernel: 1024 wide,
// MLP 4096, PRISM, B 1 136 / 70, B 8 148 / 102, without PRISM, B 8 90 / 79; 2048 wide, MLP 8192, PRISM, B 1 180 / 127, B 8 197 / 202, without, B 1 122 / 109, B 8
// 138 / 155; 2560 wide, MLP 10240, PRISM, B 4 209 / 238, without, B 8 157 / 260; 4096 wide, MLP 8192, PRISM, B 1 239 / 196, B 4 252 / 286.
bool efla_decode_better(const EflaDims& m, const Cut* cut) {
  int again = 0;
  for (int i = 0; i < 5; ++i)
    if (cut[i].rounds > 1) again += (cut[i].rounds - 1) * ((cut[i].ks + BLOCK_ROWS - 1) / BLOCK_ROWS) * (cut[i].narrow ? 1 : 2);
  return (m.prism ? 28 : 17) > 1.6 * (double)(m.B * m.T * m.D) / 1024 + again;
}

}  // namespace

bool efla_decode_fits(const EflaDims& m) {
  const long long M = m.B * m.T;
  if (M > SKINNY_ROWS || m.D > 4096 || m.D % 8 || (m.d != 32 && m.d != 64 && m.d != 96 && m.d != 128) || (m.prism && m.tail == 0) ||
      m.layers > (long long)EFLA_LAYERS * DECODE_COUNTERS)
    return false;
  if (m.prism && (2 * m.T * m.L * m.d + m.T * m.L) * 4 > part_bytes((int)M)) return false;
  if (!skinny((int)M, m.H * m.d, m.D) || !skinny((int)M, m.D, m.H * m.d) || !skinny((int)M, m.F, m.D) || !skinny((int)M, m.D, m.F) ||
      (m.prism && (!skinny((int)M, 3 * m.L * m.d, m.D) || m.D % m.d || elfa_shortconv_stream_rows((int)m.B, (int)m.tail, (int)m.T, (int)m.D, (int)m.W))))
    return false;
  Cut cut[5];
  efla_cuts(m, cut);
  const int lda = pitch_of((int)m.D, cut, 5), bytes = shared_bytes((int)M, lda, ring_halves((int)M, lda));
  const int clusters = m.d == 32 ? room<efla_decode_kernel<32>>(bytes)
                                 : (m.d == 64 ? room<efla_decode_kernel<64>>(bytes)
                                              : (m.d == 96 ? room<efla_decode_kernel<96>>(bytes) : room<efla_decode_kernel<128>>(bytes)));
  if (clusters <= 0) return false;
  deal_out(cut, 5, clusters);
  return efla_decode_better(m, cut);
}

int efla_decode(const unsigned long long* p, const EflaDims& m, const EflaWork& w, const float* forget, float eps, cudaStream_t s) {
  EflaDecode a{};
  efla_cuts(m, a.cut);
  a.w = w;
  a.tok = reinterpret_cast<const bf16*>(p[1]);
  a.B = (int)m.B;
  a.T = (int)m.T;
  a.D = (int)m.D;
  a.H = (int)m.H;
  a.V = (int)m.V;
  a.L = (int)m.L;
  a.W = (int)m.W;
  a.tails = (int)m.tail;
  a.act = (int)m.act;
  a.kind = (int)m.kind;
  a.prism = (int)m.prism;
  a.ring = m.W == 4 || m.W == 8 || m.W == 16;
  a.lda = pitch_of(a.D, a.cut, 5);
  a.eps = eps;
  a.status = status_word();
  ELFA_REQUIRE(a.status != nullptr, "decode: no status word");
  a.halves = ring_halves((int)(m.B * m.T), a.lda);
  const int bytes = shared_bytes((int)(m.B * m.T), a.lda, a.halves), per = 19 + 3 * (int)m.L;
  ELFA_CUDA(cudaMemsetAsync(w.arrived, 0, DECODE_COUNTERS * 4, s));
  for (int l = 0, n = 0; l < m.layers; l += EFLA_LAYERS, ++n) {
    a.layers = std::min((int)m.layers - l, EFLA_LAYERS);
    for (int i = 0; i < a.layers; ++i) {
      memcpy(&a.layer[i], p + 7 + per * (l + i), per * sizeof(*p));
      a.forget[i] = forget[l + i];
    }
    a.ids = l == 0 ? reinterpret_cast<const long long*>(p[0]) : nullptr;
    const bool last = l + a.layers == m.layers;
    a.nw = last ? reinterpret_cast<const bf16*>(p[2]) : nullptr;
    a.nb = last ? reinterpret_cast<const bf16*>(p[3]) : nullptr;
    a.arrived = w.arrived + n;
    const int rc = m.d == 32 ? launch<efla_decode_kernel<32>>(a, bytes, s)
                             : (m.d == 64 ? launch<efla_decode_kernel<64>>(a, bytes, s)
                                          : (m.d == 96 ? launch<efla_decode_kernel<96>>(a, bytes, s) : launch<efla_decode_kernel<128>>(a, bytes, s)));
    if (rc != ELFA_OK) return rc;
    a.cur ^= (a.layers - (l == 0)) & 1;                // a sum per layer, but for the first rows
  }
  return ELFA_OK;
}

}  // namespace elfa
