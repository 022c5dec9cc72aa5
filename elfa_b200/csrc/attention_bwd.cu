// Attention backward on tcgen05, recompute style: only O and the row log-sum-exp are kept by
// forward; the probabilities are rebuilt per [128 x 128] block of (query, key) pairs.
//
//   delta = rowsum(dO * O)                                    (small pre-pass)
//   MODE_DKV (CTA owns a key tile, loops over query tiles), everything transposed so that the key
//   index runs along the tensor-memory lanes:
//       S^T = K Q^T, dP^T = V dO^T                                 (tensor memory, fp32)
//       P^T = exp(S^T*scale - lse[q]), dS^T = P^T * (dP^T - delta[q]) * scale  -> bf16, written back
//       into tensor memory over the fp32 values they were computed from
//       dV += P^T dO,  dK += dS^T Q                                 (A operand read from tensor memory)
//   MODE_DQ  (CTA owns a query tile, loops over key tiles):
//       S = Q K^T, dP = dO V^T;  dS -> bf16 in tensor memory;  dQ += dS K
// P / dS never touch shared memory; the Q / K / V / dO tiles are used K-major or MN-major through
// the descriptor only, so no transpose is materialised. Two passes keep every accumulator in tensor
// memory and make the result deterministic (no floating-point atomics on dQ).
//
// S 4096, 32 heads of 128, causal: 260 + 192 us and 15 us of row sums. A block pair takes 3250 / 2400 cycles of an SM (at the 1.42 GHz that it
// runs at under this load) for 2048 / 1536 cycles of products: the key-tile pass waits on the chain S -> P -> dV -> next S (tensor memory is full: S, dP and two accumulators, so S has one
// place), the query-tile pass on shared memory (S and dP read 16 KB per 64 cycles of product, and 64 KB arrive per pair). The
// resident operands in tensor memory instead were slower (212 against 192 us).
//
// reference: the op is defined by src/futhark/attention.fut:28-51; the reference ships no
// attention backward at all.
//
// Roles per CTA: warp 0 TMA, warp 1 MMA issue, warp 2 row vectors (key-tile pass), the rest compute: the four (key-tile pass) or two warps with
// the same number modulo 4 share a tensor-memory lane quarter and split the columns.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "elfa_native.h"

namespace elfa {

int make_qkv_tmap(CUtensorMap* tm, const void* qkv, int S, int B, int H, int hd, long long stride_s, long long stride_b,
                  int planes, uint32_t box_rows);

namespace {

constexpr int SUBB = 128 * 128;
// Compute warps per tensor-memory lane quarter, each on its own columns of a block, and the pieces in which they hand P and dS to the MMA warp.
// Key-tile pass: its chain is P -> dV -> next S, so four warps (a quarter more of the exponentials' rate than two) and halves, of
// which the first is multiplied while the second is made (260 us against 268 with two warps, 279 without halves; S 4096, 32 heads of 128). Query-tile
// pass: next S waits for nothing but the read of this one; two warps, whole (192 us; four warps 200).
template <bool DKV> struct BwdWarps {
  static constexpr int SPLIT = DKV ? 4 : 2, PIECES = DKV ? 2 : 1;
  static constexpr int CW = 128 / SPLIT;                // columns of a compute warp
  static constexpr int HC = CW / PIECES;                // columns of a piece
  static constexpr int COMPUTE = 4 * SPLIT;             // compute warps
  static constexpr int THREADS = 32 * (3 + COMPUTE);
};

// Grouped-query attention (Hkv < H): the key-tile pass runs `nsplit` CTAs (a cluster) per key / value head, each walking the query
// tiles of its share of the group's query heads one head after the other; the shares are added up in rank order, so dK / dV are summed in a
// fixed order. The query-tile pass reads the group's key head. Packed sequences (doc_start, see the forward kernel): masked like the causal
// diagonal, block pairs without a visible (query, key) pair are skipped.
struct AttnBwdParams {
  int S, B, H, hd;
  int Hkv;
  int nsplit;             // key-tile pass: CTAs (of one cluster) that share the query heads of a key head
  const int* doc_start;   // [B, S] or null
  const float* lse;    // [B, H, S] natural log
  const float* delta;  // [B, H, S]
  __nv_bfloat16* dqkv;
  long long d_stride_s, d_stride_b;
  float scale, scale_log2;
  int causal;
  int n_tiles;
  unsigned int* status;
};

// P and dS are handed over in up to two pieces: BB_P, BB_DS and the one behind each
enum { BB_RES0 = 0, BB_RES1, BB_QF0, BB_QE0 = BB_QF0 + 3, BB_OF0 = BB_QE0 + 3, BB_OE0 = BB_OF0 + 2, BB_VF0 = BB_OE0 + 2, BB_S = BB_VF0 + 2,
       BB_DP, BB_P, BB_DS = BB_P + 2, BB_ACC = BB_DS + 2, BB_COUNT };

template <int HDP, bool DKV>
struct BwdSmem {
  static constexpr int NSUB = HDP / 64;
  static constexpr int TILE = NSUB * SUBB;
  // rings of the inner tiles: one slot more for the operand that two products far apart read (Q, or K in the query-tile pass)
  static constexpr int NQ = 3, NO = 2;
  static constexpr int RES0 = 0;
  static constexpr int RES1 = RES0 + TILE;
  static constexpr int INQ = RES1 + TILE;
  static constexpr int INO = INQ + NQ * TILE;
  static constexpr int VEC = 2 * 128 * 4 + 128;            // -lse2, -delta * scale (fp32), document start relative to the key tile (bytes)
  static constexpr int VEC_OFF = INO + NO * TILE;          // [2 slots]
  static constexpr int BAR_OFF = VEC_OFF + 2 * VEC;
  static constexpr int TOTAL = BAR_OFF + BB_COUNT * 8 + 16;
  static constexpr int RED_LD = 2 * HDP + 4;               // fp32 pitch of the accumulators handed to the cluster, over the rings
  static_assert(!DKV || 128 * RED_LD * 4 <= (NQ + NO) * TILE, "accumulators fit the rings");
  static_assert(TOTAL <= 232448, "shared memory of a CTA");
};

// delta[b,h,s] = sum_d dO[s,b,h,d] * O[s,b,h,d]; LPR lanes per (s, b, h), 16 bytes each, so that every lane has work at hd = 8 LPR, and two rows in
// flight per lane. Bound by memory: 131072 rows of 128 (67 MB read) 14.7 us, with one warp per row 32.
template <int LPR>
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                                                         long long o_stride_s, long long o_stride_b, float* __restrict__ delta, int S,
                                                         int B, int H, int hd) {
  constexpr int ROWS = 256 / LPR;            // rows of a block per round
  const int l = threadIdx.x & (LPR - 1);
  const long long total = (long long)S * B * H;
  const long long row0 = (long long)blockIdx.x * (2 * ROWS) + threadIdx.x / LPR;
  float acc[2] = {0.f, 0.f};
  long long at[2];
  uint4 a[2], d[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const long long row = row0 + u * ROWS;
    a[u] = d[u] = make_uint4(0, 0, 0, 0);
    at[u] = -1;
    if (row < total) {
      const int h = (int)(row % H);
      const long long sb = row / H;
      const int b = (int)(sb % B), s = (int)(sb / B);
      at[u] = ((long long)b * H + h) * S + s;
      if (l * 8 < hd) {
        const long long off = (long long)s * o_stride_s + (long long)b * o_stride_b + (long long)h * hd + l * 8;
        a[u] = *reinterpret_cast<const uint4*>(o + off);
        d[u] = *reinterpret_cast<const uint4*>(dout + off);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const uint32_t* pa = reinterpret_cast<const uint32_t*>(&a[u]);
    const uint32_t* pd = reinterpret_cast<const uint32_t*>(&d[u]);
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[u] += bf16_lo(pa[j]) * bf16_lo(pd[j]) + bf16_hi(pa[j]) * bf16_hi(pd[j]);
#pragma unroll
    for (int m = LPR / 2; m > 0; m >>= 1) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], m);
    if (l == 0 && at[u] >= 0) delta[at[u]] = acc[u];
  }
}

// tcgen05.wait::ld that the 32 loaded registers pass through, so that no use of them can be scheduled ahead of it
__device__ __forceinline__ void tmem_ld_wait32(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]),
                 "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]),
                 "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])::"memory");
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// a compute warp's columns of a block
template <int CW>
__device__ __forceinline__ void load_cols(uint32_t taddr, uint32_t (&r)[CW]) {
#pragma unroll
  for (int c = 0; c < CW / 32; ++c) tmem_ld32(taddr + c * 32, reinterpret_cast<uint32_t(&)[32]>(r[c * 32]));
#pragma unroll
  for (int c = 0; c < CW / 32; ++c) tmem_ld_wait32(reinterpret_cast<uint32_t(&)[32]>(r[c * 32]));
}

template <int HDP, bool DKV>
__global__ void __launch_bounds__(BwdWarps<DKV>::THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmDO, const AttnBwdParams p) {
  using L = BwdSmem<HDP, DKV>;
  constexpr int NSUB = L::NSUB, NQ = L::NQ, NO = L::NO, CW = BwdWarps<DKV>::CW, HC = BwdWarps<DKV>::HC, PIECES = BwdWarps<DKV>::PIECES,
                SPLIT = BwdWarps<DKV>::SPLIT, COMPUTE = BwdWarps<DKV>::COMPUTE;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + BB_COUNT);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = smem_u32(bars);
  auto bar = [&](int i) { return bar0 + 8u * i; };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // one-dimensional grid, heaviest outer tile first over the whole grid: every (batch, head) runs its longest tile before any
  // runs its second longest, so the short CTAs fill the tail of the launch
  const int n_heads = DKV ? p.Hkv : p.H;
  const int nsplit = DKV ? p.nsplit : 1;
  const int bid = (int)blockIdx.x / nsplit, share = (int)blockIdx.x % nsplit;
  const int hb = bid % (n_heads * p.B);
  const int rank = bid / (n_heads * p.B);
  const int h = hb % n_heads, b = hb / n_heads;     // DKV: key / value head; DQ: query head
  const int group = p.H / p.Hkv;
  const int kvh = DKV ? h : h / group;
  // outer tile and the inner range it loops over
  const int outer = DKV ? rank : p.n_tiles - 1 - rank;   // heaviest first in both modes
  int in_begin = DKV ? (p.causal ? outer : 0) : 0;
  int in_end = DKV ? p.n_tiles : (p.causal ? outer + 1 : p.n_tiles);
  const int* dstart = p.doc_start ? p.doc_start + (long long)b * p.S : nullptr;
  if (dstart) {
    if (DKV) {      // query tiles whose first row's document starts after this key tile see none of it; 32 tiles asked at once
      int e = in_begin + 1;
      while (e < in_end) {
        const int t = e + lane;
        const unsigned hidden = __ballot_sync(0xffffffffu, t < in_end && dstart[(long long)min(t, in_end - 1) * 128] > outer * 128 + 127);
        if (hidden) {
          in_end = e + __ffs(hidden) - 1;
          break;
        }
        e += 32;
      }
    } else {
      in_begin = dstart[outer * 128] / 128;
    }
  }
  const int n_in = in_end - in_begin;                     // inner tiles per head
  const int heads = DKV ? group / nsplit : 1;             // query heads of this CTA
  const int hq0 = DKV ? kvh * group + share * heads : h;
  const int n_iter = n_in * heads;                        // DKV: every query head of the share in turn

  if (threadIdx.x == 0) {
    prefetch_tmap(&tmQKV);
    prefetch_tmap(&tmDO);
    for (int i = 0; i < BB_COUNT; ++i)      // one arrival per compute warp, or one
      mbar_init(bar(i), i >= BB_P && i < BB_ACC ? COMPUTE : 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_holder), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  // fp32 S (or S^T) and dP (or dP^T); their bf16 successors P / dS overwrite the first half of the columns of the warp they come from
  const uint32_t TM_S = tmem_base, TM_DP = tmem_base + 128, TM_ACC0 = tmem_base + 256, TM_ACC1 = tmem_base + 256 + HDP;

  // resident pair: (K_j, V_j) in DKV mode, (Q_i, dO_i) in DQ mode; the inner pair is the other one
  const uint32_t sRes0 = sbase + L::RES0, sRes1 = sbase + L::RES1;
  auto sQ = [&](int slot) { return sbase + L::INQ + slot * L::TILE; };
  auto sO = [&](int slot) { return sbase + L::INO + slot * L::TILE; };

  if (warp == 0) {
    if (lane == 0) {
      auto load = [&](uint32_t dst, const CUtensorMap* tm, int head, int tile, int bar_id) {
        mbar_expect_tx(bar(bar_id), L::TILE);
        for (int s = 0; s < NSUB; ++s) tma_load_4d(dst + s * SUBB, tm, s * 64, head, b, tile * 128, bar(bar_id));
      };
      auto load_q = [&](int it) {                         // Q, or K in the query-tile pass
        const int hq = hq0 + it / n_in, t = in_begin + it % n_in;
        load(sQ(it % NQ), &tmQKV, DKV ? hq : p.H + kvh, t, BB_QF0 + it % NQ);
      };
      auto load_o = [&](int it) {                         // dO, or V
        const int hq = hq0 + it / n_in, t = in_begin + it % n_in;
        load(sO(it % NO), DKV ? &tmDO : &tmQKV, DKV ? hq : p.H + p.Hkv + kvh, t, BB_OF0 + it % NO);
      };
      load(sRes0, &tmQKV, DKV ? p.H + kvh : h, outer, BB_RES0);
      load_q(0);
      load(sRes1, DKV ? &tmQKV : &tmDO, DKV ? p.H + p.Hkv + kvh : h, outer, BB_RES1);
      load_o(0);
      for (int it = 1; it < NQ; ++it) {                   // NO = NQ - 1
        if (it < n_iter) load_q(it);
        if (it < NO && it < n_iter) load_o(it);
      }
      for (int it = 0; it + NO < n_iter; ++it) {          // slots in the order in which the products give them back
        if (!mbar_wait(bar(BB_OE0 + it % NO), (it / NO) & 1, abort_flag, p.status)) break;
        load_o(it + NO);
        if (it + NQ < n_iter) {
          if (!mbar_wait(bar(BB_QE0 + it % NQ), (it / NQ) & 1, abort_flag, p.status)) break;
          load_q(it + NQ);
        }
      }
    }
  } else if (warp == 1) {
    // MMA issuer: the warp runs converged, one elected lane issues (descriptors stay in uniform registers)
    {
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);
      constexpr uint32_t idesc_acc = make_idesc_bf16(128, HDP, false, true);   // A from tensor memory, B MN-major
      auto wait = [&](int bi, uint32_t ph) { return __all_sync(0xffffffffu, mbar_wait(bar(bi), ph, abort_flag, p.status)) != 0; };
      // Issue order per iteration: [dV(it)] S(it+1) | dK or dQ (it) dP(it+1). The products of the next inner tile are
      // queued as soon as the tensor-memory columns they overwrite have been consumed (S after the probabilities were
      // read, dP after dS was multiplied), so the exponentials of tile it+1 overlap the accumulator MMAs of tile it.
      // DKV: S^T = K Q^T, dP^T = V dO^T (A = resident);  DQ: S = Q K^T, dP = dO V^T (A = resident)
      auto issue_s = [&](int it) {
        const uint32_t a0 = sRes0, b0 = sQ(it % NQ);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < HDP / 16; ++kk) {
            const uint32_t off = (kk / 4) * SUBB + (kk % 4) * 32;
            tc_mma_f16(TM_S, make_smem_desc(a0 + off, 16, 1024, 2), make_smem_desc(b0 + off, 16, 1024, 2), idesc_s, kk != 0);
          }
          tc_commit(bar(BB_S));
        }
        __syncwarp();
      };
      auto issue_dp = [&](int it) {
        const uint32_t a1 = sRes1, b1 = sO(it % NO);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < HDP / 16; ++kk) {
            const uint32_t off = (kk / 4) * SUBB + (kk % 4) * 32;
            tc_mma_f16(TM_DP, make_smem_desc(a1 + off, 16, 1024, 2), make_smem_desc(b1 + off, 16, 1024, 2), idesc_s, kk != 0);
          }
          tc_commit(bar(BB_DP));
          if (!DKV) tc_commit(bar(BB_OE0 + it % NO));
        }
        __syncwarp();
      };
      // A (16 columns of P or dS per step, 8 tensor-memory columns) lies in the first half of its compute warp's columns; acc += A B over the
      // steps that this piece of every warp's columns makes up
      auto issue_acc = [&](uint32_t acc, uint32_t a, uint32_t b, int piece, bool first) {
        if (elect_one()) {
#pragma unroll
          for (int i = 0; i < 8 / PIECES; ++i) {
            const int w = i / (HC / 16), u = i % (HC / 16);
            tc_mma_f16_ts(acc, a + w * CW + piece * (HC / 2) + u * 8, make_smem_desc(b + ((w * CW + piece * HC) / 16 + u) * 2048, SUBB, 1024, 2), idesc_acc,
                          !(first && piece == 0 && i == 0));
          }
        }
        __syncwarp();
      };
      bool ok = wait(BB_RES0, 0) && wait(BB_QF0, 0);
      if (ok) {
        tc_fence_after();
        issue_s(0);
        ok = wait(BB_RES1, 0) && wait(BB_OF0, 0);
      }
      if (ok) {
        tc_fence_after();
        issue_dp(0);
      }
      for (int it = 0; it < n_iter && ok; ++it) {
        const uint32_t b0 = sQ(it % NQ), b1 = sO(it % NO);
        if (DKV) {          // dV[key, d] += sum_q P^T[key, q] dO[q, d]
#pragma unroll
          for (int piece = 0; piece < PIECES && ok; ++piece) {
            ok = wait(BB_P + piece, it & 1);
            if (!ok) break;
            tc_fence_after();
            issue_acc(TM_ACC0, TM_S, b1, piece, it == 0);
          }
          if (!ok) break;
          if (elect_one()) tc_commit(bar(BB_OE0 + it % NO));
          __syncwarp();
        }
        if (it + 1 < n_iter) {
          if (!wait(BB_QF0 + (it + 1) % NQ, ((it + 1) / NQ) & 1)) { ok = false; break; }
          if (!DKV && !wait(BB_P, it & 1)) { ok = false; break; }          // the S columns have been read
          tc_fence_after();
          issue_s(it + 1);
        }
        // dK[key, d] += sum_q dS^T[key, q] Q[q, d], or dQ[q, d] += sum_key dS[q, key] K[key, d]
#pragma unroll
        for (int piece = 0; piece < PIECES && ok; ++piece) {
          ok = wait(BB_DS + piece, it & 1);
          if (!ok) break;
          tc_fence_after();
          issue_acc(DKV ? TM_ACC1 : TM_ACC0, TM_DP, b0, piece, it == 0);
        }
        if (!ok) break;
        if (elect_one()) tc_commit(bar(BB_QE0 + it % NQ));
        __syncwarp();
        if (it + 1 < n_iter) {
          if (!wait(BB_OF0 + (it + 1) % NO, ((it + 1) / NO) & 1)) { ok = false; break; }
          tc_fence_after();
          issue_dp(it + 1);
        }
      }
      if (ok) {
        if (elect_one()) tc_commit(bar(BB_ACC));
        __syncwarp();
      }
    }
  } else if (warp == 2) {
    // per-query vectors of the inner query tiles, one iteration ahead of the compute warps (loaded by them, each iteration began with the
    // latency of these loads)
    if (DKV) {
      for (int it = 0; it < n_iter; ++it) {
        const int q_tile = in_begin + it % n_in, hq = hq0 + it / n_in;
        const long long base = ((long long)b * p.H + hq) * p.S;
        float lv[4], dv[4];
        int ds[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int qrow = q_tile * 128 + u * 32 + lane;
          const bool in = qrow < p.S;
          // stored negated (and delta pre-multiplied by the softmax scale) so that both uses are one fused multiply-add
          lv[u] = in ? -p.lse[base + qrow] * 1.4426950408889634f : -INFINITY;   // -inf -> exp2(-inf) = 0 for rows past the end
          dv[u] = in ? -p.delta[base + qrow] * p.scale : 0.f;
          ds[u] = dstart ? min(max(dstart[min(qrow, p.S - 1)] - outer * 128, 0), 128) : 0;
        }
        if (it >= 2) {        // the slot was last read before the product that gave back the Q tile of it - 2
          const bool free = mbar_wait(bar(BB_QE0 + (it - 2) % NQ), ((it - 2) / NQ) & 1, abort_flag, p.status);
          if (!__all_sync(0xffffffffu, free)) break;
        }
        uint8_t* vs = smem + L::VEC_OFF + (it & 1) * L::VEC;
        float* vf = reinterpret_cast<float*>(vs);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          vf[u * 32 + lane] = lv[u];
          vf[128 + u * 32 + lane] = dv[u];
          vs[1024 + u * 32 + lane] = (uint8_t)ds[u];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(BB_VF0 + (it & 1)));
      }
    }
  } else {
    // ---------------------------------------------------------------- compute warps
    const int quarter = warp & 3;
    const int part = (warp - 3) >> 2;             // which columns of the block
    const int row_local = quarter * 32 + lane;    // lane of tensor memory: key row (DKV) or query row (DQ)
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const int colw = part * CW;
    bool ok = true;
    float lse2 = 0.f, dlt = 0.f;
    bool row_ok = true;
    int lower = 0;                                // DQ: first key this query row may see (packed sequences)
    int doc_last = 0;                             // DQ: document start of the last query row
    if (!DKV) {
      const int row = outer * 128 + row_local;
      row_ok = row < p.S;
      if (row_ok) {   // negated / pre-scaled like the shared-memory vectors of the other mode
        lse2 = -p.lse[((long long)b * p.H + h) * p.S + row] * 1.4426950408889634f;
        dlt = -p.delta[((long long)b * p.H + h) * p.S + row] * p.scale;
        if (dstart) lower = dstart[row];
      }
      if (dstart) doc_last = dstart[min(outer * 128 + 127, p.S - 1)];
    }
    const float sc2 = p.scale_log2;
    const uint64_t sc2x2 = pack_f32x2(sc2, sc2), scx2 = pack_f32x2(p.scale, p.scale);
    for (int it = 0, in_tile = in_begin; it < n_iter; ++it, in_tile = in_tile + 1 < in_end ? in_tile + 1 : in_begin) {
      const int k_tile = DKV ? outer : in_tile;
      const uint8_t* vs = smem + L::VEC_OFF + (it & 1) * L::VEC;
      const float* vl = reinterpret_cast<const float*>(vs);
      const uint8_t* vdoc = vs + 1024;
      if (DKV && ok) ok = mbar_wait(bar(BB_VF0 + (it & 1)), (it >> 1) & 1, abort_flag, p.status);
      if (ok) ok = mbar_wait(bar(BB_S), it & 1, abort_flag, p.status);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const bool diag = p.causal && in_tile == outer;
      uint32_t rs[CW];                   // S, then the probabilities (fp32, kept for dS)
      load_cols(TM_S + lane_addr + colw, rs);
      if (!DKV) {                        // the S columns have been read: the next S product may overwrite them
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(BB_P));
      }
      // ---- phase 1: P = exp2(S * scale - lse), a piece of the columns at a time. `diag` (and a ragged last tile) is uniform over the CTA: only
      // those tiles pay for the per-element mask test. The per-query vectors come from shared memory four at a time.
      auto phase1 = [&](auto masked_tag, int piece) {
        constexpr bool MASK = decltype(masked_tag)::value;
        uint32_t docs[4] = {};           // key-tile pass: document starts of the piece's 16 queries
        if (DKV && MASK) {
          const uint4 q4 = *reinterpret_cast<const uint4*>(vdoc + colw + piece * HC);
          docs[0] = q4.x; docs[1] = q4.y; docs[2] = q4.z; docs[3] = q4.w;
        }
#pragma unroll
        for (int i = piece * HC; i < piece * HC + HC; i += 4) {
          float l4[4] = {lse2, lse2, lse2, lse2};
          if (DKV) {
            const float4 t4 = *reinterpret_cast<const float4*>(vl + colw + i);
            l4[0] = t4.x; l4[1] = t4.y; l4[2] = t4.z; l4[3] = t4.w;
          }
          if (MASK) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int col = colw + i + u;
              float e = fast_exp2(fmaf(__uint_as_float(rs[i + u]), sc2, l4[u]));
              // DKV: lane = key, column = query -> masked when key > query; DQ: lane = query, column = key
              const int j = i + u - piece * HC;
              const bool masked = DKV ? (diag && row_local > col) || row_local < (int)((docs[(j >> 2) & 3] >> (8 * (j & 3))) & 255u)
                                      : !row_ok || (diag && col > row_local) || k_tile * 128 + col < lower;
              if (masked) e = 0.f;
              rs[i + u] = __float_as_uint(e);
            }
          } else {
#pragma unroll
            for (int u = 0; u < 4; u += 2) {   // packed pairs: one FFMA instruction per two elements
              float x0, x1;
              unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(rs[i + u]), __uint_as_float(rs[i + u + 1])), sc2x2,
                                     pack_f32x2(l4[u], l4[u + 1])), x0, x1);
              rs[i + u] = __float_as_uint(fast_exp2(x0));
              rs[i + u + 1] = __float_as_uint(fast_exp2(x1));
            }
          }
        }
      };
      // a piece's bf16 pairs into tensor memory, then it is handed to the MMA warp
      auto hand_over = [&](uint32_t at, const uint32_t (&t)[HC / 2], int bar_id, int piece) {
        const uint32_t dst = at + lane_addr + colw + piece * (HC / 2);
        __syncwarp();                    // one lane's arrival for the piece before: the stores want the warp together
        static_assert(HC == 64 || HC == 16, "the stores that follow");
        if constexpr (HC == 64) tmem_st32(dst, t); else tmem_st8(dst, t);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(bar_id + piece));
      };
      // a document boundary inside the block pair: the key tile starts before the query tile's last document does
      const bool doc_mask = dstart && (DKV ? vdoc[127] > 0 : k_tile * 128 < doc_last);
      const bool any_mask = diag || doc_mask || (!DKV && (outer + 1) * 128 > p.S);
#pragma unroll
      for (int piece = 0; piece < PIECES; ++piece) {
        if (any_mask) phase1(std::true_type{}, piece); else phase1(std::false_type{}, piece);
        if (DKV) {
          uint32_t t[HC / 2];
#pragma unroll
          for (int i = 0; i < HC / 2; ++i) t[i] = pack_bf16(__uint_as_float(rs[piece * HC + 2 * i]), __uint_as_float(rs[piece * HC + 2 * i + 1]));
          hand_over(TM_S, t, BB_P, piece);
        }
      }
      // ---- phase 2: dS = P * (dP - delta) * scale
      ok = mbar_wait(bar(BB_DP), it & 1, abort_flag, p.status);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      uint32_t rd[CW];
      load_cols(TM_DP + lane_addr + colw, rd);
#pragma unroll
      for (int piece = 0; piece < PIECES; ++piece) {
        uint32_t t[HC / 2];
#pragma unroll
        for (int i = piece * HC; i < piece * HC + HC; i += 4) {
          float d4[4] = {dlt, dlt, dlt, dlt};
          if (DKV) {
            const float4 t4 = *reinterpret_cast<const float4*>(vl + 128 + colw + i);
            d4[0] = t4.x; d4[1] = t4.y; d4[2] = t4.z; d4[3] = t4.w;
          }
          // dS = P * (dP * scale - delta * scale): one packed FFMA and one packed FMUL per two elements
          float x0, x1, x2, x3;
          const uint64_t t01 = fma_f32x2(pack_f32x2(__uint_as_float(rd[i]), __uint_as_float(rd[i + 1])), scx2, pack_f32x2(d4[0], d4[1]));
          const uint64_t t23 = fma_f32x2(pack_f32x2(__uint_as_float(rd[i + 2]), __uint_as_float(rd[i + 3])), scx2, pack_f32x2(d4[2], d4[3]));
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(rs[i]), __uint_as_float(rs[i + 1])), t01, 0ull), x0, x1);
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(rs[i + 2]), __uint_as_float(rs[i + 3])), t23, 0ull), x2, x3);
          t[(i - piece * HC) >> 1] = pack_bf16(x0, x1);
          t[((i - piece * HC) >> 1) + 1] = pack_bf16(x2, x3);
        }
        hand_over(TM_DP, t, BB_DS, piece);
      }
    }
    // ---------------------------------------------------------------- epilogue
    if (ok) {
      ok = mbar_wait(bar(BB_ACC), 0, abort_flag, p.status);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok) {
      tc_fence_after();
      const int row = outer * 128 + row_local;   // key row (DKV) or query row (DQ)
      constexpr int CHUNKS = HDP / 32;           // 32-column chunks per accumulator
      constexpr int NACC = DKV ? 2 : 1;
      // split the NACC * CHUNKS chunks between the warps that share this lane quarter
      for (int idx = part; idx < NACC * CHUNKS; idx += SPLIT) {
        const int acc = idx / CHUNKS, c = idx % CHUNKS;
        uint32_t r[32];
        tmem_ld32((acc == 0 ? TM_ACC0 : TM_ACC1) + lane_addr + c * 32, r);
        tmem_ld_wait32(r);
        if (DKV && nsplit > 1) {                 // to the cluster, over the tiles: every product that read them is done
          float* red = reinterpret_cast<float*>(smem + L::INQ) + row_local * L::RED_LD + idx * 32;
#pragma unroll
          for (int g = 0; g < 8; ++g) *reinterpret_cast<uint4*>(red + g * 4) = make_uint4(r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3]);
          continue;
        }
        // DKV: acc 0 = dV, acc 1 = dK of key head `kvh`; DQ: dQ of query head `h`; heads are [H query | Hkv key | Hkv value]
        const int head = DKV ? (acc == 0 ? p.H + p.Hkv + kvh : p.H + kvh) : h;
        if (row < p.S) {
          __nv_bfloat16* dst = p.dqkv + (long long)row * p.d_stride_s + (long long)b * p.d_stride_b + (long long)head * p.hd;
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const int d0 = c * 32 + g * 8;
            if (d0 < p.hd) {
              uint4 v = make_uint4(pack_bf16(__uint_as_float(r[g * 8]), __uint_as_float(r[g * 8 + 1])),
                                   pack_bf16(__uint_as_float(r[g * 8 + 2]), __uint_as_float(r[g * 8 + 3])),
                                   pack_bf16(__uint_as_float(r[g * 8 + 4]), __uint_as_float(r[g * 8 + 5])),
                                   pack_bf16(__uint_as_float(r[g * 8 + 6]), __uint_as_float(r[g * 8 + 7])));
              *reinterpret_cast<uint4*>(dst + d0) = v;
            }
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (DKV && nsplit > 1) {                       // dV | dK of 128 / nsplit rows: the shares of the cluster, added up in rank order
    cluster_sync_all();
    const int rows = 128 / nsplit;
    const uint32_t red = sbase + L::INQ;
    if (!*abort_flag) {
      for (int i = threadIdx.x; i < rows * (2 * HDP / 8); i += BwdWarps<DKV>::THREADS) {
        const int rl = share * rows + i / (2 * HDP / 8), c = i % (2 * HDP / 8) * 8, d0 = c % HDP;
        const int row = outer * 128 + rl;
        if (row >= p.S || d0 >= p.hd) continue;
        float s[8] = {};
        for (int w = 0; w < nsplit; ++w) {
          const uint32_t src = map_to_cta(red + (uint32_t)(rl * L::RED_LD + c) * 4, w);
          const float4 x = ld_cluster_f4(src), y = ld_cluster_f4(src + 16);
          s[0] += x.x; s[1] += x.y; s[2] += x.z; s[3] += x.w;
          s[4] += y.x; s[5] += y.y; s[6] += y.z; s[7] += y.w;
        }
        const int head = c < HDP ? p.H + p.Hkv + kvh : p.H + kvh;
        *reinterpret_cast<uint4*>(p.dqkv + (long long)row * p.d_stride_s + (long long)b * p.d_stride_b + (long long)head * p.hd + d0) =
            make_uint4(pack_bf16(s[0], s[1]), pack_bf16(s[2], s[3]), pack_bf16(s[4], s[5]), pack_bf16(s[6], s[7]));
      }
    }
    __syncwarp();
    cluster_sync_all();                          // nobody leaves while its shared memory is being read
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int HDP, bool DKV>
int launch_attn_bwd(const CUtensorMap& tmQKV, const CUtensorMap& tmDO, const AttnBwdParams& p, cudaStream_t stream) {
  using L = BwdSmem<HDP, DKV>;
  auto kern = attn_bwd_kernel<HDP, DKV>;
  static std::atomic<unsigned long long> configured{0};      // devices on which the kernel may use this much; asking each time costs the host 1 to 2 us
  int dev = 0;
  ELFA_CUDA(cudaGetDevice(&dev));
  if (dev > 63 || !(configured.load(std::memory_order_relaxed) >> dev & 1)) {
    ELFA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL));
    if (dev <= 63) configured.fetch_or(1ull << dev, std::memory_order_relaxed);
  }
  const unsigned nsplit = DKV ? p.nsplit : 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)p.n_tiles * (DKV ? p.Hkv : p.H) * p.B * nsplit);
  cfg.blockDim = dim3(BwdWarps<DKV>::THREADS);
  cfg.dynamicSmemBytes = L::TOTAL;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = nsplit;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = nsplit > 1 ? 1 : 0;
  ELFA_CUDA(cudaLaunchKernelEx(&cfg, kern, tmQKV, tmDO, p));
  ::elfa::count_launches(1);
  return ELFA_OK;
}

}  // namespace
}  // namespace elfa

using namespace elfa;

// How many CTAs (a cluster of 1, 2 or 4) share the query heads of a key head in the key-tile pass: the number with the least estimated time. A CTA
// costs its start and end (10, 11 or 13 us) and 1.4 or 1.9 us per block pair (64- or 128-wide heads); one fits an SM, and of clusters of four
// 32 at a time. Causal tiles differ and run longest first: the longest CTA, or the whole work spread over the SMs and a tenth; others are
// alike and run in whole rounds. Document masks count as causal. Of 43 shapes (12 to 512 tiles x heads, 1 to 32 tiles) it misses the fastest
// number once, by 3 %. Measured (us, 1 / 2 / 4 shares; 4 query heads to a key head, causal unless said): S 1777 x 2, 4 key heads of 64, 5 documents 75 / 44 / 58;
// S 2048, 4 of 128 120 / 69 / 60; S 1024 x 4, 4 of 128 68 / 55 / 89, not causal 70 / 82 / 114; S 1024 x 4, 8 of 128 81 / 106 / 175;
// S 128 x 36, 4 of 128 21 / 35 / 78.
ELFA_API int elfa_attention_bwd_shares(int S, int B, int H, int Hkv, int hd, int causal) {
  if (S <= 0 || B <= 0 || Hkv <= 0 || H <= 0 || H % Hkv) return 1;
  const long long sms = device_sm_count() > 0 ? device_sm_count() : 148, tiles = (S + 127) / 128, units = tiles * Hkv * B, group = H / Hkv;
  const double pair = hd <= 64 ? 1.4 : 1.9, pairs = (double)units * (double)(tiles + 1) / 2 * (double)group;      // causal
  double best = 0;
  int at = 1;
  for (int n = 1; n <= 4 && group % n == 0; n *= 2) {
    const double ends = n == 1 ? 10 : (n == 2 ? 11 : 13), longest = ends + (double)(tiles * (group / n)) * pair;
    const long long room = n < 4 ? sms : sms * 32 / 37;
    const double t = causal ? std::max(longest, 1.1 * ((double)(units * n) * ends + pairs * pair) / (double)room)
                            : (double)((units * n + room - 1) / room) * longest;
    if (n == 1 || t < best) {
      best = t;
      at = n;
    }
  }
  return at;
}

// Gradients of attention w.r.t. the fused qkv tensor (heads [H query | Hkv key | Hkv value], see elfa_attention_fwd_ex).
// `out` / `dout` share strides (o_stride_*), `dqkv` has the layout of qkv with its own strides; `delta` is [B, H, S] fp32
// scratch. doc_start: [B, S] int32 or null.
ELFA_API int elfa_attention_bwd_ex(const void* qkv, long long stride_s, long long stride_b, const void* out, const void* dout,
                                   long long o_stride_s, long long o_stride_b, const float* lse, float* delta, void* dqkv,
                                   long long d_stride_s, long long d_stride_b, int S, int B, int H, int Hkv, int hd, float scale,
                                   int causal, const int* doc_start, void* stream) {
  ELFA_REQUIRE(qkv && out && dout && lse && delta && dqkv && S > 0 && B > 0 && H > 0, "attention_bwd: bad arguments");
  ELFA_REQUIRE(Hkv > 0 && H % Hkv == 0, "attention_bwd: the query heads must be a multiple of the key / value heads");
  ELFA_REQUIRE(!doc_start || causal, "attention_bwd: document masks need causal attention");
  ELFA_REQUIRE(hd % 8 == 0 && hd >= 8 && hd <= 128, "attention_bwd: head_dim must be a multiple of 8 in [8, 128]");
  ELFA_REQUIRE(stride_s % 8 == 0 && stride_b % 8 == 0 && o_stride_s % 8 == 0 && o_stride_b % 8 == 0 && d_stride_s % 8 == 0 &&
                   d_stride_b % 8 == 0,
               "attention_bwd: strides must be multiples of 8");
  unsigned int* st = status_word();
  ELFA_REQUIRE(st != nullptr, "attention_bwd: no status word");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const long long rows = (long long)S * B * H;
  const int per = hd <= 64 ? 64 : 32;      // rows of a block
  ELFA_REQUIRE((rows + per - 1) / per < (1ll << 31), "attention_bwd: too many rows");
  auto delta_kernel = hd <= 64 ? attn_delta_kernel<8> : attn_delta_kernel<16>;
  delta_kernel<<<(unsigned)((rows + per - 1) / per), 256, 0, s>>>(static_cast<const __nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(dout),
                                                                  o_stride_s, o_stride_b, delta, S, B, H, hd);
  ELFA_CUDA(cudaGetLastError());
  ::elfa::count_launches(1);
  CUtensorMap tmQKV, tmDO;
  int rc = make_qkv_tmap(&tmQKV, qkv, S, B, H + 2 * Hkv, hd, stride_s, stride_b, 1, 128);
  if (rc != ELFA_OK) return rc;
  rc = make_qkv_tmap(&tmDO, dout, S, B, H, hd, o_stride_s, o_stride_b, 1, 128);
  if (rc != ELFA_OK) return rc;
  AttnBwdParams p{};
  p.S = S; p.B = B; p.H = H; p.hd = hd;
  p.Hkv = Hkv;
  p.doc_start = doc_start;
  p.lse = lse; p.delta = delta;
  p.dqkv = static_cast<__nv_bfloat16*>(dqkv);
  p.d_stride_s = d_stride_s; p.d_stride_b = d_stride_b;
  p.scale = scale;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = causal;
  p.n_tiles = (S + 127) / 128;
  p.nsplit = elfa_attention_bwd_shares(S, B, H, Hkv, hd, causal);
  p.status = st;
  if (hd <= 64) {
    rc = launch_attn_bwd<64, true>(tmQKV, tmDO, p, s);
    if (rc != ELFA_OK) return rc;
    return launch_attn_bwd<64, false>(tmQKV, tmDO, p, s);
  }
  rc = launch_attn_bwd<128, true>(tmQKV, tmDO, p, s);
  if (rc != ELFA_OK) return rc;
  return launch_attn_bwd<128, false>(tmQKV, tmDO, p, s);
}

ELFA_API int elfa_attention_bwd(const void* qkv, long long stride_s, long long stride_b, const void* out, const void* dout,
                                long long o_stride_s, long long o_stride_b, const float* lse, float* delta, void* dqkv,
                                long long d_stride_s, long long d_stride_b, int S, int B, int H, int hd, float scale, int causal,
                                void* stream) {
  return elfa_attention_bwd_ex(qkv, stride_s, stride_b, out, dout, o_stride_s, o_stride_b, lse, delta, dqkv, d_stride_s, d_stride_b, S, B,
                               H, H, hd, scale, causal, nullptr, stream);
}
