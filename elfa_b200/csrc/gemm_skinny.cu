// Products of up to eight rows with a weight matrix (decoding, one token of a small batch): C[M, N] = epilogue(alpha * A[M, K] op(B)), bf16
// operands, fp32 sums. The matrix is read once with 16-byte loads and that read is the cost, so the matrix is the left operand of
// mma.sync m16n8k16 (its output index runs along the 16 rows) and the rows of A are its eight columns: a loaded vector needs no conversion (or one
// byte permutation per register) and eight rows cost what one costs. A tcgen05 tile of 128 rows does sixteen rows of padding for each
// real one and leaves most SMs idle (8 to 32 tiles). Four rows, microseconds here / in such tiles: 1536 x 1024 4.2 / 8.3, 4096 x 1024 5.9 / 8.9, 1024 x 4096
// 7.4 / 21, 4096 x 11008 20 / 50, and with the contraction contiguous 11008 x 4096 22 / 37, 32000 x 1024 15 / 22; eight rows take 0 to 10 % more. With packed
// multiply-adds instead of products, eight rows of 4096 x 1024 took 16 us.
//
// The sums are short (a warp's share of the contraction) and joined in fp32: of the outputs, as many as lie beside the bf16 value nearest to the 64-bit product,
// in millionths here / in such tiles: K 1024 93 / 556, 4096 174 / 2550, 11008 308 / 6091.
//
// The order of a contraction is free as long as both operands share it, and so is which output a fragment row stands for; both are
// chosen so that a thread's 16 bytes are whole fragments.
//
// reference: src/eval/evaluator.zig:419-470 (generation, one token at a time).
#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "elfa_native.h"
#include "gemm_skinny.cuh"
#include "mma_sync.cuh"

namespace elfa {
namespace {

__device__ __forceinline__ uint4 ld_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// eight neighbouring columns of one row: + bias, value before the activation, activation, one 16-byte store
__device__ __forceinline__ void skinny_store(const SkinnyParams& p, int m, int n, const float (&acc)[8]) {
  float f[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    f[j] = acc[j] * p.alpha;
    if (p.flags & ELFA_EPI_BIAS) f[j] += __bfloat162float(p.bias[n + j]);
  }
  auto put = [&](__nv_bfloat16* dst) {
    *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
  };
  if (p.flags & ELFA_EPI_STORE_PREACT) put(p.preact + m * p.ldpre + n);
  if (p.flags & ELFA_EPI_GELU) {
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = gelu_tanh(f[j]);
  }
  put(p.C + m * p.ldc + n);
}

// B [K, N], output index contiguous. A CTA owns 64 HALVES columns and a slice of the contraction, its eight warps 16 rows of B in turn: thread (g, q) of a
// warp loads 16 bytes (columns 8 g .. and 64 + 8 g ..) of rows 2 q, 2 q + 1, 2 q + 8 and 2 q + 9, pairs the rows by byte permutation, and product
// j of eight takes column 8 g + j (fragment row g) and 64 + 8 g + j (row g + 8). The slices of a column block are the CTAs of one cluster; warps
// and slices add up in a fixed order.
template <int HALVES>
__global__ void __launch_bounds__(256) skinny_nn_kernel(const SkinnyParams p, int ks) {
  __shared__ __align__(16) float part[8][8][132];      // [warp][row of A][column]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int n0 = blockIdx.x * (64 * HALVES), k1 = min(p.K, (int)(blockIdx.y + 1) * ks);
  const int na = n0 + 8 * g, nb = na + 64;
  const bool ina = na < p.N, inb = HALVES > 1 && nb < p.N;           // N is a multiple of 8
  float acc[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int x = 0; x < 4; ++x) acc[j][x] = 0.f;
  // the rows 2 q, 2 q + 1, 2 q + 8, 2 q + 9 of both column halves; the first ones before the launches ahead are waited for
  uint4 w[4][2];
  auto load = [&](int k) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int kr = k + 2 * q + (r & 1) + (r >> 1) * 8;
      const __nv_bfloat16* row = p.B + kr * p.ldb;
      w[r][0] = w[r][1] = make_uint4(0, 0, 0, 0);
      if (kr < k1 && ina) w[r][0] = ld_stream(row + na);
      if (kr < k1 && inb) w[r][1] = ld_stream(row + nb);
    }
  };
  const int kfirst = blockIdx.y * ks + warp * 16;
  load(kfirst);
  pdl_wait();
  pdl_next();
  for (int k = kfirst; k < k1; k += 128) {
    uint4 v[4][2];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      v[r][0] = w[r][0];
      v[r][1] = w[r][1];
    }
    if (k + 128 < k1) load(k + 128);
    uint32_t x0 = 0, x1 = 0;                           // A[g][2 q ..] and A[g][2 q + 8 ..]; K is a multiple of 8
    if (g < p.M) {
      const __nv_bfloat16* a = p.A + g * p.lda + k + 2 * q;
      x0 = *reinterpret_cast<const uint32_t*>(a);
      if (k + 8 < k1) x1 = *reinterpret_cast<const uint32_t*>(a + 8);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      uint32_t f[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {                    // a0, a1: rows 2 q, 2 q + 1 of halves 0, 1; a2, a3: the rows 8 further
        const uint32_t lo = reinterpret_cast<const uint32_t*>(&v[x / 2 * 2][x & 1])[j / 2], hi = reinterpret_cast<const uint32_t*>(&v[x / 2 * 2 + 1][x & 1])[j / 2];
        f[x] = HALVES == 1 && (x & 1) ? 0u : __byte_perm(lo, hi, j & 1 ? 0x7632 : 0x5410);
      }
      mma_bf16(acc[j], f, x0, x1);
    }
  }
#pragma unroll
  for (int x = 0; x < 2 * HALVES; ++x) {               // x = 0, 1: column 8 g + j, rows 2 q, 2 q + 1 of A; 2, 3: column 64 + 8 g + j
    float* dst = &part[warp][2 * q + (x & 1)][(x >> 1) * 64 + 8 * g];
    *reinterpret_cast<float4*>(dst) = make_float4(acc[0][x], acc[1][x], acc[2][x], acc[3][x]);
    *reinterpret_cast<float4*>(dst + 4) = make_float4(acc[4][x], acc[5][x], acc[6][x], acc[7][x]);
  }
  __syncthreads();
  float* sum = &part[0][0][0];                         // the warps' parts, added up over those of warp 0
  for (int i = threadIdx.x; i < p.M * 16 * HALVES; i += 256) {
    const int at = i / (16 * HALVES) * 132 + i % (16 * HALVES) * 4;
    float4 s = *reinterpret_cast<const float4*>(sum + at);
#pragma unroll
    for (int w = 1; w < 8; ++w) {
      const float4 v = *reinterpret_cast<const float4*>(sum + w * 8 * 132 + at);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    *reinterpret_cast<float4*>(sum + at) = s;
  }
  const int shares = gridDim.y, rank = blockIdx.y;
  if (shares > 1) cluster_sync_all();
  else __syncthreads();
  for (int i = rank + threadIdx.x * shares; i < p.M * 8 * HALVES; i += 256 * shares) {
    const int m = i / (8 * HALVES), c = i % (8 * HALVES) * 8;
    float f[8] = {};
    for (int r = 0; r < shares; ++r) {
      const uint32_t at = smem_u32(sum + m * 132 + c), src = shares > 1 ? map_to_cta(at, r) : at;
      const float4 x = ld_cluster_f4(src), y = ld_cluster_f4(src + 16);
      f[0] += x.x; f[1] += x.y; f[2] += x.z; f[3] += x.w;
      f[4] += y.x; f[5] += y.y; f[6] += y.z; f[7] += y.w;
    }
    if (n0 + c < p.N) skinny_store(p, m, n0 + c, f);
  }
  __syncwarp();
  if (shares > 1) cluster_sync_all();                  // nobody leaves while its sums are being read
}

// B [N, K], contraction contiguous. A warp owns 16 columns: thread (g, q) loads 16 bytes of rows g and g + 8 of B, k = 8 q .., which are the
// fragments of two products (k 8 q .. 8 q + 3 and 8 q + 4 .. 8 q + 7 of every q), and the same of row g of A. WK warps of a CTA share 16 columns,
// 32 J values of k each in turn, where there are few columns: with J = 4 or 2 a warp asks for whole lines (J = 1, for short contractions: half of
// one). N 9480, K 4096: WK 4, J 1 / 2 25 / 20 us; N 32000, K 1024: WK 8, J 1 / 4 16.6 / 15.0 us.
template <int WK, int J>
__global__ void __launch_bounds__(256) skinny_nt_kernel(const SkinnyParams p) {
  __shared__ __align__(16) float part[8][8][20];       // [warp][row of A][column]
  constexpr int UN = 4;                                // 32 values of k each, in flight
  static_assert(UN % J == 0, "steps of a warp");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int group = warp / WK, n0 = (blockIdx.x * (8 / WK) + group) * 16;
  const bool in0 = n0 + g < p.N, in1 = n0 + g + 8 < p.N;
  const __nv_bfloat16 *b0 = p.B + (n0 + g) * p.ldb + 8 * q, *b1 = b0 + 8 * p.ldb, *a = p.A + g * p.lda + 8 * q;
  float acc[2][4] = {};
  pdl_wait();
  pdl_next();
  for (int kb = warp % WK * (32 * J); kb < p.K; kb += WK * UN * 32) {
    uint4 w0[UN], w1[UN], x[UN];
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      const int k = kb + u / J * (WK * 32 * J) + u % J * 32;
      const bool in = k + 8 * q < p.K;
      w0[u] = w1[u] = x[u] = make_uint4(0, 0, 0, 0);
      if (in && in0) w0[u] = ld_stream(b0 + k);
      if (in && in1) w1[u] = ld_stream(b1 + k);
      if (in && g < p.M) x[u] = *reinterpret_cast<const uint4*>(a + k);
    }
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      const uint32_t f0[4] = {w0[u].x, w1[u].x, w0[u].y, w1[u].y}, f1[4] = {w0[u].z, w1[u].z, w0[u].w, w1[u].w};
      mma_bf16(acc[0], f0, x[u].x, x[u].y);
      mma_bf16(acc[1], f1, x[u].z, x[u].w);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) part[warp][2 * q + (i & 1)][g + (i >> 1) * 8] = acc[0][i] + acc[1][i];
  if (WK > 1) __syncthreads();
  else __syncwarp();
  constexpr int GROUPS = WK > 1 ? 8 / WK : 1;          // of 16 columns, added up by the CTA, or by each warp its own
  for (int i = (WK > 1 ? threadIdx.x : lane); i < p.M * 2 * GROUPS; i += WK > 1 ? 256 : 32) {
    const int m = i / (2 * GROUPS), at = i / 2 % GROUPS, c = i % 2 * 8, first = WK > 1 ? at * WK : warp;
    const int n = WK > 1 ? (blockIdx.x * GROUPS + at) * 16 : n0;
    float f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      f[j] = part[first][m][c + j];
#pragma unroll
      for (int w = 1; w < WK; ++w) f[j] += part[first + w][m][c + j];
    }
    if (n + c < p.N) skinny_store(p, m, n + c, f);
  }
}

// Clusters of n CTAs that run at once, asked once per width and size: SMs that do not fill a cluster are left out. (On a B200 with 148 SMs 148, 93, 71 and 33
// clusters of 2, 3, 4 and 8 CTAs of 128 columns, 222, 142, 104 and 48 of 64.)
int skinny_room(bool narrow, int n, int sms) {
  static std::atomic<int> known[2][9];
  int v = known[narrow][n].load(std::memory_order_relaxed);
  if (v > 0) return v;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(1, n);
  cfg.blockDim = dim3(256);
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = at[0].val.clusterDim.z = 1;
  at[0].val.clusterDim.y = n;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&v, narrow ? skinny_nn_kernel<1> : skinny_nn_kernel<2>, &cfg) != cudaSuccess || v <= 0) {
    cudaGetLastError();
    return std::max(1, (narrow ? 3 : 2) * sms / n);      // two CTAs of 128 columns or three of 64 fit an SM
  }
  known[narrow][n].store(v, std::memory_order_relaxed);
  return v;
}

// How a [K, N] matrix is cut: in as many slices (1, 2, 3, 4 or 8 of at least 256 rows; of 128 where SMs are idle otherwise) as run at once, in the width that
// fills more of the room; past one round whole columns of 128. One slice too many starts a second round. Four to eight rows, us: N 8192, K 4096, 128 wide
// 4 / 8 slices 15 / 19; N 11008, K 4096, 3 / 4 20 / 30; N 32000, K 4096, 1 / 2 45 / 52; N 6144, K 2048, 64 wide 4 / 128 wide 8 9.3 / 15;
// N 12288, K 8192, 64 wide 2 / 128 wide 3 (96 clusters, 93 fit) 43 / 57.
SkinnyPlan plan_for(int N, int K, int sms) {
  const bool few = (N + 127) / 128 * 8 < sms;          // 128 wide would leave SMs idle even with eight slices
  SkinnyPlan best{few, 1};
  double fill = 0;
  for (int w = few ? 1 : 0; w < 2; ++w) {
    const int tiles = w ? (N + 63) / 64 : (N + 127) / 128;
    for (int n : {1, 2, 3, 4, 8}) {
      const int room = skinny_room(w != 0, n, sms);
      if (n > 1 && (tiles > room || K / n < (K >= 1024 && tiles * n <= sms ? 128 : 256))) continue;
      if (n == 1 && tiles > room) {                    // several rounds
        if (!w) return {false, 1};
        continue;
      }
      if ((double)tiles / room > fill) {
        fill = (double)tiles / room;
        best = {w != 0, n};
      }
    }
  }
  return best;
}

}  // namespace

SkinnyPlan skinny_plan(int N, int K) { return plan_for(N, K, device_sm_count() > 0 ? device_sm_count() : 148); }

// The tensor-core tiles are faster for a large matrix whose columns make most of one wave of 128, once A has 64 K values (below, they take half as
// long again). Eight rows, us here / there: 8192 x 12288 43 / 41, x 14336 48 / 42, x 16384 49 / 45; contraction contiguous, 28672 x 12288 145 / 128,
// x 16384 161 / 153; outside 8192 x 11008 35 / 41, x 18944 50 / 54, and 4096 x 14336 27 / 35.
bool gemm_skinny_better(int M, int N, int K) {
  const int sms = device_sm_count() > 0 ? device_sm_count() : 148;
  return (long long)M * K < 65536 || N < 80 * sms || N >= 128 * sms;
}

int launch_gemm_skinny(const SkinnyParams& p, bool b_mn, cudaStream_t s) {
  const int sms = device_sm_count() > 0 ? device_sm_count() : 148;
  if (!b_mn) {
    // Warps per 16 columns: eight; four for the columns that make one round of them and a bit with eight (11008: 52 us against 60 at K 11008); one
    // where there are many columns and a contraction of a few hundred leaves nothing to share (K 256, N 64000: 7.5 us with one, 9.6 with
    // four, 13 with eight; N 11008 4.9, 3.2 and 3.4).
    auto launch = [&](auto kernel, int wk) { return launch_chain(kernel, dim3((p.N + 128 / wk - 1) / (128 / wk)), dim3(256), 0, s, 1, p); };
    if (p.K <= 512 && p.N >= 192 * sms) ELFA_CUDA(launch(skinny_nt_kernel<1, 1>, 1));
    else if (p.N >= 64 * sms && (p.K <= 512 || p.N < 80 * sms)) ELFA_CUDA(launch(skinny_nt_kernel<4, 2>, 4));
    else if (p.K >= 1024) ELFA_CUDA(launch(skinny_nt_kernel<8, 4>, 8));
    else ELFA_CUDA(launch(skinny_nt_kernel<8, 1>, 8));
  } else {
    const SkinnyPlan plan = plan_for(p.N, p.K, sms);
    ELFA_CUDA(launch_chain(plan.narrow ? skinny_nn_kernel<1> : skinny_nn_kernel<2>, dim3(plan.tiles(p.N), plan.shares), dim3(256), 0, s, plan.shares, p,
                           plan.ks(p.K)));
  }
  ELFA_CUDA(cudaGetLastError());
  ::elfa::count_launches(1);
  return ELFA_OK;
}

}  // namespace elfa
