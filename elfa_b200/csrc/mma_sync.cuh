// Warp-level tensor-core helpers (mma.sync m16n8k16, ldmatrix / stmatrix, cp.async) and the three-way bf16 split of fp32
// values, for contractions whose tiles are too small and too dependent for tcgen05 (whose smallest tile has 64 rows and
// whose accumulator has to travel through tensor memory between two dependent products).
//
// Fragment layout used throughout, g = lane / 4, q = lane % 4:
//   A (16 x 16): a0 (row g, k 2q..), a1 (row g + 8), a2 (row g, k 2q + 8..), a3 (row g + 8, k 2q + 8..)
//   B (16 x 8):  b0 (k 2q.., col g), b1 (k 2q + 8.., col g)
//   C (16 x 8):  c0, c1 (row g, col 2q, 2q + 1), c2, c3 (row g + 8)
// so two neighbouring C tiles are, packed to bf16, the A operand of a following product.
#pragma once
#include "common.cuh"

namespace elfa {

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c = a b, the first product of a sum: nothing has to be set to zero before
__device__ __forceinline__ void mma_bf16_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void stsm4_t(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(r0), "r"(r1), "r"(r2), "r"(r3)
               : "memory");
}
// 16-byte asynchronous copy, zero-filled when !ok (the source address must still be a valid one)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool ok) {
  const int n = ok ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// x = hi + mid + lo, each a bf16 (8 significant bits): 24 bits, i.e. fp32 without loss. Two values per register.
// The remainders of both are one packed operation each (exact: -1 times a part, added to what it was taken from).
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const uint64_t minus = pack_f32x2(-1.f, -1.f);
  hi = pack_bf16(x, y);
  uint64_t rest = fma_f32x2(pack_f32x2(bf16_lo(hi), bf16_hi(hi)), minus, pack_f32x2(x, y));
  unpack_f32x2(rest, x, y);
  mid = pack_bf16(x, y);
  rest = fma_f32x2(pack_f32x2(bf16_lo(mid), bf16_hi(mid)), minus, rest);
  unpack_f32x2(rest, x, y);
  lo = pack_bf16(x, y);
}
// two neighbouring values of an accumulator tile as a packed pair
__device__ __forceinline__ uint64_t pair_of(const float (&t)[4], int hf) { return pack_f32x2(t[2 * hf], t[2 * hf + 1]); }
__device__ __forceinline__ void put_pair(float (&t)[4], int hf, uint64_t v) { unpack_f32x2(v, t[2 * hf], t[2 * hf + 1]); }
// The A operand (three splits) of two neighbouring accumulator tiles.
__device__ __forceinline__ void split3_a(uint32_t (&hi)[4], uint32_t (&mid)[4], uint32_t (&lo)[4], const float (&t0)[4], const float (&t1)[4]) {
  split3(t0[0], t0[1], hi[0], mid[0], lo[0]);
  split3(t0[2], t0[3], hi[1], mid[1], lo[1]);
  split3(t1[0], t1[1], hi[2], mid[2], lo[2]);
  split3(t1[2], t1[3], hi[3], mid[3], lo[3]);
}

}  // namespace elfa
