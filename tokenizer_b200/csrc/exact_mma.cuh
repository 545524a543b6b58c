// 32-bit products on the tensor cores (mma.sync m16n8k16): both operands are cut into three bfloat16 pieces that add up to
// them exactly (8 + 8 + 8 bits and signs), and the six products of pieces that reach 2^-24 of the whole are added up in
// 32-bit, the smallest first.  The tensor core cuts a sum's low bits off instead of rounding: leave it a few dozen terms and
// add its sums to others in plain 32-bit.  A number that is an infinity, a NaN or rounds to an infinity in 16 bits has a NaN
// among its pieces, and a product just below the largest number may lie above it in its first pieces: what comes of them is no
// finite number, and whoever uses this computes it anew from the numbers themselves.
#pragma once
#include "common.cuh"

__device__ __forceinline__ unsigned xm_pack(float lo, float hi) {
  const __nv_bfloat162 pair = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&pair);
}
// two numbers as three pairs of pieces
__device__ __forceinline__ void xm_cut(float lo, float hi, unsigned& p0, unsigned& p1, unsigned& p2) {
  p0 = xm_pack(lo, hi);
  lo -= __uint_as_float(p0 << 16);                       // exact, as is the next
  hi -= __uint_as_float(p0 & 0xffff0000u);
  p1 = xm_pack(lo, hi);
  p2 = xm_pack(lo - __uint_as_float(p1 << 16), hi - __uint_as_float(p1 & 0xffff0000u));
}
__device__ __forceinline__ void xm_mma(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// large[m][n] + small[m][n] += a[m] b[n] for operands in pieces ([piece][registers]): the products of first pieces in a sum of
// their own, so that what they cut off is their own low bits alone and not those of the five others' sum, which is added to them
// in plain 32-bit.  The sums of one term are issued together: each waits for its own sum of the term before, some 20 cycles.
template <int M, int N>
__device__ __forceinline__ void xm_products(float (&large)[M][N][4], float (&small)[M][N][4], const unsigned (&a)[M][3][4],
                                            const unsigned (&b)[N][3][2]) {
  constexpr int kA[6] = {2, 0, 0, 1, 1, 0}, kB[6] = {0, 2, 0, 1, 0, 1};
#pragma unroll
  for (int e = 0; e < 6; ++e)
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int n = 0; n < N; ++n) xm_mma(e == 2 ? large[m][n] : small[m][n], a[m][kA[e]], b[n][kB[e]][0], b[n][kB[e]][1]);
}
