// bit_sums.cuh — the bit columns of the signature AIRs' constraint kernels.
//
// Nine tenths of their cells are bits t_b of limbs and carries, each with a booleanity
// constraint lambda_b t_b (1 - t_b). Both routines accumulate negatives into *neg: one
// small product lambda_b (...) kept to 64 bits of its residue class, and one unreduced
// product with t_b (gl::AccProd), some 45 clocks a bit and warp where a reduced product, a
// 32-bit product into a sum and a shifted add took 70. One out-of-line copy serves every
// range check and carry of a kernel: inlined at each, the unrolled bodies overflowed the
// instruction cache.
#pragma once
#include "gl.cuh"

namespace sg {
namespace bsum {

// lam u + e for any u, as some u64 of its residue class; (lam + 1) 2^32 + e at most 2^64 (so
// lam < 2^18 and e < 2^63, or any lam and e = 0)
__device__ __forceinline__ uint64_t mul18_add(uint32_t lam, uint64_t u, uint64_t e) {
  const uint64_t w = (uint64_t)lam * (uint32_t)u + e;
  const uint64_t v = (uint64_t)lam * (uint32_t)(u >> 32) + (w >> 32);
  uint64_t r;
  // (v : low word of w) with the word h above 2^64 folded: + h 2^32 - h
  asm("{\n\t.reg .u32 w0, w1, v0, h, t, lo, hi;\n\tmov.b64 {w0, w1}, %1;\n\tmov.b64 {v0, h}, %2;\n\t"
      "add.cc.u32 t, v0, h;\n\taddc.u32 h, h, 0;\n\tadd.u32 hi, v0, h;\n\t"
      "sub.cc.u32 lo, w0, h;\n\tsubc.u32 hi, hi, 0;\n\tmov.b64 %0, {lo, hi};\n\t}"
      : "=l"(r) : "l"(w), "l"(v));
  return r;
}

template <int NB>
struct Batch {
  static constexpr int H = NB > 26 ? NB / 2 : NB;  // loads that go out together: up to 26, or 2 x 18 for a 36-bit carry
  static_assert(NB % H == 0 && NB <= 64, "bit batch");
};

// The NB bit cells bits .. bits + NB - 1: booleanity with lambdas lam + b; returns the
// pack sum_b t_b 2^b (canonical).
template <int NB>
static __device__ __noinline__ uint64_t bool_pack(const uint64_t* L, uint64_t n, uint32_t bits, uint32_t lam,
                                                  gl::AccProd* neg) {
  constexpr int H = Batch<NB>::H;
  gl::AccProd a = *neg;
  gl::Acc128 s;
#pragma unroll
  for (int h = 0; h < NB / H; ++h) {
    uint64_t t[H];
#pragma unroll
    for (int j = 0; j < H; ++j) t[j] = __ldg(L + (uint64_t)(bits + h * H + j) * n);
#pragma unroll
    for (int j = 0; j < H; ++j) {
      const int b = h * H + j;
      a.add(t[j], mul18_add(lam + b, gl::sub(t[j], 1), 0));
      if (b < 32)
        s.add_shl(t[j], b);
      else
        s.add_shl32(t[j], b - 32);
    }
  }
  *neg = a;
  return s.reduce();
}

// The same cells as the bits of a limb: booleanity with lambdas lam + b and, with lambda
// lam_pack > lam + NB, limb - sum_b t_b 2^b without its first term: together
// -sum_b t_b (lambda_b t_b + lam_pack 2^b - lambda_b). NB <= 32.
template <int NB>
static __device__ __noinline__ void range_bits(const uint64_t* L, uint64_t n, uint32_t bits, uint32_t lam,
                                               uint32_t lam_pack, gl::AccProd* neg) {
  static_assert(NB <= 32, "limb bits");
  gl::AccProd a = *neg;
  uint64_t t[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) t[b] = __ldg(L + (uint64_t)(bits + b) * n);
#pragma unroll
  for (int b = 0; b < NB; ++b) a.add(t[b], mul18_add(lam + b, t[b], ((uint64_t)lam_pack << b) - (lam + b)));
  *neg = a;
}

}  // namespace bsum
}  // namespace sg
