// hash_phi.cuh — pieces of the SHA-256 and SHA-512 constraint kernels: runs of 32
// constraints of one shape, folded into Phi as they are formed.
//
// A run's value is kept as any u64 of its residue class (gl::mul_any, and gl::add /
// gl::sub with a canonical second operand), and lambda times it goes unreduced into a
// 160-bit sum (gl::AccProd) that is reduced once per chunk. Runs that end in "cell -
// expression" accumulate the negative, expression - cell, so that the product comes
// first; their chunk's sum is negated at the end.
#pragma once
#include "gl.cuh"

namespace sg {
namespace hphi {

// Iterations unrolled together: their loads go out before the first product (all 32 at once
// spill in 64 registers: 717 us for 2^17 SHA-256 points, 405 with 8, 324 with 4).
constexpr int kUnroll = 4;

// cell `col` of a point: column-major evaluations, `stride` words a column
struct Cells {
  const uint64_t* p;
  uint64_t stride;
  __device__ __forceinline__ uint64_t operator()(uint32_t col) const { return __ldg(p + (uint64_t)col * stride); }
};

// booleanity of the 32 cells at `bits` (lambdas lam[0..31]) and word - sum_b bit_b 2^b (lam_pack)
__device__ __forceinline__ void bool_pack(gl::AccProd& acc, const Cells& C, uint32_t bits, uint32_t word,
                                          const uint64_t* lam, const uint64_t* lam_pack) {
  gl::Acc128 s;
#pragma unroll kUnroll
  for (int b = 0; b < 32; ++b) {
    const uint64_t v = C(bits + b);
    acc.add(__ldg(lam + b), gl::mul_any(v, gl::sub(1, v)));
    s.add_shl_var(v, b);
  }
  acc.add(__ldg(lam_pack), gl::sub(C(word), s.reduce()));
}
// the negative of t - (x xor y) = t - (x + y - 2xy)
__device__ __forceinline__ uint64_t xor_neg(uint64_t t, uint64_t x, uint64_t y) {
  return gl::sub(gl::add(gl::mul_any(y, gl::sub(1, gl::add(x, x))), x), t);
}
// negatives of t_b - (x_b xor y_b), x(b) and y(b) giving the operands, for b < 32; with
// PACK also of word - sum_b t_b 2^b
template <bool PACK, class X, class Y>
__device__ __forceinline__ void xor_run(gl::AccProd& acc, const Cells& C, uint32_t t, X&& x, Y&& y,
                                        const uint64_t* lam, uint32_t word, const uint64_t* lam_pack) {
  gl::Acc128 s;
#pragma unroll kUnroll
  for (int b = 0; b < 32; ++b) {
    const uint64_t tv = C(t + b);
    acc.add(__ldg(lam + b), xor_neg(tv, x(b), y(b)));
    if (PACK) s.add_shl_var(tv, b);
  }
  if (PACK) acc.add(__ldg(lam_pack), gl::sub(s.reduce(), C(word)));
}
// negatives of ch_b - (e_b f_b + g_b - e_b g_b) and of word - sum_b ch_b 2^b
__device__ __forceinline__ void ch_run(gl::AccProd& acc, const Cells& C, uint32_t e, uint32_t f, uint32_t g,
                                       uint32_t ch, uint32_t word, const uint64_t* lam, const uint64_t* lam_pack) {
  gl::Acc128 s;
#pragma unroll kUnroll
  for (int b = 0; b < 32; ++b) {
    const uint64_t gv = C(g + b), cv = C(ch + b);
    acc.add(__ldg(lam + b), gl::sub(gl::add(gl::mul_any(C(e + b), gl::sub(C(f + b), gv)), gv), cv));
    s.add_shl_var(cv, b);
  }
  acc.add(__ldg(lam_pack), gl::sub(s.reduce(), C(word)));
}
// negatives of ab_b - a_b b_b, ac_b - a_b c_b, bc_b - b_b c_b, in this order for each b
__device__ __forceinline__ void maj_run(gl::AccProd& acc, const Cells& C, uint32_t a, uint32_t b, uint32_t c,
                                        uint32_t ab, uint32_t ac, uint32_t bc, const uint64_t* lam) {
#pragma unroll kUnroll / 2
  for (int k = 0; k < 32; ++k) {
    const uint64_t av = C(a + k), bv = C(b + k), cv = C(c + k);
    acc.add(__ldg(lam + 3 * k), gl::sub(gl::mul_any(av, bv), C(ab + k)));
    acc.add(__ldg(lam + 3 * k + 1), gl::sub(gl::mul_any(av, cv), C(ac + k)));
    acc.add(__ldg(lam + 3 * k + 2), gl::sub(gl::mul_any(bv, cv), C(bc + k)));
  }
}

// the remaining constraints, one by one in emission order (positive sign)
struct Push {
  gl::AccProd acc;
  const uint64_t* lam;
  __device__ __forceinline__ void push(uint64_t v) { acc.add(__ldg(lam++), v); }
  __device__ __forceinline__ void zeros(uint32_t cnt) { lam += cnt; }  // disabled slots contribute 0
};

// phi[out(i)] = sum over the chunks of part[c count + i]
template <class Out>
__device__ __forceinline__ void sum_parts(const uint64_t* part, uint64_t count, int chunks, uint64_t* phi, Out&& out) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= count) return;
  uint64_t s = 0;
#pragma unroll 8
  for (int c = 0; c < chunks; ++c) s = gl::add(s, part[(uint64_t)c * count + i]);
  phi[out(i)] = s;
}

}  // namespace hphi
}  // namespace sg
