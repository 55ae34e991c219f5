// ntt_tc.cu — NTT passes of 2^8 .. 2^10 points on the int8 tensor cores.
//
// A Goldilocks DFT of R points is a product with a constant matrix of field
// elements. Written in bytes it is an integer product without any carries: with
// x = sum_b x_b 2^(8b) and W_(k,b) = (2^(8b) w^(ik) mod p) = sum_d W_(k,b),d 2^(8d),
//   X[i] = sum_d 2^(8d) D_d,   D_d = sum_k sum_b x_(k,b) W_(k,b),d   (mod p),
// so a row of R field elements, taken as its 8 R bytes in memory, times an
// (8 R) x (8 R) byte matrix gives each output's 8 digit sums D_d < 8 R 255^2 < 2^24:
// one u8 x u8 -> s32 tcgen05.mma chain, whose operand A is the data as it is.
// A pass of M = R1 R2 points (R1 in {16, 32}, R2 in {16, 32}) takes two such products,
// with one field product per element (the twiddle) between them:
//   m = m2 R1 + m1,  j = j' + S i1:
//   X[j] = sum_m1 w_R1^(i1 m1) w_EM^(j' m1) sum_m2 w_S^(j' m2) x[m],   S = E R2,
// E > 1 evaluating E M points from M coefficients (zero padding, coset LDE): the
// first matrix of a chunk of R1 values of j' carries the coset shift and 1/N too.
//
// What bounds it: a tile's serial chain (load, product, join, twiddle, product, join, store),
// of which an SM holds two tiles (R1 = 32) or four (R1 = 16); their accumulators fill its
// tensor memory. No pipe is full: 32 x 32 has the FMA pipe active 37-52 %, ALU 30-42 %, tensor
// 22-39 % of the time; 16 x 16, in bulk, FMA 62 %, ALU 51 %, tensor 26 %. Measured (one call,
// device tensors, before = the radix-16 butterfly passes of ntt.cu, after): LDE of 4099 x 1024
// points x 32: 1666 -> 662 us (600 on buffers that the call before used); 756 x 256 x 32:
// 102 -> 53 us; 64 x 2^20 x 8: 14.7 -> 7.1 ms; inverse 6 x 2^20: 177 -> 123 us; one column of
// 2^8: 25 -> 19 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <new>
#include <tuple>
#include <vector>

#include "counters.hpp"
#include "gl.cuh"
#include "ntt.cuh"
#include "ntt_tc.cuh"

namespace sg {
namespace {

// ------------------------------------------------------------------ lazy field arithmetic
// Any u64 stands for its residue here; only values that leave a transform are canonical.

// sum_d D_d 2^(8d) mod p as some u64, for D_d <= 256 * 255^2: pairs D_d + 256 D_(d+1)
// fit 32 bits (257 * 256 * 255^2 < 2^32), the four pairs are 16 bits apart, and the
// word above 2^64 (below 2^17) is folded once.
// The multipliers come as values the compiler cannot see through, so that the joins stay
// multiply-adds on the FMA pipe instead of shifts on the busier ALU pipe.
__device__ __forceinline__ uint64_t join_digits(const uint32_t* d, uint32_t c8, uint32_t c16) {
  uint64_t r;
  asm("{\n\t.reg .u32 e0, e1, e2, e3, p0, p1, q0, q1, s, h, t, lo, hi;\n\t.reg .u64 p, q, z;\n\t"
      "mad.lo.u32 e0, %2, %9, %1;\n\tmad.lo.u32 e1, %4, %9, %3;\n\t"
      "mad.lo.u32 e2, %6, %9, %5;\n\tmad.lo.u32 e3, %8, %9, %7;\n\t"
      "cvt.u64.u32 z, e0;\n\tmad.wide.u32 p, e1, %10, z;\n\t"
      "cvt.u64.u32 z, e2;\n\tmad.wide.u32 q, e3, %10, z;\n\t"
      "mov.b64 {p0, p1}, p;\n\tmov.b64 {q0, q1}, q;\n\t"
      "add.cc.u32 s, p1, q0;\n\taddc.u32 h, q1, 0;\n\t"
      "add.cc.u32 t, s, h;\n\taddc.u32 h, h, 0;\n\t"
      "add.u32 hi, s, h;\n\t"
      "sub.cc.u32 lo, p0, h;\n\tsubc.u32 hi, hi, 0;\n\t"
      "mov.b64 %0, {lo, hi};\n\t}"
      : "=l"(r)
      : "r"(d[0]), "r"(d[1]), "r"(d[2]), "r"(d[3]), "r"(d[4]), "r"(d[5]), "r"(d[6]), "r"(d[7]),
        "r"(c8), "r"(c16));
  return r;
}

// the canonical form: x >= p exactly when its high word is all ones and its low word is not zero
__device__ __forceinline__ uint64_t canonical(uint64_t x) {
  uint64_t r;
  asm("{\n\t.reg .pred a, b;\n\t.reg .u32 lo, hi;\n\tmov.b64 {lo, hi}, %1;\n\t"
      "setp.ne.u32 a, lo, 0;\n\tsetp.eq.and.u32 b, hi, 0xFFFFFFFF, a;\n\t"
      "@b sub.u32 lo, lo, 1;\n\t@b mov.u32 hi, 0;\n\tmov.b64 %0, {lo, hi};\n\t}"
      : "=l"(r) : "l"(x));
  return r;
}
// base + i * step bytes
__device__ __forceinline__ const char* at(const void* base, uint32_t i, uint32_t step) {
  return (const char*)base + (uint64_t)i * step;
}
__device__ __forceinline__ char* at(void* base, uint32_t i, uint32_t step) { return (char*)base + (uint64_t)i * step; }

// ------------------------------------------------------------------ tcgen05 and barriers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_group(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Waits for a phase with a limit: 2^18 tries, each of which the hardware ends after 4 us, are
// about a second. When it runs out, the host is told through *fail, and *pending = 1 + parity
// says what is outstanding on the barrier: whoever issues for it issues nothing more and waits
// for nothing, so that the loops run to their end on data that nobody uses, and the CTA waits
// for it once more before it exits.
constexpr uint32_t kWaitLimit = 1u << 18;
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* pending, int* fail) {
  for (uint32_t i = 0; i < kWaitLimit; ++i)
    if (mbar_try(bar, parity)) return true;
  *pending = 1 + (int)parity;
  *(volatile int*)fail = 1;
  __threadfence_system();
  return false;
}

__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// contiguous copy into shared memory (16-byte aligned, a multiple of 16 bytes); bytes counted on `bar`
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// one thread of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok));
  return ok != 0;
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mma_i8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
// 32 consecutive columns (4 outputs' digits) of this thread's lane
__device__ __forceinline__ void tmem_load32(uint32_t addr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr)
      : "memory");
}
// K-major operand with the 128-byte swizzle: 128-byte row segments, groups of 8 rows
// 1024 bytes apart; a segment's 16-byte chunk c of row r sits at chunk c ^ (r & 7).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)2 << 61;
}
// u8 x u8 -> s32, M = 128, N columns
__host__ __device__ constexpr uint32_t i8_idesc(uint32_t n) { return 2u << 4 | (n >> 3) << 17 | (128u >> 4) << 24; }

// ------------------------------------------------------------------ the kernel
constexpr int kRows = 128;          // rows of a tile: lanes x R1 = lanes x chunk

// A [128 x 32 KS bytes] times B [N x 32 KS bytes]^T into N accumulator columns, by one
// thread of a warp; `bar` gets the completion
template <int KS, int N>
__device__ __forceinline__ void issue(uint32_t d, uint32_t a, uint32_t b, uint32_t bar) {
  tc_fence_after();
  if (elect_one()) {
#pragma unroll
    for (int ks = 0; ks < KS; ++ks)
      mma_i8(d, smem_desc(a + (ks >> 2) * (kRows * 128) + (ks & 3) * 32),
             smem_desc(b + (ks >> 2) * (N * 128) + (ks & 3) * 32), i8_idesc(N), ks > 0);
    mma_commit(bar);
  }
  __syncwarp();
}

// PT (pass twiddle of a four-step transform's first pass): 0 none, canonical results; 1 formed
// as a geometric sequence; 2 from tables of the tile's lanes, shared by many columns
template <int LR1, int LR2, int PT>
struct Shape {
  static constexpr int R1 = 1 << LR1, R2 = 1 << LR2;
  static constexpr int L = kRows / R1;                                     // lanes of a tile
  static constexpr int GROUPS = 2;
  static constexpr int PARTS = LR1 == 5 ? 4 : 2;    // warps of a group per TMEM lane quarter
  static constexpr int GT = 128 * PARTS;            // threads of a group
  static constexpr int T = GROUPS * GT;
  static constexpr int OUT = R1 / PARTS;            // outputs of a thread, either stage
  static constexpr int COLS = 8 * R1;                                      // accumulator columns (both stages)
  static constexpr uint32_t A_BYTES = kRows * 8 * (R1 > R2 ? R1 : R2);     // operand A, either stage
  static constexpr uint32_t B1_BYTES = 8 * R1 * 8 * R2, B2_BYTES = 8 * R1 * 8 * R1;
  static constexpr uint32_t T_BYTES = R1 * R1 * 8;
  static constexpr uint32_t Q_BYTES = B1_BYTES + T_BYTES;                  // a chunk's tables
  // twiddles in shared memory: the chunk's [x][m1], or for PT = 2 [x][row] times w_N^(j' lane)
  // and the factors w_N^(S i1 lane) at [i1][l]
  static constexpr uint32_t TW_BYTES = PT == 2 ? kRows * R1 * 8 + L * R1 * 8 : T_BYTES;
  static constexpr uint32_t SMEM = B2_BYTES + B1_BYTES + TW_BYTES + GROUPS * A_BYTES + 64 + 1024;
};

// byte matrix entries of one (output, input) pair: out[d] byte b = byte d of v 2^(8b) mod p
__device__ __forceinline__ void digit_words(uint64_t v, uint64_t* out) {
  uint32_t lo[8], hi[8];
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    lo[b] = (uint32_t)v;
    hi[b] = (uint32_t)(v >> 32);
    v = gl::mul2e(v, 8);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t* w = h ? hi : lo;
    uint32_t t[2][4];
#pragma unroll
    for (int g = 0; g < 2; ++g) {  // 4 x 4 byte transposes of w[4g .. 4g+3]
      const uint32_t a = __byte_perm(w[4 * g], w[4 * g + 1], 0x5140), b = __byte_perm(w[4 * g], w[4 * g + 1], 0x7362);
      const uint32_t c = __byte_perm(w[4 * g + 2], w[4 * g + 3], 0x5140),
                     d = __byte_perm(w[4 * g + 2], w[4 * g + 3], 0x7362);
      t[g][0] = __byte_perm(a, c, 0x5410);
      t[g][1] = __byte_perm(a, c, 0x7632);
      t[g][2] = __byte_perm(b, d, 0x5410);
      t[g][3] = __byte_perm(b, d, 0x7632);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) out[4 * h + k] = (uint64_t)t[1][k] << 32 | t[0][k];
  }
}

// row (output x, digit d), input m of a byte matrix of N rows
__device__ __forceinline__ void store_digits(char* mat, int n_rows, int x, int m, uint64_t v) {
  uint64_t w[8];
  digit_words(v, w);
  char* p = mat + (m >> 4) * (n_rows * 128) + x * 1024 + (m & 1) * 8;
  const int c = (m & 15) >> 1;
#pragma unroll
  for (int d = 0; d < 8; ++d) *(uint64_t*)(p + d * 128 + ((c ^ d) << 4)) = w[d];
}

// tile row of (lane l, index x): lanes apart (LF = false: a warp's rows are one or two
// lanes' consecutive x, so its global accesses run along x), or lanes together (LF: a
// half-warp has all L lanes of 16 / L values of x, so that its global accesses are whole
// 8 L-byte pieces). For LF the low row bits are the lane's, so that a half-warp's
// column-wise stores into the 128-byte swizzle (16 bytes at chunk ^ (row & 7)) touch
// every bank once.
template <int L, int R, bool LF>
__device__ __forceinline__ void row_split(int r, int* l, int* x) {
  if constexpr (!LF) {
    *l = r / R;
    *x = r % R;
  } else if constexpr (L == 4) {
    *x = (r >> 3) * 2 + (r & 1);
    *l = (r >> 1) & 3;
  } else {
    *x = r >> 3;
    *l = r & 7;
  }
}
template <int L, int R, bool LF>
__device__ __forceinline__ constexpr int row_of(int l, int x) {
  if constexpr (!LF)
    return l * R + x;
  else if constexpr (L == 4)
    return (x >> 1) * 8 + l * 2 + (x & 1);
  else
    return x * 8 + l;
}

template <int LR1, int LR2, bool LF, int PT>
__global__ void __launch_bounds__(Shape<LR1, LR2, PT>::T, LR1 == 4 && LR2 == 4 ? 2 : 1) ntt_tc_kernel(TcPass a) {
  using S = Shape<LR1, LR2, PT>;
  constexpr int R1 = S::R1, R2 = S::R2, L = S::L, PARTS = S::PARTS, OUT = S::OUT;
  constexpr int NE = R2 / PARTS;  // input elements a thread loads
  extern __shared__ char raw[];
  char* base = raw + ((1024 - (smem_u32(raw) & 1023)) & 1023);
  char* b2 = base;
  char* b1 = b2 + S::B2_BYTES;
  uint64_t* tw = (uint64_t*)(b1 + S::B1_BYTES);
  uint64_t* tw_lane = tw + kRows * R1;  // (PT = 2)
  char* a_all = (char*)tw + S::TW_BYTES;
  char* tail = a_all + S::GROUPS * S::A_BYTES;
  uint32_t* tmem_slot = (uint32_t*)tail;
  // (mbar_wait) a group's products, then the tables
  volatile int* pending = (volatile int*)(tail + 4);
  const uint32_t bars = smem_u32(tail + 16), tab_bar = bars + 8 * S::GROUPS;
  // the warp's number through a shuffle, so that what depends on it alone is uniform
  const int t = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, t >> 5, 0), grp = warp / (4 * PARTS);
  const int gw = warp % (4 * PARTS);  // warp within the group
  const int row = (gw & 3) * 32 + (t & 31), part = gw >> 2;
  const uint32_t bar = bars + 8 * grp;
  // this group's operand A, both stages in place
  const uint32_t at_u = smem_u32(a_all + grp * S::A_BYTES), b1_u = smem_u32(b1), b2_u = smem_u32(b2);

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(S::GROUPS * S::COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (t == 0) {
    for (int g = 0; g <= S::GROUPS; ++g) {
      pending[g] = 0;
      mbar_init(bars + 8 * g, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot + grp * S::COLS;
  const uint32_t tmem_row = tmem + ((uint32_t)((gw & 3) * 32) << 16) + 8 * (gw >> 2) * OUT;

  int l, m1;  // stage 1: this thread's row; stage 2: (l, x2)
  row_split<L, R1, LF>(row, &l, &m1);
  const int l2 = l, x2 = m1;  // chunk = R1 values of j': the same split
  const int i0 = part * OUT;  // this thread's outputs i0 .. i0 + OUT - 1, either stage
  // first-stage results of this thread go to column m1 of rows (l, i0 ..)
  const int r0 = row_of<L, R1, LF>(l, i0);
  const uint32_t st_u =
      at_u + (m1 >> 4) * (kRows * 128) + r0 * 128 + (m1 & 1) * 8 + ((((m1 & 15) >> 1) ^ (r0 & 7)) << 4);
  // input elements m2 = 2c and 2c + 1, c = part + PARTS i, go to 16-byte chunk c of this thread's row
  const uint32_t ld_u = at_u + row * 128 + ((part ^ (row & 7)) << 4);
  // (block layouts only with lanes together)
  const char* in_t = LF ? at(at(a.in, m1 >> a.in_blog, a.in_hb), m1 & ((1u << a.in_blog) - 1), a.in_mb)
                        : at(a.in, m1, a.in_mb);
  in_t = at(in_t, 2 * part, a.in_step);
  char* out_t = at(at(a.out, x2, a.out_xb), i0, a.out_step);
  constexpr int TS = PT == 2 ? kRows : R1;  // stride of the first-stage twiddles
  const uint64_t* tw_t = tw + i0 * TS + (PT == 2 ? row : m1);

  // Tiles (chunk q, column y, lane group g) go in pairs, one to each group.
  // PT = 2: a unit is a chunk, a lane group and a range of columns; a CTA takes every
  // gridDim-th unit (CTAs that run together touch neighbouring lanes together) and its pairs
  // are neighbouring columns. Otherwise a unit is a chunk, pairs run over lane groups, then
  // columns, and a CTA has a contiguous range of pairs (few changes of chunk) or every
  // gridDim-th pair.
  const uint32_t lgroups = a.lgroups, per_q = a.lgroups * a.n_y, pairs_q = (per_q + 1) / 2;
  const uint32_t pairs = PT == 2 ? a.n_q * lgroups * a.y_parts : pairs_q * a.n_q;
  uint32_t pair, pair_end, step;
  if (PT == 2 || a.strided) {
    pair = blockIdx.x;
    pair_end = pairs;
    step = gridDim.x;
  } else {
    pair = (uint32_t)((uint64_t)pairs * blockIdx.x / gridDim.x);
    pair_end = (uint32_t)((uint64_t)pairs * (blockIdx.x + 1) / gridDim.x);
    step = 1;
  }
  const uint32_t gstep = PT == 2 ? S::GROUPS : S::GROUPS * step;
  const uint32_t gstep_y = PT == 2 ? S::GROUPS : gstep / lgroups, gstep_g = PT == 2 ? 0 : gstep % lgroups;
  uint32_t phase = 0, tab_phase = 0;
  uint32_t q_loaded = ~0u;
  uint64_t x[NE];

  // Lanes past the last are done as copies of the last one (same loads, same stores).
  const uint32_t last_lane = a.n_lanes - 1, c8 = a.c8, c16 = a.c16;
  auto load_tile = [&](uint32_t y, uint32_t g) {
    const uint32_t lane = min(g * L + l, last_lane);
    const char* src = at(in_t, y, a.in_colb);
    src = LF ? at(at(src, g, a.in_gb), lane - g * L, a.in_laneb) : at(src, lane, a.in_laneb);
    if (!a.masked) {
#pragma unroll
      for (int i = 0; i < NE; ++i) {
        const int m2 = 2 * PARTS * (i >> 1) + (i & 1);  // + 2 part
        x[i] = __ldg(!LF ? (const uint64_t*)src + m2 * R1 : (const uint64_t*)at(src, m2, a.in_step));
      }
    } else {
      const uint64_t flat0 = lane * a.flat_lane + (uint64_t)(m1 + 2 * part * R1) * a.flat_m;
#pragma unroll
      for (int i = 0; i < NE; ++i) {
        const int m2 = 2 * PARTS * (i >> 1) + (i & 1);
        x[i] = flat0 + (uint64_t)(m2 * R1) * a.flat_m < a.in_valid ? __ldg((const uint64_t*)at(src, m2, a.in_step)) : 0;
      }
    }
  };

  // the group's first warp issues its products and polls for them (until one fails to come), the
  // others wait at the group's barrier
  bool lead = gw == 0;
  auto wait_group = [&](uint32_t b, uint32_t parity) {
    if (lead) lead = __all_sync(0xFFFFFFFFu, mbar_wait(b, parity, pending + grp, a.fail));
    bar_group(1 + grp, S::GT);
    tc_fence_after();
  };

  while (pair < pair_end) {
    uint32_t q, it, it_end, y, g;
    if constexpr (PT == 2) {
      const uint32_t per = lgroups * a.y_parts, r = pair % per;
      q = pair / per;
      g = r % lgroups;
      y = r / lgroups * a.y_len;
      it_end = min(y + a.y_len, a.n_y);
      it = y += grp;
      pair += step;
    } else {
      q = pair / pairs_q;
      const uint32_t p0 = q * pairs_q, p_end = min(p0 + pairs_q, pair_end);
      it = 2 * (pair - p0) + grp;  // within the chunk
      it_end = min(2 * (p_end - p0), per_q);
      y = it / lgroups;
      g = it % lgroups;
      pair += (p_end - pair + step - 1) / step * step;
    }
    // the chunk's first-stage matrix and twiddles (and once the second-stage matrix)
    if (q_loaded != ~0u) {
      fence_async_smem();
      __syncthreads();
    }
    const char* q_tab = a.tab + S::B2_BYTES + (uint64_t)q * S::Q_BYTES;
    if (q != q_loaded) {
      if (t == 0 && pending[S::GROUPS] == 0) {
        const uint32_t bytes = PT == 2 ? S::B1_BYTES : S::Q_BYTES;
        mbar_expect(tab_bar, bytes + (q_loaded == ~0u ? S::B2_BYTES : 0));
        if (q_loaded == ~0u) bulk_load(b2_u, a.tab, S::B2_BYTES, tab_bar);
        bulk_load(b1_u, q_tab, bytes, tab_bar);
      }
    }
    if (it < it_end) load_tile(y, g);
    if constexpr (PT == 2) {
      // w_EM^(j' m1) w_N^(j' lane) g^(m1 + lane) of every row, and w_N^(S i1 lane)
      const uint64_t* q_tw = (const uint64_t*)(q_tab + S::B1_BYTES);
      for (int e = t; e < kRows * R1; e += S::T) {
        const int r = e % kRows, xx = e / kRows;
        int ll, mm;
        row_split<L, R1, LF>(r, &ll, &mm);
        const uint64_t lane = (uint64_t)g * L + ll, j = a.j0 + (uint64_t)q * a.jq + (uint64_t)xx * a.jx;
        uint64_t v = gl::mul(__ldg(q_tw + xx * R1 + mm), tw_pow(a.tw_lo, a.tw_hi, j * lane, a.pt_log));
        if (a.pre.active()) v = gl::mul(v, pow_at(a.pre, lane * a.flat_lane));
        tw[e] = v;
      }
      for (int e = t; e < L * R1; e += S::T)
        tw_lane[e] = tw_pow(a.tw_lo, a.tw_hi, ((uint64_t)(e / L) * ((uint64_t)g * L + e % L)) << a.log_s, a.pt_log);
      __syncthreads();
    }
    if (q != q_loaded) {
      if (pending[S::GROUPS] == 0) mbar_wait(tab_bar, tab_phase, pending + S::GROUPS, a.fail);
      if (lead) lead = __all_sync(0xFFFFFFFFu, pending[S::GROUPS] == 0);
      tab_phase ^= 1;
      q_loaded = q;
    }
    char* out_q = out_t + q * a.out_q * 8;
    for (; it < it_end; it += gstep) {
      // operand A of the first stage
#pragma unroll
      for (int i = 0; i < NE / 2; ++i) {
        const int c = PARTS * i;  // + part
        const uint32_t p = (ld_u ^ ((c & 7) << 4)) + (c >> 3) * (kRows * 128);
        asm volatile("st.shared.v2.u64 [%0], {%1, %2};" ::"r"(p), "l"(x[2 * i]), "l"(x[2 * i + 1]) : "memory");
      }
      fence_async_smem();
      tc_fence_before();
      bar_group(1 + grp, S::GT);
      if (lead) issue<R2 / 4, 8 * R1>(tmem, at_u, b1_u, bar);
      const uint32_t lane = min(g * L + l2, last_lane);
      char* o = at(out_q, y, a.out_colb);
      o = LF ? at(at(o, g, a.out_gb), lane - g * L, a.out_laneb) : at(o, lane, a.out_laneb);
      y += gstep_y;
      g += gstep_g;
      if (PT != 2 && g >= lgroups) {
        g -= lgroups;
        ++y;
      }
      if (it + gstep < it_end) load_tile(y, g);
      wait_group(bar, phase);
      phase ^= 1;
      // digits -> element, twiddle, column m1 of the second stage's rows
#pragma unroll
      for (int k = 0; k < OUT / 4; ++k) {
        uint32_t d[32];
        tmem_load32(tmem_row + 32 * k, d);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint64_t v = gl::mul_any(join_digits(d + 8 * u, c8, c16), tw_t[(4 * k + u) * TS]);
          // row_of(l, i0 + x) = row_of(l, i0) + row_of(0, x), low three bits without carries
          const int ro = row_of<L, R1, LF>(0, 4 * k + u);
          const uint32_t p = (st_u ^ ((ro & 7) << 4)) + ro * 128;
          asm volatile("st.shared.u64 [%0], %1;" ::"r"(p), "l"(v) : "memory");
        }
      }
      fence_async_smem();
      tc_fence_before();
      bar_group(1 + grp, S::GT);
      if (lead) issue<R1 / 4, 8 * R1>(tmem, at_u, b2_u, bar);
      uint64_t f = 0, rho = 0;
      if constexpr (PT == 1) {  // w_N^((j' + S i1) lane) g^lane as a geometric sequence in i1
        rho = tw_pow(a.tw_lo, a.tw_hi, (uint64_t)lane << a.log_s, a.pt_log);
        const uint64_t j = a.j0 + (uint64_t)q * a.jq + (uint64_t)x2 * a.jx + ((uint64_t)i0 << a.log_s);
        f = tw_pow(a.tw_lo, a.tw_hi, j * lane, a.pt_log);
        if (a.pre.active()) f = gl::mul(f, pow_at(a.pre, (uint64_t)lane * a.flat_lane));
      }
      wait_group(bar, phase);
      phase ^= 1;
#pragma unroll
      for (int k = 0; k < OUT / 4; ++k) {
        uint32_t d[32];
        tmem_load32(tmem_row + 32 * k, d);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          uint64_t v = join_digits(d + 8 * u, c8, c16);
          if constexpr (PT == 1) {
            v = gl::mul_any(v, f);
            f = gl::mul_any(f, rho);
          }
          if constexpr (PT == 2) v = gl::mul_any(v, tw_lane[(i0 + 4 * k + u) * L + l2]);
          if (PT == 0 || a.canon) v = canonical(v);
          *(uint64_t*)at(o, 4 * k + u, a.out_step) = v;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    // what was given up has its time once more to finish, before its memory is given back
    if (t <= S::GROUPS && pending[t] != 0) {
      for (uint32_t i = 0; i < kWaitLimit && !mbar_try(bars + 8 * t, pending[t] - 1); ++i) {
      }
    }
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*tmem_slot), "r"(S::GROUPS * S::COLS));
  }
}

template <int LR1, int LR2, bool LF, int PT>
cudaError_t launch(TcPass a, cudaStream_t s) {
  using S = Shape<LR1, LR2, PT>;
  auto kern = ntt_tc_kernel<LR1, LR2, LF, PT>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
  if (e != cudaSuccess) return e;
  const uint64_t lgroups = (a.n_lanes + S::L - 1) / S::L, fit = 148 * (LR1 == 4 && LR2 == 4 ? 2 : 1);
  const uint64_t in_m2 = a.in_block ? S::R1 / a.in_block * a.in_h : S::R1 * a.in_m;
  const uint64_t in_g = a.in_g ? a.in_g : S::L * a.in_lane, out_g = a.out_g ? a.out_g : S::L * a.out_lane;
  // the kernel's strides are 32-bit byte counts
  const uint64_t strides[] = {in_m2, in_g, a.in_col, a.in_h, a.out_i, a.out_x, out_g, a.out_col};
  for (uint64_t v : strides)
    if (v >= 1ull << 29) return cudaErrorInvalidValue;
  a.lgroups = (uint32_t)lgroups;
  a.in_blog = 31;
  if (a.in_block)
    for (a.in_blog = 0; (1u << a.in_blog) < a.in_block;) ++a.in_blog;
  a.in_mb = (uint32_t)(a.in_m * 8);
  a.in_hb = (uint32_t)(a.in_h * 8);
  a.in_step = (uint32_t)(in_m2 * 8);
  a.in_laneb = (uint32_t)(a.in_lane * 8);
  a.in_gb = (uint32_t)(in_g * 8);
  a.in_colb = (uint32_t)(a.in_col * 8);
  a.out_xb = (uint32_t)(a.out_x * 8);
  a.out_step = (uint32_t)(a.out_i * 8);
  a.out_laneb = (uint32_t)(a.out_lane * 8);
  a.out_gb = (uint32_t)(out_g * 8);
  a.out_colb = (uint32_t)(a.out_col * 8);
  a.masked = a.in_valid <= (a.n_lanes - 1) * a.flat_lane + (uint64_t)(S::R1 * S::R2 - 1) * a.flat_m;
  a.c8 = 1u << 8;
  a.c16 = 1u << 16;
  // a CTA takes up to 24 pairs of tiles (about 100 us), so that CTAs of a higher-priority
  // stream get in between
  uint64_t units, pairs;
  if (PT == 2) {
    // column ranges of at least 8 columns, as many as it takes to fill whole waves of CTAs
    uint32_t parts = 1;
    while ((a.n_y + 2 * parts - 1) / (2 * parts) >= 8 && parts < 16) {
      const uint64_t u = lgroups * a.n_q * parts;
      if (u * 100 >= (u + fit - 1) / fit * fit * 93) break;
      parts *= 2;
    }
    a.y_len = (a.n_y + parts - 1) / parts;
    a.y_parts = (a.n_y + a.y_len - 1) / a.y_len;
    units = lgroups * a.n_q * a.y_parts;
    pairs = units * ((a.y_len + 1) / 2);
  } else {
    units = pairs = (lgroups * a.n_y + 1) / 2 * a.n_q;
  }
  if (pairs >= 1ull << 30 || lgroups * a.n_y >= 1ull << 30) return cudaErrorInvalidValue;
  const uint64_t waves = (pairs + 24 * fit - 1) / (24 * fit);
  const uint64_t grid = std::min(units, waves * fit);
  SG_LAUNCH_SCOPE("ntt_pass", s);
  kern<<<(unsigned)grid, S::T, S::SMEM, s>>>(a);
  return cudaGetLastError();
}

template <int LR1, int LR2>
cudaError_t launch_mode(const TcPass& a, bool lanes_fast, int pt, cudaStream_t s) {
  if (pt == 1) return launch<LR1, LR2, true, 1>(a, s);
  if (pt == 2) return launch<LR1, LR2, true, 2>(a, s);
  return lanes_fast ? launch<LR1, LR2, true, 0>(a, s) : launch<LR1, LR2, false, 0>(a, s);
}

// ------------------------------------------------------------------ tables
// Image of a pass: the second-stage matrix w_R1^(i1 m1), then per chunk q the first-stage
// matrix w_S^(j' m2) g^(R1 m2) scale and the twiddles w_EM^(j' m1) g^(m1) at [x][m1],
// j' = q jq + x jx, matrices as they lie in shared memory.
struct PrepArgs {
  char* out;
  int lr1, lr2, log_s;
  uint32_t n_q, j0, jq, jx;
  uint64_t flat_m, scale;
  PowSpec pre;
  const uint64_t *lo, *hi;
};
__global__ void __launch_bounds__(256) tc_prep_kernel(PrepArgs a) {
  const int R1 = 1 << a.lr1, R2 = 1 << a.lr2;
  const uint64_t n2 = (uint64_t)R1 * R1, n1 = (uint64_t)R1 * R2;
  const uint64_t q_bytes = 64 * n1 + 8 * n2, total = n2 + a.n_q * (n1 + n2);
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < total;
       e += (uint64_t)gridDim.x * blockDim.x) {
    if (e < n2) {
      const int m = (int)(e & (R1 - 1)), x = (int)(e >> a.lr1);
      store_digits(a.out, 8 * R1, x, m, tw_pow(a.lo, a.hi, (uint64_t)(m * x), a.lr1));
      continue;
    }
    const uint64_t q = (e - n2) / (n1 + n2), r = (e - n2) - q * (n1 + n2);
    char* o = a.out + 64 * n2 + q * q_bytes;
    if (r < n1) {
      const int m = (int)(r & (R2 - 1)), x = (int)(r >> a.lr2);
      uint64_t v = tw_pow(a.lo, a.hi, (a.j0 + q * a.jq + (uint64_t)x * a.jx) * m, a.log_s);
      if (a.pre.active()) v = gl::mul(v, pow_at(a.pre, ((uint64_t)m << a.lr1) * a.flat_m));
      if (a.scale != 1) v = gl::mul(v, a.scale);
      store_digits(o, 8 * R1, x, m, v);
    } else {
      const int m = (int)((r - n1) & (R1 - 1)), x = (int)((r - n1) >> a.lr1);
      uint64_t v = tw_pow(a.lo, a.hi, (a.j0 + q * a.jq + (uint64_t)x * a.jx) * m, a.log_s + a.lr1);
      if (a.pre.active()) v = gl::mul(v, pow_at(a.pre, (uint64_t)m * a.flat_m));
      ((uint64_t*)(o + 64 * n1))[x * R1 + m] = v;
    }
  }
}

uint64_t image_bytes(int lr1, int lr2, uint32_t n_q) {
  const uint64_t n2 = 1ull << (2 * lr1), n1 = 1ull << (lr1 + lr2);
  return 64 * n2 + n_q * (64 * n1 + 8 * n2);
}

}  // namespace

int ntt_tc_lanes(int log_m) { return log_m == 10 ? 4 : 8; }

bool ntt_tc_ok(int log_m) { return log_m >= 8 && log_m <= 10; }

TcPass ntt_tc_args(int log_m, int log_e) {
  TcPass a{};
  a.log_m = log_m;
  if (!ntt_tc_ok(log_m)) return a;
  const int lr1 = log_m == 10 ? 5 : 4;
  a.n_y = 1;
  a.log_s = log_e + log_m - lr1;
  a.n_q = 1u << (a.log_s - lr1);
  a.jq = 1u << lr1;
  a.jx = 1;
  a.flat_m = 1;
  a.scale = 1;
  return a;
}

// Tables that depend on the shape alone are kept with the context's twiddle tables and
// shared by the contexts that borrow those: at most kCacheBytes; a later stream waits
// for the event of the stream that built them.
constexpr uint64_t kCacheBytes = 64ull << 20;
struct TcCache {
  struct Entry {
    char* d = nullptr;
    cudaEvent_t ready = nullptr;
    bool done = false;
  };
  std::mutex mu;
  std::map<std::tuple<int, int, uint32_t, uint32_t, uint32_t, uint32_t, bool, uint64_t>, Entry> map;
  uint64_t bytes = 0;
};
TcCache* tc_cache_new() { return new (std::nothrow) TcCache; }
void tc_cache_free(TcCache* c) {
  if (!c) return;
  for (auto& kv : c->map) {
    cudaFree(kv.second.d);
    cudaEventDestroy(kv.second.ready);
  }
  delete c;
}

static cudaError_t build(const NttTables& t, const TcPass& a, bool inverse, char* d, cudaStream_t s) {
  const int lr1 = a.log_m == 10 ? 5 : 4, lr2 = a.log_m - lr1;
  PrepArgs p{d, lr1, lr2, a.log_s, a.n_q, a.j0, a.jq, a.jx, a.flat_m, a.scale, a.pre,
             inverse ? t.d_inv_lo : t.d_fwd_lo, inverse ? t.d_inv_hi : t.d_fwd_hi};
  const uint64_t total = (1ull << (2 * lr1)) + a.n_q * ((1ull << (2 * lr1)) + (1ull << a.log_m));
  SG_LAUNCH_SCOPE("ntt_tables", s);
  tc_prep_kernel<<<(unsigned)std::min<uint64_t>((total + 255) / 256, 148 * 8), 256, 0, s>>>(p);
  return cudaGetLastError();
}

// False (and *a unchanged) when there is no room for the tables.
bool ntt_tc_tables(const NttTables& t, TcPass* a, bool inverse, cudaStream_t s) {
  if (!t.tc || !t.fail || t.no_room || !ntt_tc_ok(a->log_m)) return false;
  const int lr1 = a->log_m == 10 ? 5 : 4, lr2 = a->log_m - lr1;
  const uint64_t bytes = image_bytes(lr1, lr2, a->n_q);
  if (bytes > kCacheBytes) return false;
  a->tw_lo = inverse ? t.d_inv_lo : t.d_fwd_lo;
  a->tw_hi = inverse ? t.d_inv_hi : t.d_fwd_hi;
  a->fail = t.fail;
  if (!a->pre.active()) {
    std::lock_guard<std::mutex> g(t.tc->mu);
    const auto key = std::make_tuple(a->log_m, a->log_s, a->n_q, a->j0, a->jq, a->jx, inverse, a->scale);
    auto it = t.tc->map.find(key);
    if (it != t.tc->map.end()) {
      TcCache::Entry& e = it->second;
      if (!e.done) {
        if (cudaEventQuery(e.ready) == cudaSuccess)
          e.done = true;
        else if (cudaStreamWaitEvent(s, e.ready, 0) != cudaSuccess)
          return false;
      }
      a->tab = e.d;
      return true;
    }
    if (t.tc->bytes + bytes <= kCacheBytes) {
      TcCache::Entry e;
      if (cudaMallocAsync((void**)&e.d, bytes, s) != cudaSuccess) {
        cudaGetLastError();
        return false;
      }
      if (cudaEventCreateWithFlags(&e.ready, cudaEventDisableTiming) != cudaSuccess ||
          build(t, *a, inverse, e.d, s) != cudaSuccess || cudaEventRecord(e.ready, s) != cudaSuccess) {
        cudaGetLastError();
        if (e.ready) cudaEventDestroy(e.ready);
        cudaFreeAsync(e.d, s);
        return false;
      }
      t.tc->bytes += bytes;
      t.tc->map[key] = e;
      a->tab = e.d;
      return true;
    }
  }
  // this call's own tables, freed in stream order by ntt_tc_pass
  char* d = nullptr;
  if (cudaMallocAsync((void**)&d, bytes, s) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (build(t, *a, inverse, d, s) != cudaSuccess) {
    cudaGetLastError();
    cudaFreeAsync(d, s);
    return false;
  }
  a->tab = d;
  a->own_tab = true;
  return true;
}

// Words for contexts, 1024 (a page) allocated at a time and kept for the process: contexts
// (a server's workers) come and go.
namespace {
struct FailWords {
  std::mutex mu;
  std::vector<int*> free;
};
FailWords& fail_words() {
  static FailWords* w = new FailWords;
  return *w;
}
}  // namespace

int* ntt_tc_fail_new() {
  FailWords& w = fail_words();
  std::lock_guard<std::mutex> g(w.mu);
  if (w.free.empty()) {
    int* p = nullptr;
    constexpr int kWords = 1024;
    if (cudaHostAlloc((void**)&p, kWords * sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    for (int i = kWords - 1; i >= 0; --i) w.free.push_back(p + i);
  }
  int* p = w.free.back();
  w.free.pop_back();
  *p = 0;
  return p;
}

void ntt_tc_fail_free(int* p) {
  if (!p) return;
  FailWords& w = fail_words();
  std::lock_guard<std::mutex> g(w.mu);
  w.free.push_back(p);
}

void ntt_tc_drop(const TcPass& a, cudaStream_t s) {
  if (a.own_tab) cudaFreeAsync((void*)a.tab, s);
}

cudaError_t ntt_tc_pass(const TcPass& a, bool lanes_fast, cudaStream_t s) {
  if (!ntt_tc_ok(a.log_m) || !a.tab) return cudaErrorInvalidValue;
  if (a.n_lanes == 0 || a.n_y == 0 || a.n_q == 0) {
    ntt_tc_drop(a, s);
    return cudaSuccess;
  }
  // The lane tables of PT = 2 cost about as much as a pair of tiles, so they are shared by at
  // least 8 columns, and there have to be two waves of such units. Inverse transforms with
  // them and without: 8 x 2^20 157 and 149 us, 32 x 2^20 491 and 500, 64 x 2^20 910 and 962; 16
  // x 2^18 79 and 76, 64 x 2^18 235 and 238, 320 x 2^18 969 and 1037; 80 x 2^16 78 and 78, 320
  // x 2^16 222 and 222. (From two to some four waves they cost up to 6 %, 16 x 2^20 282 and 266.)
  const uint64_t units = (uint64_t)(a.n_lanes / ntt_tc_lanes(a.log_m)) * a.n_q * (a.n_y / 8);
  const int pt = a.pt_log == 0 ? 0 : units < 2 * 148 * (a.log_m == 8 ? 2 : 1) ? 1 : 2;
  cudaError_t e = cudaErrorInvalidValue;
  if (!pt || lanes_fast) switch (a.log_m) {
      case 8: e = launch_mode<4, 4>(a, lanes_fast, pt, s); break;
      case 9: e = launch_mode<4, 5>(a, lanes_fast, pt, s); break;
      default: e = launch_mode<5, 5>(a, lanes_fast, pt, s);
    }
  ntt_tc_drop(a, s);
  return e;
}

}  // namespace sg
