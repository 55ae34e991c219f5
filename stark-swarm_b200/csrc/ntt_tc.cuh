// ntt_tc.cuh — one NTT pass of M = 2^8 .. 2^10 points on the int8 tensor cores (ntt_tc.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "ntt.cuh"

namespace sg {

// n_y outer columns of n_lanes independent transforms of M = R1 R2 points, each giving
// E M outputs j = j' + S i1 (S = E R2 = 2^log_s, i1 < R1) in n_q chunks of R1 values of j':
// j' = j0 + q jq + x jx (adjacent ones, or with jx = E a coset's). R1 = 16 for M = 2^8 and 2^9, 32 for 2^10.
//   input  (y, lane, m):      in + y in_col + lane in_lane + m in_m
//   output (y, lane, q, x, i1): out + y out_col + lane out_lane + q out_q + x out_x + i1 out_i
// Inputs at flat index m flat_m + lane flat_lane >= in_valid are zero; pre multiplies
// by g^(flat index). The result is sum_m x[m] w_EM^(jm) scale, times w_(2^pt_log)^(j lane) if
// pt_log > 0 (then any u64 of its residue class unless canon, for a next pass; else canonical).
struct TcPass {
  const uint64_t* in;
  uint64_t* out;
  uint64_t in_col, out_col, in_lane, in_m, out_lane, out_q, out_x, out_i;
  // optional layouts in blocks: lane groups (a tile's lanes, ntt_tc_lanes) at their own stride, and
  // input points m at m / in_block * in_h + m % in_block * in_m
  uint64_t in_g, out_g, in_h;
  uint32_t in_block;
  uint32_t n_lanes, n_y, n_q, j0, jq, jx;
  uint64_t flat_m, flat_lane, in_valid;
  int log_m, log_s, pt_log;
  uint64_t scale;
  PowSpec pre;
  bool canon;    // with pt_log: canonical results all the same
  bool strided;  // CTAs take every gridDim-th pair of tiles (neighbouring lanes at the same time) instead of a range
  // filled in by ntt_tc_tables and ntt_tc_pass
  const char* tab;
  const uint64_t *tw_lo, *tw_hi;
  int* fail;
  uint32_t lgroups, y_parts, y_len, in_blog, in_step, in_mb, in_hb, in_laneb, in_gb, in_colb;
  uint32_t out_step, out_xb, out_laneb, out_gb, out_colb, c8, c16;
  bool masked, own_tab;
};

bool ntt_tc_ok(int log_m);
int ntt_tc_lanes(int log_m);  // lanes of a tile
// the fields that follow from M = 2^log_m and E = 2^log_e (chunks of adjacent j'); the caller sets the rest
TcPass ntt_tc_args(int log_m, int log_e);
// The pass's byte matrices and twiddles (from pre, scale, flat_m, jq, jx and the shape), in
// stream order. False when the tables have no tensor-core cache or there is no room.
bool ntt_tc_tables(const NttTables& t, TcPass* a, bool inverse, cudaStream_t s);
// Frees the tables of a pass that will not run (ntt_tc_pass does it itself).
void ntt_tc_drop(const TcPass& a, cudaStream_t s);
// lanes_fast: a warp's accesses run over the lanes (in_lane or out_lane of 1) instead of along m and j'
cudaError_t ntt_tc_pass(const TcPass& a, bool lanes_fast, cudaStream_t s);
// A host-mapped word for NttTables::fail, zero (null: no memory for it), and its return once
// no kernel runs that might set it.
int* ntt_tc_fail_new();
void ntt_tc_fail_free(int* p);

TcCache* tc_cache_new();
void tc_cache_free(TcCache* c);

}  // namespace sg
