// Split-K contractions of the RI-K term on CTA pairs (tcgen05 cta_group::2), see tc_pair.cu.
#pragma once
#include <cstdint>

#include "ctx.cuh"

namespace cphf {

// A stack of operand planes, K-major rows of `ld` elements: plane t of depth d at
// p[t] + (d rows) ld (separate arrays), or with depth_stride > 0 at p[0] + ((t depth_stride + d) rows) ld.
// Columns at and beyond kext (0: the contraction's K) read as zero.
struct PairPlanes {
  const void* p[2];
  int64_t rows, ld, depth, depth_stride;
  int64_t kext = 0;
};

// out[m + ld_out n] += rowscale[m] colscale[n] (*scale) sum_{P < np} sum_{k < K} X_(x_off+P)[m, k] Y_P[n, k]
// m < M (X rows), n < N (Y rows); null scales: 1; exact slices: rowscale holds powers of two.
struct PairTerm {
  PairPlanes x, y;
  int64_t x_off;  // depth of X at P = 0
  int64_t np, M, N, K;
  const double* rowscale;
  const double* colscale;
  const float* scale;
  void* out;
  int64_t ld_out;
  int* err;
  int64_t x_row0 = 0;  // X row of m = 0
  int64_t y_k0 = 0;    // Y column of k = 0, a multiple of 8
  bool store = false;  // exact slices, one K range: out = the value (no accumulation)
  int64_t max_k = 0;   // split FP16, np > 1: products an FP32 accumulator sums at most (0: any number)
};

bool pair_available(int device);
// split FP16 planes (hi, lo; three products), FP32 out
void pair_split2(cphf_ctx* c, const PairTerm& t);
// exact BF16 slices (6: 21 products, 4: 10, 3: 6), FP64 out; K blocks of 32 per CTA pair (at most
// 96, the exactness bound of the FP32 group sums; 0: chosen)
constexpr int PAIR_EXACT_KB = 96;
void pair_exact(cphf_ctx* c, const PairTerm& t, int slices, int kb_per_cta);

}  // namespace cphf
