// FP64 GEMM on the tensor cores: exact BF16 digit products of fixed-point operand slices.
//
//   C(m, n) = alpha * sum_k A(m, k) B(k, n) + beta * C(m, n)
//
// GB300 retires about two DFMA per clock and SM (1.2 TFLOP/s), so the FP64 contractions of the
// response and of the Krylov solver are bound by that pipe.  The splitting of Ozaki, Ogita, Oishi
// and Rump (error-free transformation of a matrix product) moves them to the tensor pipe:
//
// Slices.  Every row of A and every column of B is scaled by a power of two 2^-e so that |v| < 1,
// rounded to F = round(v 2^BITS), BITS = 8 (S - 1) + 6, and cut into S balanced base-256 digits
// F = sum_t q_t 256^(S-1-t), |q_0| <= 64, q_t in [-128, 127], each exact in BF16.  With S = 8
// (62 bits) every FP64 element within 2^-9 of its row's maximum is represented exactly, all
// others to 2^-63 of the power of two above that maximum: an element 2^-40 of the maximum keeps 22 bits.
// The products of digits t + u <= S - 1 are formed (36 for S = 8); the seven pairs with t + u = 8
// that are dropped come to at most 7 2^-62 of the two powers of two a product (to 2^-62 for random digits).
// Accumulation.  Products of one weight g = t + u share one FP32 accumulator in TMEM (S x 64 of
// the 512 columns).  Over 64 k (more for the leading weights, group_kb) their integer sum stays
// below 2^23, so the FP32 sums are exact; then the epilogue adds them as integers into two 64-bit
// registers per element (weights 0-3 and 4-7).  The sum of these products over a K range is therefore
// exact and is rounded to FP64 once, at the end, with integer arithmetic (an FP64 instruction per
// element and group would cost more than the MMAs of a round); the sums of several K ranges (at
// most 64) are then added in FP64.
//
// Error: at most K 2^-57 max_k |A(m, k)| max_k |B(k, n)| (for random digits about sqrt(K) 2^-60 of
// it), plus a rounding per K range and per addition of ranges.  A chain of FMAs errs by ~2^-53 of sum |a||b|
// a step instead: the digits are the more accurate where that sum is above ~2^-9 of the maxima's product,
// the less accurate for an element whose large factors all meet small ones.
// Measured (max error / sum |a||b|; fixed point, FMAs):
// Gaussian 300 x 200 x 500: 1.1e-17, 2.4e-16; entries over 12 octaves, K = 36000: 4.7e-17, 1.1e-15;
// K = 17: 1.1e-16, 3.8e-16.  Where large entries of A meet small ones of B
// throughout (the Krylov basis, whose vectors shrink, and its growing coefficients; a triangular
// solve), GemmDesc::k_balance divides A(:, k) and multiplies B(k, :) by a power of two first.
//
// Kernel structure (one CTA per SM, 10 warps, tiles 128 x 64):
//   warp 0 lane 0 -- TMA producer: one 4-D load per operand and 32-wide K block brings all S
//                    planes (64B swizzle) into a two-stage ring;
//   warp 1        -- TMEM owner; lane 0 issues the MMAs, weight by weight, so that in the last
//                    block before a drain the accumulator of weight g is complete (and drained) while
//                    the MMAs of the weights after it still run, and needed again only when the
//                    next block reaches it: the drain costs the tensor pipe nothing;
//   warps 2-9     -- drain and epilogue: TMEM lane quarter warp & 3, column half (warp - 2) / 4.
// Persistent: a CTA walks the work items (tile, K range, batch) with a stride of the grid, so the
// loads and MMAs of the next item run while the epilogue rounds and writes the last one.
// The 128 x 64 tile reads 6 KB of shared memory per 32-clock MMA, so the loop is bound by the
// shared-memory read rate (128 B/clk) at two thirds of the tensor rate; a 128-wide tile would
// need 1024 TMEM columns.
// Every mbarrier wait is bounded; on expiry the kernel raises the error flag and returns.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

#include "common.cuh"
#include "gemm_fx.cuh"
#include "tc_map.cuh"
#include "tc_ptx.cuh"

namespace cphf {
namespace {
using namespace tcx;

constexpr int BM = 128, BN = 64, BK = 32;
constexpr int ROUND_KB = 2;  // K blocks per drain of the longest sums (64 k)
constexpr int SPLIT_KB = 4;  // K ranges in multiples of 128 k
constexpr int THREADS = 320, EPI_WARPS = 8;
constexpr int A_TILE = BM * BK * 2, B_TILE = BN * BK * 2;

constexpr int S = 8;                   // digits
constexpr int BITS = 8 * (S - 1) + 6;  // of the fixed-point numbers
constexpr int STAGES = 2;
constexpr int STAGE_BYTES = S * (A_TILE + B_TILE);
constexpr int EMIT_BYTES = EPI_WARPS * 4 * 32 * 16;  // four columns of sums per epilogue warp
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EMIT_BYTES + 1024 /*barriers*/ + 1024 /*alignment*/;
static_assert(SMEM_BYTES <= 232448, "shared memory");
static_assert(S * BN <= 512, "TMEM columns");
// K blocks between two drains of the accumulator of weight g: the sum of its |q_t q_u| bounds
// (|q_0| <= 64, others <= 128) times 32 per block stays at 2^23 (FP32 holds 2^24 exactly; the
// drain reads the integer from the bits of (v + 2^23) 2^-149).  The leading groups, whose products
// hold q_0 and are few, go longer.
__host__ __device__ constexpr int group_bound(int g) {
  int b = 0;
  for (int t = 0; t <= g; ++t) b += (t == 0 ? 64 : 128) * (g - t == 0 ? 64 : 128);
  return b;
}
__host__ __device__ constexpr int group_kb(int g) {
  int p = 32;
  while (p > ROUND_KB && group_bound(g) * BK * p > 1 << 23) p >>= 1;
  return p;
}
constexpr bool sums_exact() {
  for (int g = 0; g < S; ++g)
    if (group_bound(g) * BK * group_kb(g) > 1 << 23) return false;
  return true;
}
static_assert(sums_exact(), "FP32 sums between two drains");
static_assert(SPLIT_KB % ROUND_KB == 0, "K ranges of whole rounds");

// element offset of row r with the optional two-level index r = r0 + div r1
__host__ __device__ __forceinline__ int64_t off2(int64_t r, int64_t div, int64_t s1, int64_t s2) {
  if (div <= 0) return r * s1;
  const int64_t q = r / div;
  return (r - q * div) * s1 + q * s2;
}

// ---- slicing --------------------------------------------------------------------------------
struct SliceArgs {
  const double* src;
  int64_t rows, K, div, s1, s2, ks, sb;  // row and k strides, batch stride
  int64_t batch, ldk;
  __nv_bfloat16* out;                    // [S][batch][rows][ldk]
  unsigned long long* key;               // [batch][rows] bit pattern of the row maximum
  int* e_out;                            // [batch][rows] exponent
  int* flag;                             // set when a non-finite element is met
  const unsigned long long* kmax;        // k balancing: bit patterns of the maxima over A's rows (or null)
  int ksign;                             // -1: divide by the power of two above the maximum, 1: multiply
};

__device__ __forceinline__ unsigned long long absbits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
}
// exponent e with |x| < 2^e for every x whose bit pattern is at most `key`
__device__ __forceinline__ int key_exponent(unsigned long long key) { return max((int)(key >> 52), 1) - 1022; }

// element k of a row, balanced: A(m, k) / 2^e_k, B(k, n) 2^e_k with 2^e_k just above max_m |A(m, k)|
__device__ __forceinline__ double balanced(const SliceArgs& a, double x, int64_t k) {
  if (a.kmax == nullptr) return x;
  const unsigned long long m = a.kmax[k];
  const int e = m == 0 ? 0 : max(-1000, min(1000, key_exponent(m)));
  return x * __hiloint2double((1023 + a.ksign * e) << 20, 0);
}
// maxima over the rows of A per k (bit patterns, atomics)
__global__ void __launch_bounds__(256) fx_kmax_kernel(SliceArgs a, unsigned long long* __restrict__ kmax, int64_t rc) {
  const int64_t total = a.rows * a.batch;
  const int64_t r0 = blockIdx.y * rc, r1 = min(total, r0 + rc);
  if (a.ks == 1) {  // threads along k
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= a.K) return;
    unsigned long long m = 0;
    for (int64_t r = r0; r < r1; ++r)
      m = max(m, absbits(a.src[off2(r % a.rows, a.div, a.s1, a.s2) + (r / a.rows) * a.sb + k]));
    if (m) atomicMax(kmax + k, m);
  } else {  // threads along the rows of one k
    const int64_t k = blockIdx.x;
    unsigned long long m = 0;
    for (int64_t r = r0 + threadIdx.x; r < r1; r += blockDim.x)
      m = max(m, absbits(a.src[off2(r % a.rows, a.div, a.s1, a.s2) + (r / a.rows) * a.sb + k * a.ks]));
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(kmax + k, m);
  }
}

// round(x 2^k) from the bit pattern; |x| 2^k < 2^62
__device__ __forceinline__ long long fixed(double x, int k) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
  const int E = (int)((bits >> 52) & 0x7FF);
  const long long M = (long long)(bits & 0xFFFFFFFFFFFFFull) | (E ? 1ll << 52 : 0ll);
  const int sh = 1075 - k - max(E, 1);
  long long F = 0;
  if (sh <= 0) F = M << min(-sh, 9);
  else if (sh < 63) F = (M + (1ll << (sh - 1))) >> sh;
  return (bits >> 63) ? -F : F;
}

// the digits of two fixed-point numbers as BF16 pairs to dst + t plane (4-byte aligned)
__device__ __forceinline__ void put_digits(long long f0, long long f1, __nv_bfloat16* dst, int64_t plane) {
  // adding 128 in every lower digit makes each byte the balanced digit plus 128
  constexpr unsigned long long BIAS = 0x0080808080808080ull;
  const unsigned long long u0 = (unsigned long long)f0 + BIAS, u1 = (unsigned long long)f1 + BIAS;
  *reinterpret_cast<__nv_bfloat162*>(dst) =
      __floats2bfloat162_rn((float)(int)((long long)u0 >> (8 * (S - 1))), (float)(int)((long long)u1 >> (8 * (S - 1))));
#pragma unroll
  for (int t = 1; t < S; ++t) {
    const int s = 8 * (S - 1 - t);
    *reinterpret_cast<__nv_bfloat162*>(dst + t * plane) =
        __floats2bfloat162_rn((float)((int)((u0 >> s) & 0xFF) - 128), (float)((int)((u1 >> s) & 0xFF) - 128));
  }
}

// Rows contiguous in k: one warp per row, maximum and digits in one launch (the second sweep
// finds the row in cache).  Bound by HBM: 8 B in, 2 S B out per element.
__global__ void __launch_bounds__(256) fx_slice_rows_kernel(SliceArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t w0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t total = a.rows * a.batch, plane = total * a.ldk;
  for (int64_t r = w0; r < total; r += nw) {
    const double* p = a.src + off2(r % a.rows, a.div, a.s1, a.s2) + (r / a.rows) * a.sb;
    unsigned long long m = 0;
    for (int64_t k = lane; k < a.K; k += 32) m = max(m, absbits(balanced(a, p[k], k)));
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    const int e = key_exponent(m);
    if (lane == 0) {
      a.e_out[r] = e;
      if (m >= 0x7FF0000000000000ull) *a.flag = 1;
    }
    for (int64_t k = 2 * lane; k < a.K; k += 64)
      put_digits(fixed(balanced(a, p[k], k), BITS - e),
                 k + 1 < a.K ? fixed(balanced(a, p[k + 1], k + 1), BITS - e) : 0ll,
                    a.out + r * a.ldk + k, plane);
  }
}

// Few long rows, contiguous in k: the K range split over blocks; row maxima by atomics first.
__global__ void __launch_bounds__(256) fx_rowmax_long_kernel(SliceArgs a, int64_t kc) {
  const int64_t r = blockIdx.y + (int64_t)blockIdx.z * gridDim.y;
  if (r >= a.rows * a.batch) return;
  const double* p = a.src + off2(r % a.rows, a.div, a.s1, a.s2) + (r / a.rows) * a.sb;
  const int64_t k0 = blockIdx.x * kc, k1 = min(a.K, k0 + kc);
  unsigned long long m = 0;
  for (int64_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) m = max(m, absbits(balanced(a, p[k], k)));
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m) atomicMax(a.key + r, m);
}
__global__ void __launch_bounds__(256) fx_slice_long_kernel(SliceArgs a, int64_t kc) {
  const int64_t r = blockIdx.y + (int64_t)blockIdx.z * gridDim.y;
  if (r >= a.rows * a.batch) return;
  const double* p = a.src + off2(r % a.rows, a.div, a.s1, a.s2) + (r / a.rows) * a.sb;
  const int64_t k0 = blockIdx.x * kc, k1 = min(a.K, k0 + kc);  // kc even
  const unsigned long long m = a.key[r];
  const int e = key_exponent(m);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.e_out[r] = e;
    if (m >= 0x7FF0000000000000ull) *a.flag = 1;
  }
  const int64_t plane = a.rows * a.batch * a.ldk;
  for (int64_t k = k0 + 2 * threadIdx.x; k < k1; k += 2 * blockDim.x)
    put_digits(fixed(balanced(a, p[k], k), BITS - e),
               k + 1 < k1 ? fixed(balanced(a, p[k + 1], k + 1), BITS - e) : 0ll,
                  a.out + r * a.ldk + k, plane);
}

// k strided (rows adjacent): blocks of 32 rows x kc, read along the rows; the digits are
// written along k through a shared-memory transpose of 32 x 64 elements.
__global__ void __launch_bounds__(256) fx_rowmax_strided_kernel(SliceArgs a, int64_t kc) {
  __shared__ unsigned long long red[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t total = a.rows * a.batch;
  const int64_t r = (int64_t)blockIdx.x * 32 + lane;
  const int64_t k0 = blockIdx.y * kc, k1 = min(a.K, k0 + kc);
  unsigned long long m = 0;
  if (r < total) {
    const double* p = a.src + off2(r % a.rows, a.div, a.s1, a.s2) + (r / a.rows) * a.sb;
    for (int64_t k = k0 + w; k < k1; k += 8) m = max(m, absbits(balanced(a, p[k * a.ks], k)));
  }
  red[w][lane] = m;
  __syncthreads();
  if (w == 0 && r < total) {
    for (int i = 1; i < 8; ++i) m = max(m, red[i][lane]);
    if (m) atomicMax(a.key + r, m);
  }
}
__global__ void __launch_bounds__(256) fx_slice_strided_kernel(SliceArgs a, int64_t kc) {
  __shared__ double tile[64][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t total = a.rows * a.batch, plane = total * a.ldk;
  const int64_t r0 = (int64_t)blockIdx.x * 32, r = r0 + lane;
  const int64_t kb = blockIdx.y * kc, ke = min(a.K, kb + kc);
  const double* p = a.src;
  if (r < total) {
    p += off2(r % a.rows, a.div, a.s1, a.s2) + (r / a.rows) * a.sb;
    if (blockIdx.y == 0 && w == 0) {
      const unsigned long long m = a.key[r];
      a.e_out[r] = key_exponent(m);
      if (m >= 0x7FF0000000000000ull) *a.flag = 1;
    }
  }
  for (int64_t k0 = kb; k0 < ke; k0 += 64) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int64_t k = k0 + w + 8 * i;
      tile[w + 8 * i][lane] = (r < total && k < ke) ? balanced(a, p[k * a.ks], k) : 0.0;
    }
    __syncthreads();
    const int64_t k = k0 + 2 * lane;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = w + 8 * i;
      if (r0 + rr < total && k < ke) {
        const int e = key_exponent(a.key[r0 + rr]);
        put_digits(fixed(tile[2 * lane][rr], BITS - e), fixed(tile[2 * lane + 1][rr], BITS - e),
                      a.out + (r0 + rr) * a.ldk + k, plane);
      }
    }
    __syncthreads();
  }
}

// ---- the GEMM kernel ------------------------------------------------------------------------
struct FxArgs {
  int64_t M, N;            // rows of this pass, columns
  int64_t K;
  int m_tiles, n_tiles, batch;
  int items;               // m_tiles n_tiles splits batch
  int nkb, kb_per_split;   // K blocks of 32, per split (a multiple of SPLIT_KB)
  int splits;
  const int* eA;           // [batch][M], [batch][N]
  const int* eB;
  double* C;               // splits == 1: the result, else nullptr
  int64_t c_m, c_m2, m_div, c_n, c_n2, n_div, c_b;
  int64_t m_base;          // first row of this pass
  double alpha, beta;
  int use_alpha, use_beta; // a factor alpha / beta to be multiplied out
  int e_alpha;             // a power of two alpha joins the exponents, its sign the result's
  unsigned flip;           // 0x80000000 to negate
  double* ws;              // splits > 1: [split][batch][N][M] exact-range sums rounded to FP64
  const int* flag;
  int* err;
};

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2,
                                            int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

// (hi 2^32 + lo) 2^e rounded to nearest FP64, in branch-free integer arithmetic (from its leading 64
// bits: to 2^-11 of the last place, ties among them to even);
// EDGE: also for results outside the normal range of FP64.
template <bool EDGE>
__device__ __forceinline__ double fx_round(long long hi, long long lo, int e, unsigned flip) {
  hi += lo >> 32;
  unsigned lw = (unsigned)lo;
  const int neg = (int)(hi >> 63);  // -1 or 0: magnitude of the 96-bit number hi : lw
  lw = (lw ^ (unsigned)neg) - (unsigned)neg;
  unsigned long long h = (unsigned long long)(hi ^ (long long)neg) + (neg != 0 && lw == 0u ? 1u : 0u);
  const bool small = h == 0;
  h = small ? (unsigned long long)lw << 32 : h;
  lw = small ? 0u : lw;
  const int lz = __clzll((long long)h);
  const unsigned long long top = (h << (lz & 63)) | (((unsigned long long)lw << 31) >> (63 - (lz & 63)));
  // value = top 2^(32 - lz) (2^-(32 + lz) when small): 53 bits and the rounding bit
  unsigned long long mant = top >> 11;
  mant += ((unsigned)top & 0x7FFu) + ((unsigned)mant & 1u) > 0x400u ? 1 : 0;
  const int be = (small ? -32 : 32) - lz + 11 + e + 1075;  // biased exponent of mant in [2^52, 2^53]
  if (EDGE && (be < 1 || be > 2045)) {
    const double v = h == 0 ? 0.0 : ldexp((double)(long long)mant, be - 1075);
    return (neg != 0) != (flip != 0) ? -v : v;
  }
  const unsigned long long bits = ((unsigned long long)(be - 1) << 52) + mant;
  const unsigned top32 = (unsigned)(bits >> 32) | (((unsigned)neg ^ flip) & 0x80000000u);
  return h == 0 ? 0.0 : __hiloint2double((int)top32, (int)(unsigned)bits);
}

__device__ __forceinline__ void fx_put(const FxArgs& args, double* p, double x) {
  // (flags: an FP64 comparison per element would cost as much as the product)
  if (args.use_alpha) x *= args.alpha;
  if (args.use_beta) x = fma(args.beta, *p, x);
  *p = x;
}
// Columns j0 .. j0 + EMIT of a tile with exponents near the ends of the FP64 range, from the sums
// in shared memory (rare: not inlined)
constexpr int EMIT = 4;
__device__ __noinline__ void fx_emit_edge(const FxArgs& args, double* o, const longlong2* sums, int e, int ebl,
                                          int64_t col, int j0, int jn, bool row_ok) {
  for (int j = 0; j < EMIT; ++j) {
    const double x = fx_round<true>(sums[j * 32].x, sums[j * 32].y, e + __shfl_sync(0xffffffffu, ebl, j0 + j), args.flip);
    const int64_t c = __shfl_sync(0xffffffffu, col, j0 + j);
    if (row_ok && j0 + j < jn) fx_put(args, o + c, x);
  }
}

// one work item: a tile of one K range and batch
struct FxItem {
  int m0, n0, bz, split, kb0, total;
};
__device__ __forceinline__ FxItem fx_item(const FxArgs& a, int w) {
  FxItem t;
  t.m0 = w % a.m_tiles * BM;
  w /= a.m_tiles;
  t.n0 = w % a.n_tiles * BN;
  w /= a.n_tiles;
  t.split = w % a.splits;
  t.bz = w / a.splits;
  t.kb0 = t.split * a.kb_per_split;
  t.total = min(a.nkb - t.kb0, a.kb_per_split);  // >= 1 (host)
  return t;
}

__global__ void __launch_bounds__(THREADS, 1)
    fx_gemm_kernel(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB,
                   const __grid_constant__ FxArgs args) {
  if (*args.flag) return;  // non-finite operands: the native kernel computes this product
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES + EMIT_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 2 * S + 1);
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES);
  const uint32_t gfull0 = smem_u32(bars + 2 * STAGES), gempty0 = smem_u32(bars + 2 * STAGES + S);
  const uint32_t done = smem_u32(bars + 2 * STAGES + 2 * S);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int g = 0; g < S; ++g) {
      mbar_init(gfull0 + 8 * g, 1);
      mbar_init(gempty0 + 8 * g, EPI_WARPS);
    }
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 512);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  constexpr int P[S] = {group_kb(0), group_kb(1), group_kb(2), group_kb(3),
                        group_kb(4), group_kb(5), group_kb(6), group_kb(7)};

  if (warp == 0 && lane == 0) {
    int gi = 0;  // K blocks loaded so far
    bool ok = true;
    for (int w = blockIdx.x; w < args.items && ok; w += gridDim.x) {
      const FxItem t = fx_item(args, w);
      for (int it = 0; it < t.total; ++it, ++gi) {
        const int s = gi % STAGES;
        if (!mbar_wait(empty0 + 8 * s, ((gi / STAGES) & 1) ^ 1, args.err)) { ok = false; break; }
        const uint32_t full = full0 + 8 * s;
        mbar_expect_tx(full, STAGE_BYTES);
        const uint32_t st = smem_u32(smem + s * STAGE_BYTES);
        tma_load_4d(st, &mA, full, (t.kb0 + it) * BK, t.m0, t.bz, 0);
        tma_load_4d(st + S * A_TILE, &mB, full, (t.kb0 + it) * BK, t.n0, t.bz, 0);
      }
    }
    // the copies of the last round of every stage have landed before the CTA may exit
    for (int i = max(0, gi - STAGES); i < gi; ++i) mbar_wait(full0 + 8 * (i % STAGES), (i / STAGES) & 1, nullptr);
  } else if (warp == 1) {
    constexpr uint32_t idesc = instr_desc_f16(BM, BN, true);
    const bool el = elect_one();
    int gi = 0;
    int runs[S];  // accumulations of group g begun so far
#pragma unroll
    for (int g = 0; g < S; ++g) runs[g] = 0;
    bool ok = true;
    for (int w = blockIdx.x; w < args.items && ok; w += gridDim.x) {
      const FxItem tile = fx_item(args, w);
      for (int it = 0; it < tile.total && ok; ++it, ++gi) {
        const int s = gi % STAGES;
        // (waits are agreed on by the whole warp)
        if (!__all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, (gi / STAGES) & 1, args.err))) { ok = false; break; }
        fence_after_sync();
        // one descriptor per stage, constants per MMA (see desc_off)
        const uint64_t da = smem_desc<64>(smem_u32(smem + s * STAGE_BYTES));
        const uint64_t db = da + desc_off(S * A_TILE);
        // a last block of at most 16 k needs one MMA step
        const bool two = args.K - (int64_t)(tile.kb0 + it) * BK > 16;
#pragma unroll
        for (int g = 0; g < S; ++g) {
          const bool first = it % P[g] == 0, last = it % P[g] == P[g] - 1 || it == tile.total - 1;
          if (first) {
            // the previous accumulation of this group has been drained
            if (runs[g] > 0 && ok) ok = __all_sync(0xffffffffu, mbar_wait(gempty0 + 8 * g, (runs[g] - 1) & 1, args.err));
            fence_after_sync();
            ++runs[g];
          }
          if (el && ok) {
#pragma unroll
            for (int t = 0; t <= g; ++t)
              mma_f16(tmem + (uint32_t)(g * BN), da + desc_off(t * A_TILE), db + desc_off((g - t) * B_TILE), idesc,
                      (first && t == 0) ? 0u : 1u);
            if (two) {
#pragma unroll
              for (int t = 0; t <= g; ++t)
                mma_f16(tmem + (uint32_t)(g * BN), da + desc_off(t * A_TILE + 32), db + desc_off((g - t) * B_TILE + 32),
                        idesc, 1u);
            }
            if (last) mma_commit(gfull0 + 8 * g);
          }
          __syncwarp();
        }
        if (el) mma_commit(empty0 + 8 * s);
        __syncwarp();
      }
    }
    // every issued MMA has retired before TMEM is released (also after an early exit)
    if (el) mma_commit(done);
    __syncwarp();
    mbar_wait(done, 0, nullptr);
  } else if (warp >= 2) {
    const int q = warp & 3, h = (warp - 2) >> 2;
    longlong2* const sums = reinterpret_cast<longlong2*>(smem + STAGES * STAGE_BYTES) + (warp - 2) * EMIT * 32 + lane;
    int runs[S];  // drains of group g done so far
#pragma unroll
    for (int g = 0; g < S; ++g) runs[g] = 0;
    bool ok = true;
    for (int w = blockIdx.x; w < args.items && ok; w += gridDim.x) {
      const FxItem tile = fx_item(args, w);
      long long hi[32], lo[32];
      {
        // minus the 2^23 that every drain adds
        long long h0 = 0, l0 = 0;
#pragma unroll
        for (int g = 0; g < S; ++g) {
          const long long drains = (tile.total + P[g] - 1) / P[g];
          if (g < 4) h0 -= drains << (23 + 8 * (3 - g));
          else l0 -= drains << (23 + 8 * (7 - g));
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) hi[j] = h0, lo[j] = l0;
      }
      for (int e0 = 0; e0 < tile.total && ok; e0 += ROUND_KB) {
        const int end = min(tile.total, e0 + ROUND_KB);  // K blocks accumulated by the end of the round
#pragma unroll
        for (int g = 0; g < S; ++g) {
          if (!ok || (end % P[g] != 0 && end != tile.total)) continue;
          // warp-uniform decision: tcgen05.ld is a whole-warp instruction
          ok = __all_sync(0xffffffffu, mbar_wait(gfull0 + 8 * g, runs[g] & 1, args.err));
          if (!ok) continue;
          ++runs[g];
          fence_after_sync();
          float v[32];
          tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(g * BN + h * 32), v);
          fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(gempty0 + 8 * g);
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            // v is an integer, |v| <= 2^23: the float (v + 2^23) 2^-149 is exact and its bits
            // are v + 2^23 (a float-to-integer conversion is 16 times slower than this FMA)
            const unsigned x = __float_as_uint(fmaf(v[j], __uint_as_float(1u), __uint_as_float(1u << 23)));
            if (g < 4) hi[j] += (long long)((unsigned long long)x << (8 * (3 - g)));
            else lo[j] += (long long)((unsigned long long)x << (8 * (7 - g)));
          }
        }
      }
      if (!ok) break;
      // the MMAs of the next item already run: only registers are read from here on
      const int64_t m = tile.m0 + q * 32 + lane;
      const bool row_ok = m < args.M;
      const int64_t nb0 = tile.n0 + h * 32;
      // exponent of the unit of lo: digits of weight 7
      const int ea =
          (row_ok ? args.eA[(int64_t)tile.bz * args.M + m] : 0) - 2 * BITS + 8 * (2 * (S - 1) - 7) + args.e_alpha;
      // this lane's column: exponent and offset, broadcast by shuffles
      const int64_t n = nb0 + lane;
      const int jn = (int)max((int64_t)0, min((int64_t)32, args.N - nb0));
      const int ebl = lane < jn ? args.eB[(int64_t)tile.bz * args.N + n] : 0;
      const bool part = args.splits > 1;
      const int64_t col = part ? n * args.M : off2(n, args.n_div, args.c_n, args.c_n2);
      double* const o =
          part ? args.ws + ((int64_t)tile.split * args.batch + tile.bz) * args.N * args.M + m
               : args.C + tile.bz * args.c_b + (row_ok ? off2(args.m_base + m, args.m_div, args.c_m, args.c_m2) : 0);
      // every result is zero or a normal number when the scales stay away from the range's ends
      const bool normal = __all_sync(0xffffffffu, abs(ea) < 420 && abs(ebl) < 420);
      if (normal) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const double x = fx_round<false>(hi[j], lo[j], ea + __shfl_sync(0xffffffffu, ebl, j), args.flip);
          const int64_t c = __shfl_sync(0xffffffffu, col, j);
          if (row_ok && j < jn) fx_put(args, o + c, x);
        }
      } else {
#pragma unroll
        for (int c = 0; c < 32; c += EMIT) {
#pragma unroll
          for (int j = 0; j < EMIT; ++j) sums[j * 32] = make_longlong2(hi[c + j], lo[c + j]);
          fx_emit_edge(args, o, sums, ea, ebl, col, c, jn, row_ok);
        }
      }
    }
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

// C = alpha sum_s ws[s] + beta C in a fixed order (rows fastest)
__global__ void __launch_bounds__(256) fx_reduce_kernel(FxArgs a, int64_t batch) {
  if (*a.flag) return;
  const int64_t per = a.M * a.N, total = per * batch;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t bz = e / per, r = e - bz * per;
    const int64_t n = r / a.M, m = r - n * a.M;
    double s = a.ws[e];
    for (int k = 1; k < a.splits; ++k) s += a.ws[e + k * total];
    double* p = a.C + bz * a.c_b + off2(a.m_base + m, a.m_div, a.c_m, a.c_m2) + off2(n, a.n_div, a.c_n, a.c_n2);
    s *= a.alpha;
    if (a.beta != 0.0) s = fma(a.beta, *p, s);
    *p = s;
  }
}

// ---- host side ------------------------------------------------------------------------------
// 4-D map {K, rows, batch, S} of BF16 planes, box {32, box_rows, 1, S}, 64B swizzle
bool make_map(CUtensorMap& m, const void* base, int64_t K, int64_t rows, int64_t batch, int64_t ldk, int S, int box_rows) {
  std::memset(&m, 0, sizeof(m));
  cuuint64_t dims[4] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)batch, (cuuint64_t)S};
  cuuint64_t strides[3] = {(cuuint64_t)(ldk * 2), (cuuint64_t)(ldk * 2 * rows), (cuuint64_t)(ldk * 2 * rows * batch)};
  cuuint32_t box[4] = {(cuuint32_t)BK, (cuuint32_t)box_rows, 1, (cuuint32_t)S};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// slice rows [row0, row0 + rows) of one operand; the row strides are (div, s1, s2)
cudaError_t slice(SliceArgs a, cudaStream_t s, int num_sms) {
  const int64_t total = a.rows * a.batch;
  if (a.ks == 1 && (a.K <= 1024 || total >= 8 * (int64_t)num_sms * 4)) {
    const unsigned grid = (unsigned)std::min<int64_t>(div_up(total, 8), 16 * (int64_t)num_sms);
    fx_slice_rows_kernel<<<grid, 256, 0, s>>>(a);
    count_launch();
  } else if (a.ks == 1) {
    const int64_t kc = std::max<int64_t>(2048, div_up(div_up(a.K * total, 16 * (int64_t)num_sms), 512) * 512);
    const unsigned gy = (unsigned)std::min<int64_t>(total, 32768);
    const dim3 grid((unsigned)div_up(a.K, kc), gy, (unsigned)div_up(total, gy));
    fx_rowmax_long_kernel<<<grid, 256, 0, s>>>(a, kc);
    fx_slice_long_kernel<<<grid, 256, 0, s>>>(a, kc);
    count_launch(2);
  } else {
    const int64_t gx = div_up(total, 32);
    // K chunks: about eight blocks per SM, 64-wide tiles
    const int64_t ny = std::max<int64_t>(1, std::min<int64_t>(div_up(a.K, 64), div_up(8 * (int64_t)num_sms, gx)));
    const int64_t kc = div_up(div_up(a.K, ny), 64) * 64;
    const dim3 grid((unsigned)gx, (unsigned)div_up(a.K, kc));
    fx_rowmax_strided_kernel<<<grid, 256, 0, s>>>(a, kc);
    fx_slice_strided_kernel<<<grid, 256, 0, s>>>(a, kc);
    count_launch(2);
  }
  return cudaGetLastError();
}

}  // namespace

cudaError_t fx_gemm(const FxPlan& p, cudaStream_t st, void* ws, int* err, int num_sms, const int** nonfinite) {
  if (nonfinite != nullptr && p.m_chunk < p.d.M) return cudaErrorInvalidValue;
  const GemmDesc& d = p.d;
  char* w = static_cast<char*>(ws);
  int* flag = reinterpret_cast<int*>(w);
  unsigned long long* keyB = reinterpret_cast<unsigned long long*>(w + 256);
  unsigned long long* kmax = d.k_balance ? keyB + d.N * d.batch1 : nullptr;
  unsigned long long* keyA = keyB + d.N * d.batch1 + (d.k_balance ? d.K : 0);
  int* eA = reinterpret_cast<int*>(w + p.off_ea);
  int* eB = reinterpret_cast<int*>(w + p.off_eb);
  __nv_bfloat16* pa = reinterpret_cast<__nv_bfloat16*>(w + p.off_a);
  __nv_bfloat16* pb = reinterpret_cast<__nv_bfloat16*>(w + p.off_b);
  cudaError_t e = cudaMemsetAsync(w, 0, p.key_bytes, st);
  if (e != cudaSuccess) return e;
  if (d.k_balance) {
    SliceArgs a{};
    a.src = static_cast<const double*>(d.A);
    a.rows = d.M; a.K = d.K; a.div = d.m_div; a.s1 = d.a_m; a.s2 = d.a_m2; a.ks = d.a_k; a.sb = d.a_b1; a.batch = d.batch1;
    const int64_t gx = d.a_k == 1 ? div_up(d.K, 256) : d.K, total = d.M * d.batch1;
    const int64_t gy = std::max<int64_t>(1, std::min<int64_t>(div_up(8 * (int64_t)num_sms, gx), div_up(total, 256)));
    const int64_t rc = div_up(total, gy);
    fx_kmax_kernel<<<dim3((unsigned)gx, (unsigned)gy), 256, 0, st>>>(a, kmax, rc);
    count_launch();
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  SliceArgs b{};
  b.kmax = kmax; b.ksign = 1;
  b.src = static_cast<const double*>(d.B);
  b.rows = d.N; b.K = d.K; b.div = d.n_div; b.s1 = d.b_n; b.s2 = d.b_n2; b.ks = d.b_k; b.sb = d.b_b1;
  b.batch = d.batch1; b.ldk = p.ldk; b.out = pb; b.key = keyB; b.e_out = eB; b.flag = flag;
  if ((e = slice(b, st, num_sms)) != cudaSuccess) return e;
  CUtensorMap mA, mB;
  if (!make_map(mB, pb, d.K, d.N, d.batch1, p.ldk, S, BN)) return cudaErrorUnknown;
  for (int64_t r0 = 0; r0 < d.M; r0 += p.m_chunk) {
    const int64_t rows = std::min<int64_t>(p.m_chunk, d.M - r0);
    if (r0 > 0 && (e = cudaMemsetAsync(keyA, 0, (size_t)rows * d.batch1 * 8, st)) != cudaSuccess) return e;
    SliceArgs a{};
    a.kmax = kmax; a.ksign = -1;
    // a chunk of a two-level row index starts on a multiple of its block (fx_plan)
    a.src = static_cast<const double*>(d.A) + off2(r0, d.m_div, d.a_m, d.a_m2);
    a.rows = rows; a.K = d.K; a.div = d.m_div; a.s1 = d.a_m; a.s2 = d.a_m2; a.ks = d.a_k; a.sb = d.a_b1;
    a.batch = d.batch1; a.ldk = p.ldk; a.out = pa; a.key = keyA; a.e_out = eA; a.flag = flag;
    if ((e = slice(a, st, num_sms)) != cudaSuccess) return e;
    if (!make_map(mA, pa, d.K, rows, d.batch1, p.ldk, S, BM)) return cudaErrorUnknown;
    FxArgs g{};
    g.M = rows; g.N = d.N; g.K = d.K;
    g.m_tiles = (int)div_up(rows, BM);
    g.nkb = (int)div_up(d.K, BK);
    g.kb_per_split = p.kb_per_split;
    g.splits = p.splits;
    g.eA = eA; g.eB = eB;
    g.C = static_cast<double*>(d.C);
    g.c_m = d.c_m; g.c_m2 = d.c_m2; g.m_div = d.m_div;
    g.c_n = d.c_n; g.c_n2 = d.c_n2; g.n_div = d.n_div;
    g.c_b = d.c_b1;
    g.m_base = r0;
    g.alpha = d.alpha; g.beta = d.beta;
    g.use_alpha = d.alpha != 1.0; g.use_beta = d.beta != 0.0;
    int ex = 0;
    if (p.splits == 1 && std::fabs(std::frexp(d.alpha, &ex)) == 0.5 && std::abs(ex) < 64) {
      g.e_alpha = ex - 1;
      g.flip = d.alpha < 0.0 ? 0x80000000u : 0u;
      g.use_alpha = 0;
    }
    if (p.splits > 1) g.use_alpha = g.use_beta = 0;  // fx_reduce_kernel applies them
    g.ws = reinterpret_cast<double*>(w + p.off_ws);
    g.flag = flag;
    g.err = err;
    g.n_tiles = p.n_tiles;
    g.batch = (int)d.batch1;
    g.items = g.m_tiles * g.n_tiles * g.splits * g.batch;
    const unsigned grid = (unsigned)std::min(g.items, num_sms);
    fx_gemm_kernel<<<grid, THREADS, SMEM_BYTES, st>>>(mA, mB, g);
    count_launch();
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (p.splits > 1) {
      const int64_t tot = rows * d.N * d.batch1;
      fx_reduce_kernel<<<(unsigned)std::min<int64_t>(div_up(tot, 256), 8 * (int64_t)num_sms), 256, 0, st>>>(g, d.batch1);
      count_launch();
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (nonfinite != nullptr) {
      *nonfinite = flag;
      continue;
    }
    // non-finite operands: the product on the native kernel (returns at once otherwise), its split-K
    // sums over the planes
    GemmDesc n = d;
    n.M = rows;
    n.A = a.src;
    n.C = static_cast<double*>(d.C) + off2(r0, d.m_div, d.c_m, d.c_m2);
    if ((e = gemm_f64_if(n, st, w + p.off_ea, p.total - p.off_ea, num_sms, flag)) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Plan and choice.  The line between the two kernels is drawn by their measured times (us, GB300):
//   native: gemm_f64_us;
//   fixed point: 9.2 per 128 k of a 128 x 64 tile and SM, at least ~10 for the rounding of its
//   results, ~4 to fill the pipeline; slicing and reducing stream at ~4.5e6 B/us; ~20 for the
//   launches around the GEMM.
// E.g. 540 x 180 x 36000: 459 (native 9200), 972 x 10800 x 180: 227 (3546), 600 x 54 x 3240: 100
// (244), 64 x 64 x 64: 33 (75); the native kernel stays for what its padded tiles do in less.
bool fx_plan(const GemmDesc& d0, int num_sms, FxPlan& p) {
  if (d0.batch2 != 1 || d0.batch1 < 1 || d0.batch1 > 65535 || d0.M < 1 || d0.N < 1 || d0.K < 1) return false;
  const double nb = (double)d0.batch1;
  const double flops = 2.0 * d0.M * d0.N * d0.K * nb;
  if (flops < 1e6) return false;
  GemmDesc t = d0;  // C^T = B^T A^T
  t.M = d0.N; t.N = d0.M;
  t.A = d0.B; t.a_m = d0.b_n; t.a_k = d0.b_k; t.m_div = d0.n_div; t.a_m2 = d0.b_n2; t.a_b1 = d0.b_b1;
  t.B = d0.A; t.b_n = d0.a_m; t.b_k = d0.a_k; t.n_div = d0.m_div; t.b_n2 = d0.a_m2; t.b_b1 = d0.a_b1;
  t.c_m = d0.c_n; t.c_m2 = d0.c_n2; t.c_n = d0.c_m; t.c_n2 = d0.c_m2;
  const int64_t tiles0 = div_up(d0.M, BM) * div_up(d0.N, BN), tiles1 = div_up(t.M, BM) * div_up(t.N, BN);
  // fewest padded tiles; equal: rows of the tile along the unit stride of C
  const bool swap = tiles1 < tiles0 || (tiles1 == tiles0 && d0.c_m != 1 && d0.c_n == 1);
  p.d = swap ? t : d0;
  const GemmDesc& d = p.d;
  p.ldk = div_up(d.K, 8) * 8;
  p.n_tiles = (int)div_up(d.N, BN);
  // rows of A per pass: planes within 3 GiB (B's planes stay for all passes)
  const int64_t row_bytes = 2 * S * p.ldk * d.batch1;
  const int64_t budget = int64_t(3) << 30;
  if (d.N * row_bytes > budget) return false;
  p.m_chunk = std::min<int64_t>(d.M, std::max<int64_t>(1, budget / row_bytes));
  if (p.m_chunk < d.M) {
    const int64_t unit = d.m_div > 0 ? d.m_div : BM;
    p.m_chunk = p.m_chunk / unit * unit;
    if (p.m_chunk < 1) return false;
  }
  p.m_tiles = (int)div_up(p.m_chunk, BM);
  const int64_t tiles = (int64_t)p.m_tiles * p.n_tiles * d.batch1;
  if (tiles * 64 > INT32_MAX || d.K > (int64_t(1) << 21)) return false;
  const int64_t rounds = div_up(d.K, SPLIT_KB * BK);
  // K split: the range count with the shortest critical path (waves of items over the SMs, then
  // the reduction of the partial sums)
  int best = 1;
  double best_t = 0.0;
  for (int s = 1; s <= 64 && s <= rounds; ++s) {
    const int64_t per = div_up(rounds, s), used = div_up(rounds, per);
    if (used != s || (size_t)s * p.m_chunk * d.N * d.batch1 * 8 > ((size_t)1 << 30)) continue;
    const double waves = (double)div_up(tiles * s, num_sms);
    const double tt = waves * (4.0 + std::max(9.2 * std::min<double>(per, d.K / 128.0), 10.0)) +
                      (s > 1 ? 5.0 + (double)(s + 1) * p.m_chunk * d.N * nb * 8 / 4.5e6 : 0.0);
    if (best_t == 0.0 || tt < best_t) best_t = tt, best = s;
  }
  p.splits = best;
  p.kb_per_split = (int)div_up(rounds, best) * SPLIT_KB;
  const double passes = (double)div_up(d.M, p.m_chunk);
  const double bytes = (double)(d.M + d.N) * d.K * nb * (16.0 + 4.0 * S) + 8.0 * d.M * d.N * nb;
  // an operand that is strided along k, or long in few rows, takes two slicing launches
  const double launches = (d.a_k != 1 || d.K > 1024 ? 6.0 : 0.0) + (d.b_k != 1 || d.K > 1024 ? 6.0 : 0.0);
  const double t_fx = passes * (best_t + 10.0) + 12.0 + launches + bytes / 4.5e6;
  const double t_native = gemm_f64_us(d0, num_sms);
  p.us = t_fx;
  if (t_fx > 0.8 * t_native) return false;
  size_t off = 256 + 8 * ((size_t)(d.N + p.m_chunk) * d.batch1 + (d.k_balance ? (size_t)d.K : 0));
  p.key_bytes = off;
  p.off_ea = align256(off);
  p.off_eb = align256(p.off_ea + 4 * (size_t)p.m_chunk * d.batch1);
  p.off_b = align256(p.off_eb + 4 * (size_t)d.N * d.batch1);
  p.off_a = align256(p.off_b + (size_t)d.N * row_bytes);
  p.off_ws = align256(p.off_a + (size_t)p.m_chunk * row_bytes);
  p.total = p.off_ws + (best > 1 ? (size_t)best * p.m_chunk * d.N * d.batch1 * 8 : 0);
  p.total = std::max(p.total, p.off_ea + gemm_workspace_bytes(d0, 8, num_sms));
  return true;
}

bool fx_available(int device) {
  static std::mutex mu;
  static int state[64] = {};  // per device: 0 unknown, 1 yes, 2 no
  if (device < 0 || device >= 64) return false;
  std::lock_guard<std::mutex> lock(mu);
  if (state[device] == 0) {
    int major = 0;
    bool ok = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) == cudaSuccess && major == 10 &&
              encode_fn() != nullptr;
    ok = ok &&
         cudaFuncSetAttribute(fx_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) ==
             cudaSuccess;
    if (!ok) cudaGetLastError();
    state[device] = ok ? 1 : 2;
  }
  return state[device] == 1;
}

}  // namespace cphf
