// Split-K contractions of the RI-K term on CTA pairs (sm_103a, tcgen05 cta_group::2).
//
//   out[m, n] += sum_P sum_k X_P[m, k] Y_P[n, k]        (src/ri_jk/hess_r.rs:159-176: terms 1 and 2)
//
// with X = B_P (term 1) or Z_P (term 2) and Y = T_P or W_P, as split FP16 planes (the inner
// operator) or exact BF16 slices (the FP64-accurate residuals).
//
// What bounds it: the TMA fill of shared memory, 44-50 B/clk and SM for 128-byte rows and 30-35
// for 64-byte rows.  A single CTA's 128 x 256 split-FP16 tile needs 64 B/clk to keep its MMAs
// going, the 128 x 128 six-slice tile 37, the three-slice tile 64, so they ran at 217 of 128, 102
// of 64 and 190 of 64 clocks an MMA.  A pair shares the second operand: each CTA loads its own
// 128 rows of one operand and half of the other, 43-47, 27 and 47 B/clk.
// The pair's 256 rows lie along n (thousands of columns, so padding is small); m, the AO index, is
// the narrow side, whose tile width fits nao (NT a multiple of 32: nao 600 runs as 3 x 224
// split-FP16 tiles).  One mixed solve of nao 600, nocc 60, naux 2000 (180 right-hand sides), ms in
// term 1 before / on pairs: split FP16 272 / 183 (the MMA issue limit: 112 clk each at 1.55 GHz),
// six slices 239 / 169, three slices 128 / 71.  A last K block of fewer than 64 / 32 k issues only the steps it needs.
//
//   warp 0 lane 0 (both CTAs) -- TMA producer of its own tiles; all of the pair's bytes complete on
//                                the leader's barrier;
//   warp 1 (leader)           -- MMA issuer (M = 256), warp-uniform with an elected lane; the
//                                multicast commit frees the stage in both CTAs;
//   warp 2 (both)             -- TMEM owner;
//   warps 0-7 (both)          -- epilogue: each CTA's 128 rows of D, transposed through shared
//                                memory so that the atomics run along m.
// Every mbarrier wait is bounded; on expiry the kernel raises the error flag and finishes.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "slices.cuh"
#include "tc_pair.cuh"
#include "tc_map.cuh"
#include "tc_ptx.cuh"

namespace cphf {
namespace {
using namespace tcx;

constexpr int BM = 128;             // rows of n per CTA
constexpr int SMEM_LIMIT = 227 * 1024;
constexpr int MAX_STAGES = 6;
constexpr int PAIR_THREADS = 256;  // eight epilogue warps: a TMEM lane quarter and a half of m each

template <class PR>
struct PairCfg {
  static constexpr bool EXACT = PR::NACC == 4;
  static constexpr int BK = EXACT ? 32 : 64;       // elements per K block: 64- / 128-byte rows
  static constexpr int ROW = BK * 2;               // bytes = the swizzle width
  static constexpr int A_TILE = BM * ROW;
  static constexpr int MAX_NT = EXACT ? 128 : 256; // four accumulators of 128 (five of 96) / two
  static constexpr int TMEM_COLS = 512;
  static constexpr int EPI_BYTES = 8 * 16 * 33 * (EXACT ? 8 : 4);
};

struct PairArgs {
  int M, N, K, NT;         // m, n, k extents, m tile width
  int m_tiles;
  int nkb, total_kb, kb_per_cta;
  int x_off, x_depth, y_depth;  // depth strides of the planes (exact), depth offset of X
  int x_row0, y_k0, store;
  int stages, b_tile, stage_bytes;
  int acc_cols, acc5;      // exact: columns of an accumulator; five of them (else four)
  const double* rowscale;  // exact: powers of two
  const double* colscale;
  const float* scale;
  void* out;
  int64_t ld_out;
  int* err;
};

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_rank0(uint32_t addr) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
// this CTA's tile; the bytes complete on the barrier `bar` of the pair's leader
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                                 int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, "
      "%5}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
// arrives on the barrier at this offset in both CTAs when the MMAs issued so far have retired
__device__ __forceinline__ void commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"((uint16_t)3)
      : "memory");
}

// float -> double on the integer pipe (subnormals, far below any group sum's unit, to zero; NaN and
// Inf, from non-finite operands, stay): the conversion instruction occupies the FP64 pipe like a
// multiplication.  Branch-free: it is unrolled over an accumulator chunk.
__device__ __forceinline__ double widen(float x) {
  const unsigned b = __float_as_uint(x), e = b & 0x7F800000u;
  const unsigned hi = (b & 0x80000000u) | (((b & 0x7FFFFFFFu) >> 3) + 0x38000000u) | (e == 0x7F800000u ? 0x7FF00000u : 0u);
  return __hiloint2double(e == 0u ? 0 : (int)hi, e == 0u ? 0 : (int)(b << 29));
}
// a0 + a1 + a2 + a3 (a0, a1, a2 exact integer sums, a3 rounded; three slices: no a3) through an FP32 pair
template <int NS>
__device__ __forceinline__ double combine4(float a0, float a1, float a2, float a3) {
  float s, e, e2;
  two_sum(a0, a1, s, e);
  two_sum(s, a2, s, e2);
  e += e2;
  if constexpr (NS > 3) {
    two_sum(s, a3, s, e2);
    e += e2;
  }
  return widen(s) + widen(e);
}
// x 2^k by the exponent field; subnormal operands and results to zero, NaN and Inf stay
__device__ __forceinline__ double shift_exp(double x, int k) {
  const int hi = __double2hiint(x), e = (hi >> 20) & 0x7FF, r = e + k;
  const bool zero = e == 0 || (r <= 0 && e != 0x7FF), inf = r >= 0x7FF && e != 0x7FF;
  const int h = e == 0x7FF ? hi : inf ? (hi & (int)0x80000000u) | 0x7FF00000 : hi + (k << 20);
  return __hiloint2double(zero ? 0 : h, zero || inf ? 0 : __double2loint(x));
}

template <class PR>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
    tc_pair_kernel(const __grid_constant__ CUtensorMap mY0, const __grid_constant__ CUtensorMap mY1,
                   const __grid_constant__ CUtensorMap mX0, const __grid_constant__ CUtensorMap mX1, const PairArgs args) {
  using C = PairCfg<PR>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int stages = args.stages;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + stages * args.stage_bytes);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * MAX_STAGES + 1);
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + MAX_STAGES), accum = smem_u32(bars + 2 * MAX_STAGES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  // pair tile: m fastest, so that the pairs sharing a Y tile run together
  const int tile = blockIdx.x >> 1;
  const int m0 = tile % args.m_tiles * args.NT, n0 = tile / args.m_tiles * (2 * BM) + (int)rank * BM;
  const int kb0 = blockIdx.y * args.kb_per_cta;
  const int total = min(args.total_kb - kb0, args.kb_per_cta);  // >= 1 (host)

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(accum, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(C::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers are initialised before either loads or commits
  fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    int issued = 0;
    for (int it = 0; it < total; ++it) {
      const int s = it % stages;
      if (!mbar_wait(empty0 + 8 * s, ((it / stages) & 1) ^ 1, args.err)) break;
      issued = it + 1;
      // the leader's barrier counts the bytes of both CTAs
      if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * (uint32_t)args.stage_bytes);
      const uint32_t full = map_to_rank0(full0 + 8 * s);
      const int kb = kb0 + it;
      const int P = kb / args.nkb, k0 = (kb - P * args.nkb) * C::BK;
      const uint32_t st = smem_u32(smem + s * args.stage_bytes);
      const uint32_t sb = st + PR::S * C::A_TILE;
      const int mb = args.x_row0 + m0 + (int)rank * (args.NT / 2);
#pragma unroll
      for (int t = 0; t < PR::S; ++t) {
        const CUtensorMap* y = !C::EXACT && t == 1 ? &mY1 : &mY0;
        const CUtensorMap* x = !C::EXACT && t == 1 ? &mX1 : &mX0;
        tma_load_3d_pair(st + t * C::A_TILE, y, full, args.y_k0 + k0, n0, C::EXACT ? t * args.y_depth + P : P);
        tma_load_3d_pair(sb + t * args.b_tile, x, full, k0, mb, (C::EXACT ? t * args.x_depth : 0) + args.x_off + P);
      }
    }
    // the pair's copies of the last round of every stage have landed (the leader's barrier counts
    // the peer's too; the cluster barrier below holds the peer until then)
    if (rank == 0)
      for (int it = max(0, issued - stages); it < issued; ++it)
        mbar_wait(full0 + 8 * (it % stages), (it / stages) & 1, nullptr);
  } else if (warp == 1 && rank == 0) {
    const uint32_t idesc = instr_desc_f16(2 * BM, args.NT, PR::BF16);
    const bool el = elect_one();
    const uint64_t bt = (uint64_t)(args.b_tile >> 4);
    for (int it = 0; it < total; ++it) {
      const int s = it % stages;
      if (!__all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, (it / stages) & 1, args.err))) break;
      fence_after_sync();
      const uint64_t da = smem_desc<C::ROW>(smem_u32(smem + s * args.stage_bytes));
      const uint64_t db = da + desc_off(PR::S * C::A_TILE);
      // k steps of 16 inside the block (the last block of an aux function may need fewer)
      const int left = args.K - (kb0 + it) % args.nkb * C::BK;
      if (el) {
#pragma unroll
        for (int k = 0; k < C::BK / 16; ++k) {
          if (16 * k >= left) break;
          const uint64_t dk = desc_off(k * 32);  // 16 elements inside the swizzle row
          if constexpr (C::EXACT) {
#pragma unroll
            for (int g = 0; g < PR::S; ++g)
#pragma unroll
              for (int t = 0; t <= g; ++t) {
                // groups 4 and 5, whose rounding is 2^-6 of group 3's, beside it where there is room
                const int acc = g < 4 ? g : 3 + args.acc5;
                const bool first = it == 0 && k == 0 && t == 0 && (g <= 3 || (g == 4 && args.acc5 != 0));
                mma_pair(tmem + (uint32_t)(acc * args.acc_cols), da + (desc_off(t * C::A_TILE) + dk), db + (uint64_t)(g - t) * bt + dk,
                         idesc, first ? 0u : 1u);
              }
          } else {
            // hi*hi, and hi*lo + lo*hi in an accumulator of their own: the small products would make
            // the large sum drop low bits three times as often
            const uint32_t more = (it > 0 || k > 0) ? 1u : 0u;
            mma_pair(tmem, da + dk, db + dk, idesc, more);
            mma_pair(tmem + 256, da + dk, db + bt + dk, idesc, more);
            mma_pair(tmem + 256, da + (desc_off(C::A_TILE) + dk), db + dk, idesc, 1u);
          }
        }
        commit_pair(empty0 + 8 * s);
      }
      __syncwarp();
    }
    if (el) commit_pair(accum);  // arrives when every issued MMA has retired (also after an early exit)
    __syncwarp();
  }
  __syncwarp();
  // epilogue: warps w and w + 4 own TMEM lanes [32 w, 32 w + 32), rows n, and half of the m tile in
  // chunks of 16, each transposed through a 16 x 33 tile over the idle load ring
  // warp-uniform decision: tcgen05.ld is a whole-warp instruction
  const bool have = __all_sync(0xffffffffu, mbar_wait(accum, 0, args.err) && *(volatile int*)args.err == 0);
  fence_after_sync();
  if (have) {
    const int q = warp & 3, h = warp >> 2;
    const int nw = n0 + q * 32, nn = min(32, args.N - nw);  // this warp's columns of out
    const uint32_t base = tmem + ((uint32_t)(q * 32) << 16);
    const int mw = min(args.NT, args.M - m0), half = args.NT / 2;
    const int c_end = min(mw, (h + 1) * half);
    // lanes of the write: 16 consecutive m of two columns n
    const int wm = lane & 15, wn = lane >> 4;
    if constexpr (C::EXACT) {
      // FP64 work per element: one addition, one multiplication, the atomic (the row factor is a
      // power of two)
      double* const tp = reinterpret_cast<double*>(smem) + warp * 16 * 33;
      const double cs = lane < nn ? args.colscale[nw + lane] : 0.0;
      for (int c = h * half; c < c_end; c += 16) {
        float v0[16], v1[16], v2[16], v3[16];
        const uint32_t ac = (uint32_t)args.acc_cols;
        tmem_ld16x4(base + (uint32_t)c, base + ac + (uint32_t)c, base + 2 * ac + (uint32_t)c, base + 3 * ac + (uint32_t)c,
                    v0, v1, v2, v3);
        if constexpr (PR::S > 4) {
          if (args.acc5) {
            float v4[16];
            tmem_ld16(base + 4 * ac + (uint32_t)c, v4);
#pragma unroll
            for (int j = 0; j < 16; ++j) v3[j] += v4[j];
          }
        }
        if constexpr (PR::S <= 3) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v3[j] = 0.f;  // groups 0-2 only: the fourth accumulator is unused
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) tp[j * 33 + lane] = combine4<PR::S>(v0[j], v1[j], v2[j], v3[j]) * cs;
        __syncwarp();
        if (c + wm < c_end) {
          const int k = ((__double2hiint(args.rowscale[m0 + c + wm]) >> 20) & 0x7FF) - 1023;
          double* o = reinterpret_cast<double*>(args.out) + (m0 + c + wm) + args.ld_out * (int64_t)nw;
#pragma unroll 4
          for (int n = wn; n < nn; n += 2) {
            const double v = shift_exp(tp[wm * 33 + n], k);
            if (args.store) o[args.ld_out * n] = v;
            else atomicAdd(o + args.ld_out * n, v);
          }
        }
        __syncwarp();
      }
    } else {
      float* const tp = reinterpret_cast<float*>(smem) + warp * 16 * 33;
      const float cs = (args.scale ? *args.scale : 1.f) * (args.colscale && lane < nn ? (float)args.colscale[nw + lane] : 1.f);
      for (int c = h * half; c < c_end; c += 16) {
        float v[16], w[16];
        tmem_ld16(base + (uint32_t)c, v);
        tmem_ld16(base + (uint32_t)(256 + c), w);
#pragma unroll
        for (int j = 0; j < 16; ++j) tp[j * 33 + lane] = (v[j] + w[j]) * cs;
        __syncwarp();
        if (c + wm < c_end) {
          const float rs = args.rowscale ? (float)args.rowscale[m0 + c + wm] : 1.f;
          float* o = reinterpret_cast<float*>(args.out) + (m0 + c + wm) + args.ld_out * (int64_t)nw;
#pragma unroll 4
          for (int n = wn; n < nn; n += 2) atomicAdd(o + args.ld_out * n, tp[wm * 33 + n] * rs);
        }
        __syncwarp();
      }
    }
  }
  fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // neither CTA leaves (or frees TMEM) while the pair's MMAs or loads may run
  fence_after_sync();
  if (warp == 2)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::TMEM_COLS) : "memory");
}

// ---- host side ------------------------------------------------------------------------------
// 3-D map: dims {K, rows, depth}, row stride ld, box {row / 2 elements, box_rows, 1}, swizzle = row bytes
CUtensorMap make_map(const void* base, int64_t K, int64_t rows, int64_t depth, int64_t ld, int row, int box_rows,
                     bool bf16) {
  CUtensorMap m;
  std::memset(&m, 0, sizeof(m));
  auto fn = encode_fn();
  if (!fn) throw Error(CPHF_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)depth};
  cuuint64_t strides[2] = {(cuuint64_t)(ld * 2), (cuuint64_t)(ld * 2 * rows)};
  cuuint32_t box[3] = {(cuuint32_t)(row / 2), (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(&m, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3,
                  const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  row == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw Error(CPHF_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
  return m;
}

template <class PR>
bool set_attr() {
  return cudaFuncSetAttribute(tc_pair_kernel<PR>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT) == cudaSuccess;
}

template <class PR>
void launch_pair(cphf_ctx* c, const PairTerm& t, int kb_per_cta) {
  using C = PairCfg<PR>;
  PairArgs a;
  std::memset(&a, 0, sizeof(a));
  a.M = (int)t.M;
  a.N = (int)t.N;
  a.K = (int)t.K;
  // tile width along m: a multiple of 32 (M = 256 MMAs), the one whose padded tiles take the least
  // time per K block, MMAs (NT / 2 clocks each) or loads, whichever is longer
  constexpr int products = C::EXACT ? PR::S * (PR::S + 1) / 2 : 3;
  double best_m = 0.0;
  for (int64_t mt = div_up(t.M, C::MAX_NT); mt <= div_up(t.M, C::MAX_NT) + 3; ++mt) {
    const int nt = (int)div_up(div_up(t.M, mt), 32) * 32;
    const double mma = products * (C::BK / 16) * nt / 2.0;
    const double load = PR::S * (C::A_TILE + nt / 2 * C::ROW) / (C::EXACT ? 32.0 : 45.0);
    const double clk = (double)div_up(t.M, nt) * std::max(mma, load);
    if (best_m == 0.0 || clk < best_m) best_m = clk, a.NT = nt, a.m_tiles = (int)div_up(t.M, nt);
  }
  // Group 3's sum is the largest that is rounded, and every product added to its accumulator rounds it
  // again: groups 4 and 5 (11 of its 15 products) get one of their own where five fit.  FP64-accurate
  // operator against FP64, four / five: nao 150 2.6e-12 / 1.3e-12, nao 400 2.8e-12 / 1.1e-12; the time is the same.
  a.acc5 = PR::S > 4 && 5 * a.NT <= C::TMEM_COLS;
  a.acc_cols = a.acc5 ? a.NT : 128;
  a.nkb = (int)div_up(t.K, C::BK);
  a.total_kb = (int)(t.np * a.nkb);
  a.x_off = (int)t.x_off;
  a.x_depth = (int)t.x.depth_stride;
  a.y_depth = (int)t.y.depth_stride;
  a.b_tile = a.NT / 2 * C::ROW;
  a.stage_bytes = PR::S * (C::A_TILE + a.b_tile);
  a.stages = std::min(MAX_STAGES, (SMEM_LIMIT - 2048) / a.stage_bytes);
  a.rowscale = t.rowscale;
  a.colscale = t.colscale;
  a.scale = t.scale;
  a.out = t.out;
  a.ld_out = t.ld_out;
  a.err = t.err;
  a.x_row0 = (int)t.x_row0;
  a.y_k0 = (int)t.y_k0;
  a.store = t.store;
  const int64_t tiles = (int64_t)a.m_tiles * div_up(t.N, 2 * BM);
  const int64_t pairs = std::max(1, c->num_sms / 2);
  if (kb_per_cta <= 0 && t.np == 1) {
    // one long K (the XC batches): the range count with the shortest time, an epilogue as above
    const int64_t r0 = C::EXACT ? div_up(a.total_kb, PAIR_EXACT_KB) : 1;
    double best_t = 0.0;
    for (int64_t r = r0; r <= r0 + 63 && r <= a.total_kb && !(t.store && r > 1); ++r) {
      const int64_t kb = div_up(a.total_kb, r), used = div_up(a.total_kb, kb);
      const double tt = (double)div_up(tiles * used, pairs) * ((double)kb + 8.0);
      if (best_t == 0.0 || tt < best_t) best_t = tt, kb_per_cta = (int)kb;
    }
    if (kb_per_cta <= 0) kb_per_cta = a.total_kb;
  }
  if (kb_per_cta <= 0) {
    // ranges of whole aux functions, long enough for the epilogue to be small beside them (each
    // tile's atomics cost about eight K blocks) and short enough to fill the SMs evenly
    // The accumulators drop low bits at every MMA, an error that grows with the products summed, so
    // max_k bounds a range.  Exchange response against FP64, in one accumulator over ranges that the
    // time alone chooses / hi*hi in one of its own and at most 32 nao products: nao 243 2.4e-5 / 6.7e-6,
    // nao 400 5.3e-5 / 1.4e-5, nao 600 5.8e-5 / 2.0e-5, for 0.5 % of a solve's time.
    int64_t best = t.np;
    double best_t = 0.0;
    const int64_t r0 = t.max_k > 0 ? div_up(t.np, std::max<int64_t>(1, t.max_k / t.K)) : 1;
    for (int64_t r = r0; r <= std::min<int64_t>(t.np, r0 + 63); ++r) {
      const int64_t ppc = div_up(t.np, r), used = div_up(t.np, ppc);
      const double tt = (double)div_up(tiles * used, pairs) * ((double)ppc * a.nkb + 8.0);
      if (best_t == 0.0 || tt < best_t) best_t = tt, best = ppc;
    }
    kb_per_cta = (int)(best * a.nkb);
  }
  a.kb_per_cta = kb_per_cta;
  const int64_t ranges = div_up(a.total_kb, kb_per_cta);
  if (2 * tiles > INT32_MAX || ranges > 65535) throw Error(CPHF_ERR_ARG, "tensor-core K term: grid too large");
  const int64_t xk = t.x.kext > 0 ? t.x.kext : t.K, yk = t.y.kext > 0 ? t.y.kext : t.K;
  const CUtensorMap y0 = make_map(t.y.p[0], yk, t.y.rows, t.y.depth, t.y.ld, C::ROW, BM, PR::BF16);
  const CUtensorMap x0 = make_map(t.x.p[0], xk, t.x.rows, t.x.depth, t.x.ld, C::ROW, a.NT / 2, PR::BF16);
  const CUtensorMap y1 = C::EXACT ? y0 : make_map(t.y.p[1], yk, t.y.rows, t.y.depth, t.y.ld, C::ROW, BM, PR::BF16);
  const CUtensorMap x1 = C::EXACT ? x0 : make_map(t.x.p[1], xk, t.x.rows, t.x.depth, t.x.ld, C::ROW, a.NT / 2, PR::BF16);
  const size_t smem = (size_t)std::max(a.stages * a.stage_bytes, C::EPI_BYTES) + 2048;
  tc_pair_kernel<PR><<<dim3((unsigned)(2 * tiles), (unsigned)ranges), PAIR_THREADS, smem, c->stream>>>(y0, y1, x0, x1, a);
  count_launch();
  CPHF_CUDA(cudaGetLastError());
}

}  // namespace

bool pair_available(int device) {
  static std::mutex mu;
  static int state[64] = {};  // per device: 0 unknown, 1 yes, 2 no
  if (device < 0 || device >= 64) return false;
  std::lock_guard<std::mutex> lock(mu);
  if (state[device] == 0) {
    int major = 0;
    const bool ok = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) == cudaSuccess &&
                    major == 10 && encode_fn() != nullptr && set_attr<Split2>() && set_attr<Exact6>() &&
                    set_attr<Exact6c>() && set_attr<Exact6c3>();
    if (!ok) cudaGetLastError();
    state[device] = ok ? 1 : 2;
  }
  return state[device] == 1;
}

void pair_split2(cphf_ctx* c, const PairTerm& t) {
  if (t.M <= 0 || t.N <= 0 || t.K <= 0 || t.np <= 0) return;
  launch_pair<Split2>(c, t, 0);
}

void pair_exact(cphf_ctx* c, const PairTerm& t, int slices, int kb_per_cta) {
  if (t.M <= 0 || t.N <= 0 || t.K <= 0 || t.np <= 0) return;
  if (kb_per_cta > PAIR_EXACT_KB || (kb_per_cta <= 0 && t.np != 1) || (t.store && div_up(t.K, 32) > PAIR_EXACT_KB))
    throw Error(CPHF_ERR_ARG, "exact slices: K range out of bounds");
  if (slices == 3) launch_pair<Exact6c3>(c, t, kb_per_cta);
  else if (slices == 4) launch_pair<Exact6c>(c, t, kb_per_cta);
  else launch_pair<Exact6>(c, t, kb_per_cta);
}

}  // namespace cphf
