// Generic strided/batched SIMT GEMM, see gemm_simt.cuh.
#include "gemm_simt.cuh"
#include "common.cuh"
#include "dfloat.cuh"

#include <algorithm>
#include <type_traits>

namespace cphf {

namespace {

// FP64: 64x64 tile, 4x4 per thread, 256 threads.  FP64-pipe bound on GB300.
struct CfgF64 {
  static constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;
};
// FP64, few or short outputs: 32x32 tile, 2x2 per thread, so that small products spread over the SMs.
struct CfgF64S {
  static constexpr int BM = 32, BN = 32, BK = 16, TM = 2, TN = 2;
};
// FP32: 128x128 tile, 8x8 per thread, 256 threads.
struct CfgF32 {
  static constexpr int BM = 128, BN = 128, BK = 16, TM = 8, TN = 8;
};
// FP32 where 64-wide columns pad less: 256x64 tile, 8x8 per thread, 256 threads.
struct CfgF32Tall {
  static constexpr int BM = 256, BN = 64, BK = 16, TM = 8, TN = 8;
};

// offset of row m (or column n) with optional two-level index m = m0 + div * m1
__device__ __forceinline__ int64_t off2(int64_t m, int64_t div, int64_t s1, int64_t s2) {
  if (div <= 0) return m * s1;
  const int64_t q = m / div;
  return (m - q * div) * s1 + q * s2;
}

template <typename T, typename Cfg, typename TA, typename TB, typename TC>
__global__ void __launch_bounds__(256) gemm_kernel(GemmDesc d, int ksplit, int64_t kchunk, T* ws,
                                                   const int* only_if) {
  if (only_if != nullptr && *only_if == 0) return;
  constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK, TM = Cfg::TM, TN = Cfg::TN;
  constexpr int NTX = BN / TN, NTY = BM / TM, NT = NTX * NTY;
  constexpr int LA = BM * BK / NT, LB = BK * BN / NT;
  // rows 16 bytes longer than the tile: operands with k contiguous are stored down a column, which
  // would meet one bank 16 times over
  constexpr int PAD = 16 / sizeof(T);
  __shared__ __align__(16) T As[2][BK][BM + PAD];
  __shared__ __align__(16) T Bs[2][BK][BN + PAD];

  const int tid = threadIdx.x;
  // tile row / column of the thread's i-th: FP32 in groups of four, read as 16 bytes, and lanes along
  // the rows, whose results are mostly contiguous
  constexpr bool VEC = std::is_same<T, float>::value;
  const int tx = VEC ? tid / NTY : tid % NTX, ty = VEC ? tid % NTY : tid / NTX;
  auto row = [&](int i) { return VEC ? (i >> 2) * (4 * NTY) + ty * 4 + (i & 3) : ty + i * NTY; };
  auto col = [&](int j) { return VEC ? (j >> 2) * (4 * NTX) + tx * 4 + (j & 3) : tx + j * NTX; };
  const int64_t m0 = (int64_t)blockIdx.x * BM;
  const int64_t n0 = (int64_t)blockIdx.y * BN;
  const int64_t z = blockIdx.z;
  const int split = (int)(z % ksplit);
  const int64_t bidx = z / ksplit;
  const int64_t b1 = bidx % d.batch1, b2 = bidx / d.batch1;

  const TA* __restrict__ A = static_cast<const TA*>(d.A) + b1 * d.a_b1 + b2 * d.a_b2;
  const TB* __restrict__ B = static_cast<const TB*>(d.B) + b1 * d.b_b1 + b2 * d.b_b2;
  TC* __restrict__ C = static_cast<TC*>(d.C) + b1 * d.c_b1 + b2 * d.c_b2;

  const int64_t kbeg = (int64_t)split * kchunk;
  const int64_t kend = min(d.K, kbeg + kchunk);
  // load mapping: consecutive threads along the unit-stride index (offsets are precomputed, so
  // a two-level index still coalesces inside each contiguous block)
  const bool a_mfast = (d.a_m == 1);
  const bool b_nfast = (d.b_n == 1);

  // per-thread fixed row / column of each load, and its offset
  int a_mm[LA], a_kk[LA], b_nn[LB], b_kk[LB];
  int64_t a_off[LA], b_off[LB];
  bool a_ok[LA], b_ok[LB];
#pragma unroll
  for (int i = 0; i < LA; ++i) {
    const int e = tid + i * NT;
    if (a_mfast) { a_mm[i] = e % BM; a_kk[i] = e / BM; } else { a_kk[i] = e % BK; a_mm[i] = e / BK; }
    const int64_t gm = m0 + a_mm[i];
    a_ok[i] = gm < d.M;
    a_off[i] = a_ok[i] ? off2(gm, d.m_div, d.a_m, d.a_m2) : 0;
  }
#pragma unroll
  for (int i = 0; i < LB; ++i) {
    const int e = tid + i * NT;
    if (b_nfast) { b_nn[i] = e % BN; b_kk[i] = e / BN; } else { b_kk[i] = e % BK; b_nn[i] = e / BK; }
    const int64_t gn = n0 + b_nn[i];
    b_ok[i] = gn < d.N;
    b_off[i] = b_ok[i] ? off2(gn, d.n_div, d.b_n, d.b_n2) : 0;
  }

  T ra[LA], rb[LB];
  auto load_tiles = [&](int64_t k0) {
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int64_t gk = k0 + a_kk[i];
      ra[i] = (a_ok[i] && gk < kend) ? (T)A[a_off[i] + gk * d.a_k] : (T)0;
    }
#pragma unroll
    for (int i = 0; i < LB; ++i) {
      const int64_t gk = k0 + b_kk[i];
      rb[i] = (b_ok[i] && gk < kend) ? (T)B[b_off[i] + gk * d.b_k] : (T)0;
    }
  };
  auto store_tiles = [&](int buf) {
#pragma unroll
    for (int i = 0; i < LA; ++i) As[buf][a_kk[i]][a_mm[i]] = ra[i];
#pragma unroll
    for (int i = 0; i < LB; ++i) Bs[buf][b_kk[i]][b_nn[i]] = rb[i];
  };

  T acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = (T)0;

  // FP64: padding is not multiplied (a padded row or column of 16 costs the FP64 pipe as much as a
  // real one): the 16-row / 16-column groups of the tile with a row or column inside the matrix
  constexpr bool SKIP = std::is_same<T, double>::value;
  const int imax = SKIP ? (int)min((int64_t)TM, (d.M - m0 + NTY - 1) / NTY) : TM;
  const int jmax = SKIP ? (int)min((int64_t)TN, (d.N - n0 + NTX - 1) / NTX) : TN;
  const bool whole = imax == TM && jmax == TN;

  int buf = 0;
  if (kbeg < kend) {
    load_tiles(kbeg);
    store_tiles(0);
    __syncthreads();
    for (int64_t k0 = kbeg; k0 < kend; k0 += BK) {
      const bool has_next = (k0 + BK < kend);
      if (has_next) load_tiles(k0 + BK);
      if (SKIP && (!whole || kend - k0 < BK)) {
        const int kn = (int)min((int64_t)BK, kend - k0);
        for (int kk = 0; kk < kn; ++kk) {
          T a[TM], b[TN];
#pragma unroll
          for (int i = 0; i < TM; ++i) a[i] = As[buf][kk][ty + i * NTY];
#pragma unroll
          for (int j = 0; j < TN; ++j) b[j] = Bs[buf][kk][tx + j * NTX];
#pragma unroll
          for (int i = 0; i < TM; ++i)
            if (i < imax) {
#pragma unroll
              for (int j = 0; j < TN; ++j)
                if (j < jmax) acc[i][j] = madd(a[i], b[j], acc[i][j]);
            }
        }
      } else
#pragma unroll
      for (int kk = 0; kk < BK; ++kk) {
        T a[TM], b[TN];
        if constexpr (VEC) {
#pragma unroll
          for (int i = 0; i < TM; i += 4) *reinterpret_cast<float4*>(a + i) = *reinterpret_cast<const float4*>(&As[buf][kk][row(i)]);
#pragma unroll
          for (int j = 0; j < TN; j += 4) *reinterpret_cast<float4*>(b + j) = *reinterpret_cast<const float4*>(&Bs[buf][kk][col(j)]);
        } else {
#pragma unroll
          for (int i = 0; i < TM; ++i) a[i] = As[buf][kk][row(i)];
#pragma unroll
          for (int j = 0; j < TN; ++j) b[j] = Bs[buf][kk][col(j)];
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[i][j] = madd(a[i], b[j], acc[i][j]);
      }
      if (has_next) {
        store_tiles(buf ^ 1);
        __syncthreads();
        buf ^= 1;
      }
    }
  }

  if (ksplit == 1) {
    const T alpha = (T)d.alpha, beta = (T)d.beta;
    if constexpr (VEC && std::is_same<TC, float>::value) {
      // whole groups of four contiguous results
      if (d.c_m == 1 && d.m_div <= 0 && m0 + BM <= d.M && d.c_n % 4 == 0 && (d.n_div <= 0 || d.c_n2 % 4 == 0) &&
          (reinterpret_cast<uintptr_t>(C) & 15) == 0) {
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          const int64_t gn = n0 + col(j);
          if (gn >= d.N) continue;
          float* p0 = C + m0 + off2(gn, d.n_div, d.c_n, d.c_n2);
#pragma unroll
          for (int i = 0; i < TM; i += 4) {
            float4* p = reinterpret_cast<float4*>(p0 + row(i));
            float4 v = make_float4(alpha * acc[i][j], alpha * acc[i + 1][j], alpha * acc[i + 2][j], alpha * acc[i + 3][j]);
            if (beta != 0.f) {
              const float4 o = *p;
              v = make_float4(madd(beta, o.x, v.x), madd(beta, o.y, v.y), madd(beta, o.z, v.z), madd(beta, o.w, v.w));
            }
            *p = v;
          }
        }
        return;
      }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int64_t gm = m0 + row(i);
      if (gm >= d.M) continue;
      const int64_t cm = off2(gm, d.m_div, d.c_m, d.c_m2);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int64_t gn = n0 + col(j);
        if (gn >= d.N) continue;
        TC* p = C + cm + off2(gn, d.n_div, d.c_n, d.c_n2);
        T v = alpha * acc[i][j];
        if (beta != (T)0) v = madd(beta, (T)(*p), v);
        *p = (TC)v;
      }
    }
  } else {
    // split-K partial sums in the workspace, [split][batch][M][N] (FP32: [N][M], the lanes' order)
    T* W = ws + ((int64_t)split * (d.batch1 * d.batch2) + bidx) * d.M * d.N;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int64_t gm = m0 + row(i);
      if (gm >= d.M) continue;
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int64_t gn = n0 + col(j);
        if (gn < d.N) W[VEC ? gn * d.M + gm : gm * d.N + gn] = acc[i][j];
      }
    }
  }
}

// Fixed-order reduction of the split-K partials: C = alpha * sum_s W[s] + beta * C.
template <typename T, typename TC>
__global__ void splitk_reduce_kernel(GemmDesc d, int ksplit, const T* __restrict__ ws, const int* only_if) {
  if (only_if != nullptr && *only_if == 0) return;
  const int64_t nb = d.batch1 * d.batch2;
  const int64_t total = nb * d.M * d.N;
  const T alpha = (T)d.alpha, beta = (T)d.beta;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    constexpr bool MFAST = std::is_same<T, float>::value;  // gemm_kernel's order of the partial sums
    const int64_t n = MFAST ? (e / d.M) % d.N : e % d.N;
    const int64_t m = MFAST ? e % d.M : (e / d.N) % d.M;
    const int64_t bidx = e / (d.N * d.M);
    const int64_t b1 = bidx % d.batch1, b2 = bidx / d.batch1;
    T s = (T)0;
    for (int k = 0; k < ksplit; ++k) s += ws[(int64_t)k * total + e];
    TC* p = static_cast<TC*>(d.C) + b1 * d.c_b1 + b2 * d.c_b2 + off2(m, d.m_div, d.c_m, d.c_m2) +
            off2(n, d.n_div, d.c_n, d.c_n2);
    T v = alpha * s;
    if (beta != (T)0) v = madd(beta, (T)(*p), v);
    *p = (TC)v;
  }
}

template <typename Cfg>
int choose_split(const GemmDesc& d, int num_sms) {
  const int64_t tiles = ((d.M + Cfg::BM - 1) / Cfg::BM) * ((d.N + Cfg::BN - 1) / Cfg::BN) *
                        d.batch1 * d.batch2;
  if (tiles >= 2 * (int64_t)num_sms) return 1;
  int64_t want = (2 * (int64_t)num_sms + tiles - 1) / tiles;
  const int64_t kmax = d.K / (4 * Cfg::BK);
  want = std::min<int64_t>(want, std::max<int64_t>(kmax, 1));
  want = std::min<int64_t>(want, 32);
  return (int)std::max<int64_t>(want, 1);
}

// Tile and K split of a native FP64 GEMM, by the time they take (us): blocks in waves over the SMs
// at 16-padded rows x columns x k / 2 clocks (1.9 GHz), a K tile at least ~0.5 us (load latency),
// the reduction of the partial sums ~3 us.  24 x 60 x 2016: 64 x 64 tiles in 31 splits 95 us,
// 32 x 32 tiles in 63 splits 15 us.
struct F64Choice {
  bool small;
  int split;
  double us;
};
template <typename Cfg>
void f64_candidates(const GemmDesc& d, int num_sms, bool small, F64Choice& best) {
  const int64_t nb = d.batch1 * d.batch2;
  const int64_t tiles = ((d.M + Cfg::BM - 1) / Cfg::BM) * ((d.N + Cfg::BN - 1) / Cfg::BN) * nb;
  const double rows = (double)std::min<int64_t>(Cfg::BM, (d.M + 15) / 16 * 16);
  const double cols = (double)std::min<int64_t>(Cfg::BN, (d.N + 15) / 16 * 16);
  for (int s = 1; s <= 128; s *= 2) {
    if (s > 1 && ((int64_t)s * 2 * Cfg::BK > d.K || tiles * s > 8 * (int64_t)num_sms ||
                  (double)s * d.M * d.N * nb * 8 > 256e6))
      break;
    const double kc = (double)div_up(div_up(d.K, s), Cfg::BK) * Cfg::BK;
    const double waves = (double)div_up(tiles * s, num_sms);
    const double t = std::max(waves * rows * cols * std::min(kc, (double)d.K) / 2.0 / 1900.0, kc / Cfg::BK * 0.5) +
                     (s > 1 ? 3.0 + (double)s * d.M * d.N * nb * 8 / 3e6 : 0.0);
    if (best.us < 0.0 || t < best.us) best = F64Choice{small, s, t};
  }
}
F64Choice f64_choice(const GemmDesc& d, int num_sms) {
  F64Choice best{false, 1, -1.0};
  f64_candidates<CfgF64>(d, num_sms, false, best);
  f64_candidates<CfgF64S>(d, num_sms, true, best);
  best.us += 3.0;
  return best;
}

template <typename T, typename Cfg, typename TA, typename TB, typename TC>
cudaError_t run(const GemmDesc& d, cudaStream_t stream, void* workspace, size_t ws_bytes, int num_sms,
                const int* only_if = nullptr, int split = 0) {
  const int64_t nb = d.batch1 * d.batch2;
  int ksplit = split > 0 ? split : choose_split<Cfg>(d, num_sms);
  if (ksplit > 1) {
    const size_t need = (size_t)ksplit * nb * d.M * d.N * sizeof(T);
    if (workspace == nullptr || need > ws_bytes) ksplit = 1;
  }
  int64_t kchunk = (d.K + ksplit - 1) / ksplit;
  kchunk = ((kchunk + Cfg::BK - 1) / Cfg::BK) * Cfg::BK;
  ksplit = (int)((d.K + kchunk - 1) / kchunk);
  const int64_t gx = (d.M + Cfg::BM - 1) / Cfg::BM;
  const int64_t gy = (d.N + Cfg::BN - 1) / Cfg::BN;
  if (gy > 65535) {
    // more column tiles than the grid's y holds (an output of millions of columns): several launches, on
    // whole blocks of a two-level column index
    int64_t step = (int64_t)65535 * Cfg::BN;
    if (d.n_div > 0) step = step / d.n_div * d.n_div;
    if (step == 0) return cudaErrorInvalidConfiguration;
    for (int64_t n0 = 0; n0 < d.N; n0 += step) {
      GemmDesc s = d;
      s.N = std::min(step, d.N - n0);
      const int64_t ob = d.n_div > 0 ? n0 / d.n_div * d.b_n2 : n0 * d.b_n;
      const int64_t oc = d.n_div > 0 ? n0 / d.n_div * d.c_n2 : n0 * d.c_n;
      s.B = static_cast<const char*>(d.B) + ob * (int64_t)sizeof(TB);
      s.C = static_cast<char*>(d.C) + oc * (int64_t)sizeof(TC);
      const cudaError_t err = run<T, Cfg, TA, TB, TC>(s, stream, workspace, ws_bytes, num_sms, only_if, split);
      if (err != cudaSuccess) return err;
    }
    return cudaSuccess;
  }
  // batches beyond the grid z limit are issued in several launches
  const int64_t zmax = 65535 / ksplit;
  for (int64_t b0 = 0; b0 < nb; b0 += zmax) {
    const int64_t bn = std::min<int64_t>(zmax, nb - b0);
    GemmDesc s = d;
    if (b0 != 0 || bn != nb) {
      if (d.batch2 != 1) return cudaErrorInvalidConfiguration;
      s.A = static_cast<const char*>(d.A) + b0 * d.a_b1 * (int64_t)sizeof(TA);
      s.B = static_cast<const char*>(d.B) + b0 * d.b_b1 * (int64_t)sizeof(TB);
      s.C = static_cast<char*>(d.C) + b0 * d.c_b1 * (int64_t)sizeof(TC);
      s.batch1 = bn;
    }
    dim3 grid((unsigned)gx, (unsigned)gy, (unsigned)(bn * ksplit));
    gemm_kernel<T, Cfg, TA, TB, TC><<<grid, 256, 0, stream>>>(s, ksplit, kchunk, static_cast<T*>(workspace), only_if);
    count_launch();
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    if (ksplit > 1) {
      const int64_t total = bn * d.M * d.N;
      const int64_t blocks = std::min<int64_t>((total + 255) / 256, 8 * (int64_t)num_sms);
      splitk_reduce_kernel<T, TC><<<(unsigned)blocks, 256, 0, stream>>>(s, ksplit, static_cast<const T*>(workspace),
                                                                                only_if);
      count_launch();
      err = cudaGetLastError();
      if (err != cudaSuccess) return err;
    }
  }
  return cudaSuccess;
}

cudaError_t run_f64(const GemmDesc& d, cudaStream_t stream, void* workspace, size_t ws_bytes, int num_sms,
                    const int* only_if) {
  const F64Choice f = f64_choice(d, num_sms);
  if (f.small) return run<double, CfgF64S, double, double, double>(d, stream, workspace, ws_bytes, num_sms, only_if, f.split);
  return run<double, CfgF64, double, double, double>(d, stream, workspace, ws_bytes, num_sms, only_if, f.split);
}

// Tile and K split of an FP32 GEMM by the time they take (us): waves of blocks, one to an SM, at
// ~0.11 us per k of a 128 x 128 or 256 x 64 tile (~65 % of the FP32 rate), the reduction of the partial
// sums ~3 us and its traffic.  2000 x 180 x 36000 and its like: 128 x 128 tiles in 10 splits (three
// waves, 30 % of the columns padding) at 13.5 TF/s, with this choice and 16-byte shared-memory reads
// at 21.7.
struct F32Choice {
  bool tall;
  int split;
  double us;
};
template <typename Cfg>
void f32_candidates(const GemmDesc& d, int num_sms, bool tall, F32Choice& best) {
  const int64_t nb = d.batch1 * d.batch2;
  const int64_t tiles = div_up(d.M, Cfg::BM) * div_up(d.N, Cfg::BN) * nb;
  for (int s = 1; s <= 64; ++s) {
    if (s > 1 && ((int64_t)s * 4 * Cfg::BK > d.K || (double)s * d.M * d.N * nb * 4 > 512e6 || tiles >= 8 * (int64_t)num_sms))
      break;
    const double kc = (double)div_up(div_up(d.K, s), Cfg::BK) * Cfg::BK;
    const double t = (double)div_up(tiles * s, num_sms) * (kc * 0.11 + 3.0) +
                     (s > 1 ? 3.0 + (double)(s + 2) * d.M * d.N * nb * 4 / 4.5e6 : 0.0);
    if (best.us < 0.0 || t < best.us) best = F32Choice{tall, s, t};
  }
}
F32Choice f32_choice(const GemmDesc& d, int num_sms) {
  F32Choice best{false, 1, -1.0};
  f32_candidates<CfgF32>(d, num_sms, false, best);
  f32_candidates<CfgF32Tall>(d, num_sms, true, best);
  return best;
}

}  // namespace

size_t gemm_workspace_bytes(const GemmDesc& d, size_t elem_bytes, int num_sms) {
  int s;
  if (elem_bytes == 8) s = std::max(choose_split<CfgF64>(d, num_sms), f64_choice(d, num_sms).split);
  else s = f32_choice(d, num_sms).split;
  if (s <= 1) return 0;
  return (size_t)s * d.batch1 * d.batch2 * d.M * d.N * elem_bytes;
}

template <typename T, typename TA, typename TB, typename TC>
cudaError_t gemm(const GemmDesc& d, cudaStream_t stream, void* workspace, size_t ws_bytes, int num_sms) {
  if (d.M <= 0 || d.N <= 0) return cudaSuccess;
  const int64_t nb = d.batch1 * d.batch2;
  if (d.K <= 0) {
    // C = beta * C (alpha term is empty)
    GemmDesc z = d;
    z.K = 0;
    splitk_reduce_kernel<T, TC><<<std::max<int64_t>(1, std::min<int64_t>(4096, (nb * d.M * d.N + 255) / 256)), 256, 0, stream>>>(z, 0, (const T*)nullptr, nullptr);
    count_launch();
    return cudaGetLastError();
  }
  if constexpr (std::is_same<T, double>::value) {
    return run_f64(d, stream, workspace, ws_bytes, num_sms, nullptr);
  } else if constexpr (sizeof(T) == 8) {
    return run<T, CfgF64, TA, TB, TC>(d, stream, workspace, ws_bytes, num_sms);
  } else {
    const F32Choice f = f32_choice(d, num_sms);
    if (f.tall) return run<T, CfgF32Tall, TA, TB, TC>(d, stream, workspace, ws_bytes, num_sms, nullptr, f.split);
    return run<T, CfgF32, TA, TB, TC>(d, stream, workspace, ws_bytes, num_sms, nullptr, f.split);
  }
}

#define CPHF_INST(T, TA, TB, TC) \
  template cudaError_t gemm<T, TA, TB, TC>(const GemmDesc&, cudaStream_t, void*, size_t, int);
CPHF_INST(double, double, double, double)
CPHF_INST(float, float, float, float)
CPHF_INST(float, float, float, double)
CPHF_INST(float, float, double, float)
CPHF_INST(float, double, float, float)
CPHF_INST(float, float, double, double)
CPHF_INST(float, double, double, float)
CPHF_INST(float, double, float, double)
CPHF_INST(float, double, double, double)
#undef CPHF_INST

cudaError_t gemm_f64_emulated(const GemmDesc& d, cudaStream_t stream, void* workspace, size_t ws_bytes,
                              int num_sms) {
  return gemm<dfloat, double, double, double>(d, stream, workspace, ws_bytes, num_sms);
}

cudaError_t gemm_f64_if(const GemmDesc& d, cudaStream_t stream, void* workspace, size_t ws_bytes, int num_sms,
                        const int* flag) {
  if (d.M <= 0 || d.N <= 0 || d.K <= 0) return cudaSuccess;
  return run_f64(d, stream, workspace, ws_bytes, num_sms, flag);
}

double gemm_f64_us(const GemmDesc& d, int num_sms) { return f64_choice(d, num_sms).us; }

}  // namespace cphf
