// Element-wise, reduction and small dense-algebra kernels, see kernels.cuh.

#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"

namespace cphf {
thread_local int64_t* g_launch_counter = nullptr;
std::atomic<int64_t> g_state_generation{0};

namespace {

constexpr int kThreads = 256;

inline unsigned grid_for(int64_t total, int64_t cap = 1 << 20) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(div_up(total, kThreads), cap));
}

// (32 x 32 tiles of the triangle, written twice, transposed through shared memory: reading the packed
// rows down a column took 1.4 ms at nao 400, naux 1333, these 0.7)
__global__ void unpack_cderi_kernel(const double* __restrict__ tp, int64_t nao, int64_t naux,
                                    double* __restrict__ dense) {
  __shared__ double tile[32][33];
  const int64_t nao_tp = nao * (nao + 1) / 2;
  const int nt = (int)((nao + 31) / 32);
  // tile (ti, tj), ti <= tj, of the upper triangle
  int tj = (int)((sqrtf(8.f * (float)blockIdx.x + 1.f) - 1.f) * 0.5f);
  while ((tj + 1) * (tj + 2) / 2 <= (int)blockIdx.x) ++tj;
  while (tj * (tj + 1) / 2 > (int)blockIdx.x) --tj;
  const int ti = (int)blockIdx.x - tj * (tj + 1) / 2;
  if (tj >= nt) return;
  const int64_t m0 = 32 * (int64_t)ti, n0 = 32 * (int64_t)tj;
  for (int64_t P = blockIdx.y; P < naux; P += gridDim.y) {
    const double* src = tp + nao_tp * P;
    double* dst = dense + nao * nao * P;
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
      const int64_t hi = n0 + y, lo = m0 + threadIdx.x;
      if (hi < nao && lo <= hi) tile[y][threadIdx.x] = src[hi * (hi + 1) / 2 + lo];
    }
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
      const int64_t nu = n0 + y, mu = m0 + threadIdx.x;  // rows nu of the tile, its diagonal mirrored
      if (nu < nao && mu < nao && (ti != tj || mu <= nu)) dst[mu + nao * nu] = tile[y][threadIdx.x];
      const int64_t nu2 = m0 + y, mu2 = n0 + threadIdx.x;
      if (nu2 < nao && mu2 < nao && (ti != tj || mu2 > nu2)) dst[mu2 + nao * nu2] = tile[threadIdx.x][y];
    }
    __syncthreads();
  }
}

template <typename TY>
__global__ void dimless_kernel(const TY* __restrict__ y, const double* __restrict__ x, int64_t ldx,
                               const double* __restrict__ e, int64_t nmo, int64_t nocc, int64_t nb,
                               double shift, double* __restrict__ out, int64_t ldo) {
  const int64_t per = nmo * nocc;
  const int64_t total = per * nb;
  const int64_t nvir = nmo - nocc;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t a = t / per;
    const int64_t r = t - a * per;
    const int64_t p = r % nmo, i = r / nmo;
    double v = 0.0;
    if (p >= nocc) {
      double yv = (double)y[(p - nocc) + nvir * (i + nocc * a)];
      if (shift != 0.0) yv -= shift * x[r + ldx * a];
      v = yv / (e[p] - e[i] + shift);
    }
    out[r + ldo * a] = v;
  }
}

template <typename T>
__global__ void xc_rho_kernel(const T* __restrict__ aobra, int64_t ld_aobra,
                              const T* __restrict__ ket, int64_t npts, int64_t nocc, int64_t nb,
                              T* __restrict__ rho, int64_t ld_rho) {
  const int64_t total = npts * nb;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t g = t % npts, a = t / npts;
    const T* k = ket + g + npts * nocc * a;
    T s = (T)0;
    for (int64_t i = 0; i < nocc; ++i) s = fma(aobra[g + ld_aobra * i], k[npts * i], s);
    rho[g + ld_rho * a] = s;
  }
}

template <typename T>
__global__ void xc_q_kernel(const T* __restrict__ aobra, int64_t ld_aobra,
                            const double* __restrict__ w, const double* __restrict__ fxc,
                            int64_t fxc_ld, int nspin, int sout, const T* __restrict__ rho,
                            int64_t ld_rho, int64_t ld_rho_spin, int64_t npts, int64_t nocc,
                            int64_t nb, T* __restrict__ q) {
  const int64_t total = npts * nb;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t g = t % npts, a = t / npts;
    double f;
    if (nspin == 1) {
      f = fxc[g] * (double)rho[g + ld_rho * a];
    } else {
      f = fxc[g + fxc_ld * (0 + 2 * sout)] * (double)rho[g + ld_rho * a] +
          fxc[g + fxc_ld * (1 + 2 * sout)] * (double)rho[g + ld_rho * a + ld_rho_spin];
    }
    const T wv = (T)(w[g] * f);
    T* qq = q + g + npts * nocc * a;
    for (int64_t i = 0; i < nocc; ++i) qq[npts * i] = wv * aobra[g + ld_aobra * i];
  }
}

// ---- residual and column norms ---------------------------------------------------------
constexpr int kResRowsPerBlock = 2048;

__device__ __forceinline__ double block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0) {
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) s += sh[k];
  }
  __syncthreads();
  return s;  // valid in thread 0
}

__global__ void residual_kernel(const double* __restrict__ b, const double* __restrict__ x,
                                const double* __restrict__ ax, double* __restrict__ r, int64_t n,
                                double* __restrict__ partials) {
  __shared__ double sh[32];
  const int64_t j = blockIdx.y;
  const int64_t r0 = (int64_t)blockIdx.x * kResRowsPerBlock;
  const int64_t r1 = min(n, r0 + kResRowsPerBlock);
  double acc = 0.0;
  for (int64_t row = r0 + threadIdx.x; row < r1; row += blockDim.x) {
    const int64_t e = row + n * j;
    const double v = b[e] - x[e] - ax[e];
    r[e] = v;
    acc = fma(v, v, acc);
  }
  const double s = block_sum(acc, sh);
  if (threadIdx.x == 0) partials[blockIdx.x + (int64_t)gridDim.x * j] = s;
}

__global__ void sum_partials_kernel(const double* __restrict__ partials, int64_t nblk, int64_t nb,
                                    double* __restrict__ out) {
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j >= nb) return;
  double s = 0.0;
  for (int64_t k = 0; k < nblk; ++k) s += partials[k + nblk * j];
  out[j] = s;
}

// ---- modified Gram-Schmidt --------------------------------------------------------------
// All columns in one cooperative launch.  Right-looking MGS needs two grid-wide steps per
// projector (its dot products with the columns after it, then their update); as launches of their
// own these cost more than the arithmetic, and even inside one launch the two barriers and the
// reduction between them take ~10 us.  Here each block keeps its rows for the whole sweep, a
// step's update also forms the partial dot products of the next, and up to kMgsPanel = 4 columns
// project at once:
//   the dots of the panel's columns v_0 .. v_3 with every later column are taken before the panel
//   is orthogonalised, and the coefficients follow by substitution, c_qj = <v_q', v_j> / d_q with
//   <v_q', v_j> = <v_q, v_j> - sum_{r<q} c_rq <v_r', v_j> and d_q = <v_q', v_q>:
// the same projections as column by column.  The substitution loses digits where a panel column
// leans on those before it; a column whose d_q falls below kMgsMinRatio <v_q, v_q> (or near lindep)
// ends the panel before it, at worst after the first column, which is plain MGS.  Relative error of the
// vectors, 4000 x 36 with correlations 0.1 / 0.5 / 0.8 / 0.96: ratio 1e-2 2.1 / 3.9 / 10.3 / 64e-16, 0.9
// 2.1 / 2.5 / 3.2 / 6.6e-16, column by column 2.1 / 2.3 / 2.8 / 4.9e-16; the solves measured run as fast.
// Bound by the FP64 pipe where the rows are many (n m^2 FMA pairs, one pair a clock and SM: 2.0 of
// the 3.8 ms at 36000 x 180; with two launches per column it took 12 ms), else by the ~20 us a
// step's barriers, reduction and latencies take: 6561 x 72 0.42 ms (3.0 ms), 741 x 18 68 us (~150).
constexpr int kMgsThreads = 512, kMgsWarps = kMgsThreads / 32, kMgsPanel = 4;
constexpr double kMgsMinRatio = 0.9;
constexpr int64_t kMgsStage = 2048;        // rows of a block whose projectors sit in shared memory
constexpr int64_t kMgsCoefs = 1024;        // columns whose coefficients sit in shared memory
constexpr unsigned kMgsSpins = 1u << 24;   // bound of the barrier's wait
constexpr int64_t kMgsMaxBlocks = 256;

// Waits until every block has arrived `target` / gridDim.x times; false when the bound is reached.
__device__ __forceinline__ bool mgs_barrier(unsigned* bar, unsigned target) {
  __shared__ int ok;
  __syncthreads();
  if (gridDim.x > 1) {
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(bar, 1u);
      unsigned seen = 0, spin = 0;
      do {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
      } while (seen < target && ++spin < kMgsSpins);
      ok = seen >= target;
    }
    __syncthreads();
    return ok != 0;
  }
  return true;
}

// Sum of each of the N (a power of two, at most 32) values over the lanes: every exchange halves
// the values a lane keeps, N + log2(32 / N) shuffles instead of 5 N.  The total of value i ends in
// the lanes i (32 / N) .. (i + 1) (32 / N) - 1.
template <int N>
__device__ __forceinline__ double warp_totals(double (&v)[N], int lane) {
  int o = 16;
#pragma unroll
  for (int h = N / 2; h >= 1; h /= 2, o /= 2) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double send = up ? v[i] : v[i + h];
      v[i] = (up ? v[i + h] : v[i]) + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  double s = v[0];
  for (; o > 0; o /= 2) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

struct MgsArgs {
  double* V;
  int64_t n, m, rows, stage;  // rows per block, of which in shared memory
  double lindep;
  double* ip;
  int* keep;
  double* coef;      // [m][kMgsPanel]; coef[4 m]: columns projected by the step
  double* partials;  // [m][kMgsPanel][block]: <v_(p0 + q), v_j> of the block's rows
  unsigned* bar;
};

__global__ void __launch_bounds__(kMgsThreads) mgs_kernel(MgsArgs a) {
  constexpr int B = kMgsPanel;
  extern __shared__ double mgs_smem[];
  const int64_t n = a.n, m = a.m, nblk = gridDim.x, stage = a.stage;
  const int64_t r0 = (int64_t)blockIdx.x * a.rows, len = max((int64_t)0, min(n, r0 + a.rows) - r0);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double* const Vb = a.V + r0;
  double* cur = mgs_smem;                       // [B][stage]: the panel (orthogonalised once projecting)
  double* nxt = mgs_smem + B * stage;           // the next panel
  double* const cfs = mgs_smem + 2 * B * stage; // [columns][B]: coefficients of the step
  unsigned target = 0;
  int64_t p0 = 0;
  int w = (int)min((int64_t)B, m);
  // row r of panel column q (panel starting at column p)
  auto panel = [&](const double* st, int64_t p, int q, int64_t r) { return r < stage ? st[q * stage + r] : Vb[r + n * (p + q)]; };
  auto publish = [&](double (&acc)[B], int64_t j, int used) {
    const double t = warp_totals<B>(acc, lane);
    const int q = lane >> 3;
    if ((lane & 7) == 0 && q < used) a.partials[blockIdx.x + nblk * (j * B + q)] = t;
  };
  for (int64_t e = threadIdx.x; e < w * len; e += blockDim.x) {
    const int64_t q = e / len, r = e - q * len;
    if (r < stage) cur[q * stage + r] = Vb[r + n * q];
  }
  __syncthreads();
  for (int64_t j = wid; j < m; j += kMgsWarps) {
    // four sums a lane: shorter chains round less (these columns may be the most correlated ones)
    double acc[B] = {0.0, 0.0, 0.0, 0.0}, part[3][B] = {};
    for (int64_t r0 = 0; r0 < len; r0 += 128) {  // (warp-uniform, the last rows predicated)
      double v[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int64_t r = r0 + 32 * h + lane;
        v[h] = r < len ? Vb[r + n * j] : 0.0;
      }
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int64_t r = r0 + 32 * h + lane;
        if (r0 + 32 * h >= len) break;
        double* const a4 = h == 0 ? acc : part[h - 1];
#pragma unroll
        for (int q = 0; q < B; ++q)
          if (q < w) a4[q] = fma(v[h], r < len ? panel(cur, 0, q, r) : 0.0, a4[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < B; ++q) acc[q] = (acc[q] + part[0][q]) + (part[1][q] + part[2][q]);
    publish(acc, j, w);
  }
  while (true) {
    target += gridDim.x;
    if (!mgs_barrier(a.bar, target)) {
      if (threadIdx.x == 0) a.keep[0] = -1;  // reported by the host
      return;
    }
    // coefficients of column j: one warp per column over the grid, each from the panel's own dot
    // products (10) and the column's (4)
    for (int64_t j = p0 + (int64_t)wid * nblk + blockIdx.x; j < m; j += nblk * kMgsWarps) {
      double v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = 0.0;
      for (int64_t k = lane; k < nblk; k += 32) {
        int i = 0;
#pragma unroll
        for (int q = 0; q < B; ++q)
#pragma unroll
          for (int r = 0; r <= q; ++r, ++i)
            if (q < w) v[i] += __ldcg(a.partials + k + nblk * ((p0 + q) * B + r));
#pragma unroll
        for (int q = 0; q < B; ++q)
          if (q < w) v[10 + q] += __ldcg(a.partials + k + nblk * (j * B + q));
      }
      const double tot = warp_totals<16>(v, lane);  // total i in lanes 2 i, 2 i + 1
      // g[r][q] = <v_r, v_(p0 + q)> (r <= q), then <v_r', .>
      double g[B][B], d[B], rd[B], c[B][B], x[B];
      int width = w;
      {
        int i = 0;
#pragma unroll
        for (int q = 0; q < B; ++q)
#pragma unroll
          for (int r = 0; r <= q; ++r, ++i) g[r][q] = __shfl_sync(0xffffffffu, tot, 2 * i);
      }
#pragma unroll
      for (int q = 0; q < B; ++q) x[q] = __shfl_sync(0xffffffffu, tot, 2 * (10 + q));
#pragma unroll
      for (int q = 0; q < B; ++q) {
        const double full = g[q][q];
#pragma unroll
        for (int r = 0; r < q; ++r) {
#pragma unroll
          for (int t = 0; t < r; ++t) g[r][q] = fma(-c[t][r], g[t][q], g[r][q]);
          c[r][q] = g[r][q] * rd[r];
          g[q][q] = fma(-c[r][q], g[r][q], g[q][q]);
        }
        d[q] = g[q][q];
        rd[q] = 1.0 / d[q];
        // (a NaN fails the comparison)
        if (q > 0 && q < width && !(d[q] > kMgsMinRatio * full && d[q] > 4.0 * a.lindep)) width = q;
      }
      const bool kept0 = d[0] > a.lindep;
      if (!kept0) width = 1;
      const int64_t e = j - p0;
      if (e < width) {  // a column of the panel itself
        double de = d[0];
#pragma unroll
        for (int q = 0; q < B; ++q) x[q] = 0.0;
#pragma unroll
        for (int q = 1; q < B; ++q)
          if (e == q) {
            de = d[q];
#pragma unroll
            for (int r = 0; r < q; ++r) x[r] = c[r][q];
          }
        if (lane == 0) {
          a.ip[j] = de;
          a.keep[j] = de > a.lindep ? 1 : 0;
          if (e == 0) a.coef[B * m] = (double)width;
        }
      } else {
#pragma unroll
        for (int q = 0; q < B; ++q) {
#pragma unroll
          for (int r = 0; r < q; ++r) x[q] = fma(-c[r][q], x[r], x[q]);
        }
#pragma unroll
        for (int q = 0; q < B; ++q) x[q] = q < width && kept0 ? x[q] * rd[q] : 0.0;
      }
      if (lane == 0) {
#pragma unroll
        for (int q = 0; q < B; ++q) a.coef[j * B + q] = x[q];
      }
    }
    target += gridDim.x;
    if (!mgs_barrier(a.bar, target)) {
      if (threadIdx.x == 0) a.keep[0] = -1;
      return;
    }
    const int64_t nc = min(m - p0, kMgsCoefs);
    for (int64_t e = threadIdx.x; e < nc * B; e += blockDim.x) cfs[e] = __ldcg(a.coef + p0 * B + e);
    const int width = (int)__ldcg(a.coef + B * m);
    const int64_t p1 = p0 + width;
    const int w1 = (int)max((int64_t)0, min((int64_t)B, m - p1));
    __syncthreads();
    auto coef = [&](int64_t j, int t) { return j - p0 < kMgsCoefs ? cfs[(j - p0) * B + t] : __ldcg(a.coef + j * B + t); };
    // the panel's own columns, a row to a thread
    if (width > 1)
      for (int64_t r = threadIdx.x; r < len; r += blockDim.x) {
        double v[B];
#pragma unroll
        for (int q = 0; q < B; ++q) {
          v[q] = q < width ? panel(cur, p0, q, r) : 0.0;
#pragma unroll
          for (int t = 0; t < q; ++t) v[q] = fma(-coef(p0 + min(q, width - 1), t), v[t], v[q]);
          if (q > 0 && q < width) {
            if (r < stage) cur[q * stage + r] = v[q];
            Vb[r + n * (p0 + q)] = v[q];
          }
        }
      }
    if (p1 >= m) return;
    __syncthreads();
    // the next panel's columns first: they are the projectors of the next step
    for (int64_t e = threadIdx.x; e < w1 * len; e += blockDim.x) {
      const int64_t q = e / len, r = e - q * len;
      double v = Vb[r + n * (p1 + q)];
#pragma unroll
      for (int t = 0; t < B; ++t)
        if (t < width) v = fma(-coef(p1 + q, t), panel(cur, p0, t, r), v);
      if (r < stage) nxt[q * stage + r] = v;
      Vb[r + n * (p1 + q)] = v;
    }
    __syncthreads();
    for (int64_t j = p1 + wid; j < m; j += kMgsWarps) {
      double acc[B] = {0.0, 0.0, 0.0, 0.0}, cj[B];
      const bool mine = j >= p1 + w1;  // not yet updated
#pragma unroll
      for (int t = 0; t < B; ++t) cj[t] = mine && t < width ? coef(j, t) : 0.0;
      if (width == B && w1 == B && mine && len <= stage) {
#pragma unroll 4
        for (int64_t r = lane; r < len; r += 32) {
          double v = Vb[r + n * j];
#pragma unroll
          for (int t = 0; t < B; ++t) v = fma(-cj[t], cur[t * stage + r], v);
          Vb[r + n * j] = v;
#pragma unroll
          for (int q = 0; q < B; ++q) acc[q] = fma(v, nxt[q * stage + r], acc[q]);
        }
      } else {
        for (int64_t r = lane; r < len; r += 32) {
          double v = Vb[r + n * j];
          if (mine) {
#pragma unroll
            for (int t = 0; t < B; ++t)
              if (t < width) v = fma(-cj[t], panel(cur, p0, t, r), v);
            Vb[r + n * j] = v;
          }
#pragma unroll
          for (int q = 0; q < B; ++q)
            if (q < w1) acc[q] = fma(v, panel(nxt, p1, q, r), acc[q]);
        }
      }
      publish(acc, j, w1);
    }
    double* const tmp = cur;
    cur = nxt;
    nxt = tmp;
    p0 = p1;
    w = w1;
  }
}

// Blocks of the sweep: a step takes 2 n m clocks of FP64 work over the blocks and ~15000 clocks for
// the two barriers and the reduction between them (a third of that with a single block).
int64_t mgs_blocks(int64_t n, int64_t m, int num_sms) {
  const double work = 2.0 * (double)n * (double)m;
  if (work < 16000.0) return 1;
  return std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(num_sms, kMgsMaxBlocks),
                                                std::min<int64_t>((int64_t)(work / 4000.0), div_up(n, 32))));
}

__global__ void gather_cols_kernel(const double* __restrict__ src, int64_t n,
                                   const int* __restrict__ idx, int64_t cnt, double* __restrict__ dst,
                                   int64_t ld_dst) {
  const int64_t total = n * cnt;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = t % n, j = t / n;
    dst[r + ld_dst * j] = src[r + n * (int64_t)idx[j]];
  }
}

__global__ void scale_rows_kernel(double* coeff, int64_t ldc, const double* ip, int64_t m, int64_t nb) {
  const int64_t total = m * nb;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t % m, j = t / m;
    coeff[i + ldc * j] /= ip[i];
  }
}

__global__ void add_diag_kernel(double* h, int64_t ldh, const double* ip, int64_t m) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < m) h[i + ldh * i] += ip[i];
}

// ---- LU with partial pivoting -----------------------------------------------------------
// Blocked right-looking LU of h with the right-hand sides carried along: per panel of kLuPanel
// columns one CTA factors the panel (pivot search, scaling, update inside the panel), one launch
// swaps and solves the panel's rows of every column to its right, one updates the trailing tiles;
// the back substitution runs over blocks of the same width.  Launches and the panel's serial chain
// bound it (5 launches per 16 columns instead of 3 per column): m = 216, 72 right-hand sides
// 1.1 ms, m = 540, 180 right-hand sides 3.1 ms.
constexpr int kLuPanel = 16;
constexpr int kLuThreads = 512;

// The row swaps of a panel as moves: row dst[i] receives row src[i], i < count (at most two rows
// per column), so that a column loads all of them at once.
struct LuMoves {
  int count, dst[2 * kLuPanel], src[2 * kLuPanel];
};

// Panel columns [k0, k0 + w), rows [k0, m): partial pivoting, multipliers in place, the row swaps
// to *moves.  The panel sits in shared memory when it fits (`smem`).  One division per column
// (LAPACK's reciprocal scaling): a division per row would occupy the FP64 pipe longer than the
// update.
__global__ void __launch_bounds__(kLuThreads) lu_panel_kernel(double* __restrict__ h, int64_t ldh, int64_t m, int64_t k0,
                                                              int w, int smem, LuMoves* __restrict__ moves, int* info) {
  extern __shared__ double sp[];
  __shared__ unsigned long long best_v[kLuThreads / 32];
  __shared__ int best_i[kLuThreads / 32];
  __shared__ int piv_sh, piv[kLuPanel];
  __shared__ double rd_sh;
  const int rows = (int)(m - k0);
  const int64_t ld = smem ? rows : ldh;
  double* const a = smem ? sp : h + k0 + ldh * k0;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  if (smem)
    for (int64_t e = t; e < (int64_t)rows * w; e += blockDim.x) sp[e] = h[(k0 + e % rows) + ldh * (k0 + e / rows)];
  __syncthreads();
  for (int j = 0; j < w; ++j) {
    // the largest |entry| (its bit pattern orders like the value and costs no FP64 comparison; a
    // NaN never wins), the lowest row among equals; 0 when every entry is zero or NaN
    unsigned long long bv = 0;
    int bi = j;
    for (int r = j + t; r < rows; r += blockDim.x) {
      const unsigned long long v = (unsigned long long)__double_as_longlong(a[r + ld * j]) & 0x7FFFFFFFFFFFFFFFull;
      if (v > bv && v <= 0x7FF0000000000000ull) { bv = v; bi = r; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if (lane == 0) { best_v[wid] = bv; best_i[wid] = bi; }
    __syncthreads();
    if (wid == 0) {
      constexpr int NW = kLuThreads / 32;
      bv = lane < NW ? best_v[lane] : 0;
      bi = lane < NW ? best_i[lane] : rows;
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
      }
      if (lane == 0) {
        if (bv == 0) bi = j;
        piv_sh = bi;
        piv[j] = bi;
        rd_sh = 1.0 / a[bi + ld * j];
        if (bv == 0 && *info == 0) *info = (int)(k0 + j + 1);
      }
    }
    __syncthreads();
    const int p = piv_sh;
    if (p != j && t < w) {
      const double x = a[j + ld * t];
      a[j + ld * t] = a[p + ld * t];
      a[p + ld * t] = x;
    }
    __syncthreads();
    const double d = a[j + ld * j], rd = rd_sh;
    for (int r = j + 1 + t; r < rows; r += blockDim.x) {
      double l = a[r + ld * j];
      // (a pivot whose reciprocal overflows is divided by)
      if (d != 0.0) a[r + ld * j] = l = isfinite(rd) ? l * rd : l / d;
      for (int c = j + 1; c < w; ++c) a[r + ld * c] = fma(-l, a[j + ld * c], a[r + ld * c]);
    }
    __syncthreads();
  }
  if (smem)
    for (int64_t e = t; e < (int64_t)rows * w; e += blockDim.x) h[(k0 + e % rows) + ldh * (k0 + e / rows)] = sp[e];
  if (t == 0) {
    // the swaps applied in order to the identity, on the rows they touch
    int n = 0, row[2 * kLuPanel], from[2 * kLuPanel];
    for (int j = 0; j < w; ++j) {
      if (piv[j] == j) continue;
      int x = -1, y = -1;
      for (int i = 0; i < n; ++i) {
        if (row[i] == j) x = i;
        if (row[i] == piv[j]) y = i;
      }
      if (x < 0) { x = n++; row[x] = from[x] = j; }
      if (y < 0) { y = n++; row[y] = from[y] = piv[j]; }
      const int f = from[x];
      from[x] = from[y];
      from[y] = f;
    }
    for (int i = 0; i < n; ++i) {
      moves->dst[i] = (int)k0 + row[i];
      moves->src[i] = (int)k0 + from[i];
    }
    moves->count = n;
  }
}

// column c of the trailing matrix (c < m - k0 - w) or right-hand side
__device__ __forceinline__ double* lu_column(double* h, int64_t ldh, double* g, int64_t ldg, int64_t m, int64_t k1,
                                             int64_t c) {
  return c < m - k1 ? h + ldh * (k1 + c) : g + ldg * (c - (m - k1));
}

// Row swaps of the panel and the unit lower triangular solve of its w rows, one thread per column.
__global__ void lu_rows_kernel(double* __restrict__ h, int64_t ldh, double* __restrict__ g, int64_t ldg, int64_t m,
                               int64_t nrhs, int64_t k0, int w, const LuMoves* __restrict__ moves) {
  __shared__ double l[kLuPanel][kLuPanel];
  __shared__ LuMoves mv;
  for (int e = threadIdx.x; e < w * w; e += blockDim.x) l[e % w][e / w] = h[(k0 + e % w) + ldh * (k0 + e / w)];
  for (int e = threadIdx.x; e < (int)(sizeof(LuMoves) / sizeof(int)); e += blockDim.x)
    reinterpret_cast<int*>(&mv)[e] = reinterpret_cast<const int*>(moves)[e];
  __syncthreads();
  const int64_t k1 = k0 + w, cols = (m - k1) + nrhs;
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= cols) return;
  double* x = lu_column(h, ldh, g, ldg, m, k1, c);
  double s[2 * kLuPanel];
#pragma unroll
  for (int i = 0; i < 2 * kLuPanel; ++i) s[i] = i < mv.count ? x[mv.src[i]] : 0.0;
#pragma unroll
  for (int i = 0; i < 2 * kLuPanel; ++i)
    if (i < mv.count) x[mv.dst[i]] = s[i];
  double v[kLuPanel];
#pragma unroll
  for (int j = 0; j < kLuPanel; ++j) v[j] = j < w ? x[k0 + j] : 0.0;
#pragma unroll
  for (int j = 0; j < kLuPanel; ++j)
#pragma unroll
    for (int q = 0; q < j; ++q)
      if (j < w) v[j] = fma(-l[j][q], v[q], v[j]);
#pragma unroll
  for (int j = 0; j < kLuPanel; ++j)
    if (j < w) x[k0 + j] = v[j];
}

// 32 x 32 tile of rows [lo, hi) and columns: X -= A(:, k0 .. k0 + w) X(k0 .. k0 + w, :), the
// columns of the trailing matrix and the right-hand sides (forward) or the right-hand sides alone
// (back substitution, k1 = m)
__global__ void __launch_bounds__(256) lu_update_kernel(double* __restrict__ h, int64_t ldh, double* __restrict__ g,
                                                        int64_t ldg, int64_t m, int64_t nrhs, int64_t k0, int w,
                                                        int64_t k1, int64_t lo, int64_t hi) {
  __shared__ double a[kLuPanel][33];
  __shared__ double b[kLuPanel][33];
  const int64_t cols = (m - k1) + nrhs;
  const int64_t r0 = lo + (int64_t)blockIdx.x * 32, c0 = (int64_t)blockIdx.y * 32;
  const int t = threadIdx.x;
  for (int e = t; e < kLuPanel * 32; e += blockDim.x) {
    const int i = e & 31, q = e >> 5;
    a[q][i] = q < w && r0 + i < hi ? h[(r0 + i) + ldh * (k0 + q)] : 0.0;
  }
  for (int e = t; e < kLuPanel * 32; e += blockDim.x) {
    const int q = e % kLuPanel, i = e / kLuPanel;
    b[q][i] = q < w && c0 + i < cols ? lu_column(h, ldh, g, ldg, m, k1, c0 + i)[k0 + q] : 0.0;
  }
  __syncthreads();
  const int i = t & 31;
  if (r0 + i >= hi) return;
#pragma unroll
  for (int cc = 0; cc < 4; ++cc) {
    const int j = (t >> 5) + 8 * cc;
    if (c0 + j >= cols) continue;
    double* x = lu_column(h, ldh, g, ldg, m, k1, c0 + j) + r0 + i;
    double v = *x;
#pragma unroll
    for (int q = 0; q < kLuPanel; ++q) v = fma(-a[q][i], b[q][j], v);
    *x = v;
  }
}

// rows [k0, k0 + w) of every right-hand side: U_kk x = g, one thread per column
__global__ void lu_back_kernel(const double* __restrict__ h, int64_t ldh, double* __restrict__ g, int64_t ldg,
                               int64_t nrhs, int64_t k0, int w) {
  __shared__ double u[kLuPanel][kLuPanel];
  __shared__ double rd[kLuPanel];
  for (int e = threadIdx.x; e < w * w; e += blockDim.x) u[e % w][e / w] = h[(k0 + e % w) + ldh * (k0 + e / w)];
  __syncthreads();
  if (threadIdx.x < w) rd[threadIdx.x] = 1.0 / u[threadIdx.x][threadIdx.x];
  __syncthreads();
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= nrhs) return;
  double* x = g + ldg * c + k0;
  double v[kLuPanel];
#pragma unroll
  for (int j = 0; j < kLuPanel; ++j) v[j] = j < w ? x[j] : 0.0;
#pragma unroll
  for (int j = kLuPanel - 1; j >= 0; --j)
    if (j < w) {
      v[j] = isfinite(rd[j]) ? v[j] * rd[j] : v[j] / u[j][j];
#pragma unroll
      for (int q = 0; q < j; ++q) v[q] = fma(-u[q][j], v[j], v[q]);
    }
#pragma unroll
  for (int j = 0; j < kLuPanel; ++j)
    if (j < w) x[j] = v[j];
}

__global__ void axpby_kernel(double alpha, const double* __restrict__ x, double beta,
                             double* __restrict__ y, int64_t n) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x)
    y[t] = alpha * x[t] + (beta == 0.0 ? 0.0 : beta * y[t]);
}

__global__ void count_nonfinite_kernel(const double* __restrict__ x, int64_t n, int* counter) {
  int local = 0;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x)
    local += isfinite(x[t]) ? 0 : 1;
  if (local) atomicAdd(counter, local);
}

}  // namespace

void launch_unpack_cderi(const double* tp, int64_t nao, int64_t naux, double* dense, cudaStream_t s) {
  const int64_t nt = div_up(nao, 32);
  unpack_cderi_kernel<<<dim3((unsigned)(nt * (nt + 1) / 2), (unsigned)std::min<int64_t>(naux, 65535)), dim3(32, 8), 0, s>>>(
      tp, nao, naux, dense);
  count_launch();
}

void launch_dimless(const double* y, const double* x, int64_t ldx, const double* e, int64_t nmo,
                    int64_t nocc, int64_t nb, double shift, double* out, int64_t ldo, cudaStream_t s) {
  dimless_kernel<double><<<grid_for(nmo * nocc * nb), kThreads, 0, s>>>(y, x, ldx, e, nmo, nocc, nb, shift, out, ldo);
  count_launch();
}

void launch_dimless_f32(const float* y, const double* x, int64_t ldx, const double* e, int64_t nmo,
                        int64_t nocc, int64_t nb, double shift, double* out, int64_t ldo,
                        cudaStream_t s) {
  dimless_kernel<float><<<grid_for(nmo * nocc * nb), kThreads, 0, s>>>(y, x, ldx, e, nmo, nocc, nb, shift, out, ldo);
  count_launch();
}

template <typename T>
void launch_xc_rho(const T* aobra, int64_t ld_aobra, const T* ket, int64_t npts,
                   int64_t nocc, int64_t nb, T* rho, int64_t ld_rho, cudaStream_t s) {
  xc_rho_kernel<T><<<grid_for(npts * nb), kThreads, 0, s>>>(aobra, ld_aobra, ket, npts, nocc, nb, rho, ld_rho);
  count_launch();
}
template void launch_xc_rho<double>(const double*, int64_t, const double*, int64_t, int64_t, int64_t, double*, int64_t, cudaStream_t);
template void launch_xc_rho<float>(const float*, int64_t, const float*, int64_t, int64_t, int64_t, float*, int64_t, cudaStream_t);

template <typename T>
void launch_xc_q(const T* aobra, int64_t ld_aobra, const double* w, const double* fxc,
                 int64_t fxc_ld, int nspin, int sout, const T* rho, int64_t ld_rho,
                 int64_t ld_rho_spin, int64_t npts, int64_t nocc, int64_t nb, T* q,
                 cudaStream_t s) {
  xc_q_kernel<T><<<grid_for(npts * nb), kThreads, 0, s>>>(aobra, ld_aobra, w, fxc, fxc_ld, nspin, sout, rho, ld_rho,
                                                         ld_rho_spin, npts, nocc, nb, q);
  count_launch();
}
template void launch_xc_q<double>(const double*, int64_t, const double*, const double*, int64_t, int, int, const double*, int64_t, int64_t, int64_t, int64_t, int64_t, double*, cudaStream_t);
template void launch_xc_q<float>(const float*, int64_t, const double*, const double*, int64_t, int, int, const float*, int64_t, int64_t, int64_t, int64_t, int64_t, float*, cudaStream_t);

__global__ void to_f32_kernel(const double* __restrict__ src, int64_t n, float* __restrict__ dst) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x)
    dst[t] = (float)src[t];
}

void launch_to_f32(const double* src, int64_t n, float* dst, cudaStream_t s) {
  if (n <= 0) return;
  to_f32_kernel<<<grid_for(n), kThreads, 0, s>>>(src, n, dst);
  count_launch();
}

int64_t residual_partials_size(int64_t n, int64_t nb) {
  return std::max<int64_t>(1, div_up(n, kResRowsPerBlock)) * nb;
}

void launch_residual_norms(const double* b, const double* x, const double* ax, double* r, int64_t n,
                           int64_t nb, double* norms2, double* partials, cudaStream_t s) {
  if (nb <= 0) return;
  const int64_t nblk = std::max<int64_t>(1, div_up(n, kResRowsPerBlock));
  dim3 grid((unsigned)nblk, (unsigned)nb);
  residual_kernel<<<grid, kThreads, 0, s>>>(b, x, ax, r, n, partials);
  sum_partials_kernel<<<(unsigned)div_up(nb, 128), 128, 0, s>>>(partials, nblk, nb, norms2);
  count_launch(2);
}

// partial dot products, the coefficients and the barrier's counter
int64_t mgs_partials_size(int64_t n, int64_t m) {
  const int64_t mm = std::max<int64_t>(m, 1);
  return kMgsPanel * mm * (std::max<int64_t>(1, std::min<int64_t>(kMgsMaxBlocks, div_up(n, 32))) + 1) + 4;
}

void launch_mgs(double* V, int64_t n, int64_t m, double lindep, double* ip, int* keep, double* partials, int num_sms,
                cudaStream_t s) {
  if (m <= 0) return;
  int64_t nblk = mgs_blocks(n, m, num_sms);
  MgsArgs a;
  a.V = V;
  a.n = n;
  a.m = m;
  a.rows = std::max<int64_t>(1, div_up(n, nblk));  // (n = 0, no occupied orbital: one block without rows)
  nblk = std::max<int64_t>(1, div_up(n, a.rows));
  a.stage = std::min(a.rows, kMgsStage);
  a.lindep = lindep;
  a.ip = ip;
  a.keep = keep;
  a.partials = partials;
  a.coef = partials + kMgsPanel * m * nblk;
  a.bar = reinterpret_cast<unsigned*>(a.coef + kMgsPanel * m + 1);
  const size_t smem = (size_t)kMgsPanel * (2 * a.stage + std::min(m, kMgsCoefs)) * 8;
  static PerDevice limit;
  allow_smem(limit, (const void*)mgs_kernel, kMgsPanel * (int)(2 * kMgsStage + kMgsCoefs) * 8);
  CPHF_CUDA(cudaMemsetAsync(a.bar, 0, sizeof(unsigned), s));
  void* args[] = {&a};
  CPHF_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(mgs_kernel), dim3((unsigned)nblk),
                                        dim3(kMgsThreads), args, smem, s));
  count_launch();
}

void launch_gather_cols(const double* src, int64_t n, const int* idx, int64_t cnt, double* dst,
                        int64_t ld_dst, cudaStream_t s) {
  if (cnt <= 0) return;
  gather_cols_kernel<<<grid_for(n * cnt), kThreads, 0, s>>>(src, n, idx, cnt, dst, ld_dst);
  count_launch();
}

void launch_scale_rows(double* coeff, int64_t ldc, const double* ip, int64_t m, int64_t nb, cudaStream_t s) {
  if (m <= 0 || nb <= 0) return;
  scale_rows_kernel<<<grid_for(m * nb), kThreads, 0, s>>>(coeff, ldc, ip, m, nb);
  count_launch();
}

void launch_add_diag(double* h, int64_t ldh, const double* ip, int64_t m, cudaStream_t s) {
  if (m <= 0) return;
  add_diag_kernel<<<(unsigned)div_up(m, kThreads), kThreads, 0, s>>>(h, ldh, ip, m);
  count_launch();
}

int64_t lu_scratch_ints() { return 1 + (int64_t)(sizeof(LuMoves) / sizeof(int)); }

void launch_lu_solve(double* h, int64_t ldh, double* g, int64_t ldg, int64_t m, int64_t nrhs, int* info,
                     cudaStream_t s) {
  LuMoves* moves = reinterpret_cast<LuMoves*>(info + 1);
  CPHF_CUDA(cudaMemsetAsync(info, 0, sizeof(int), s));
  constexpr int kMaxSmem = 200 * 1024;
  static PerDevice limit;
  allow_smem(limit, (const void*)lu_panel_kernel, kMaxSmem);
  for (int64_t k0 = 0; k0 < m; k0 += kLuPanel) {
    const int w = (int)std::min<int64_t>(kLuPanel, m - k0);
    const int64_t bytes = (m - k0) * w * 8, k1 = k0 + w, cols = (m - k1) + nrhs;
    const int smem = bytes <= kMaxSmem;
    lu_panel_kernel<<<1, kLuThreads, smem ? (size_t)bytes : 0, s>>>(h, ldh, m, k0, w, smem, moves, info);
    count_launch();
    if (cols > 0) {
      lu_rows_kernel<<<(unsigned)div_up(cols, 64), 64, 0, s>>>(h, ldh, g, ldg, m, nrhs, k0, w, moves);
      count_launch();
    }
    if (k1 < m) {
      lu_update_kernel<<<dim3((unsigned)div_up(m - k1, 32), (unsigned)div_up(cols, 32)), 256, 0, s>>>(
          h, ldh, g, ldg, m, nrhs, k0, w, k1, k1, m);
      count_launch();
    }
  }
  if (nrhs <= 0) return;
  for (int64_t k0 = (m - 1) / kLuPanel * kLuPanel; k0 >= 0 && m > 0; k0 -= kLuPanel) {
    const int w = (int)std::min<int64_t>(kLuPanel, m - k0);
    lu_back_kernel<<<(unsigned)div_up(nrhs, 64), 64, 0, s>>>(h, ldh, g, ldg, nrhs, k0, w);
    count_launch();
    if (k0 > 0) {
      lu_update_kernel<<<dim3((unsigned)div_up(k0, 32), (unsigned)div_up(nrhs, 32)), 256, 0, s>>>(h, ldh, g, ldg, m, nrhs,
                                                                                                k0, w, m, 0, k0);
      count_launch();
    }
  }
}

void launch_axpby(double alpha, const double* x, double beta, double* y, int64_t n, cudaStream_t s) {
  if (n <= 0) return;
  axpby_kernel<<<grid_for(n), kThreads, 0, s>>>(alpha, x, beta, y, n);
  count_launch();
}

namespace {
__global__ void nonzero_flags_kernel(const double* __restrict__ ao, int64_t ngrids, int64_t nao,
                                     const int64_t* __restrict__ off, int64_t nbatch, int* flags) {
  // one block per (batch, column)
  const int64_t b = blockIdx.x % nbatch, m = blockIdx.x / nbatch;
  const int64_t g0 = off[b], g1 = off[b + 1];
  int any = 0;
  for (int64_t g = g0 + threadIdx.x; g < g1; g += blockDim.x) any |= (ao[g + ngrids * m] != 0.0);
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) flags[b * nao + m] = any;
}

__global__ void finalize_kernel(const double* __restrict__ f1, const double* __restrict__ s1,
                                const double* __restrict__ resp, const double* __restrict__ e,
                                int64_t nmo, int64_t nocc, int64_t nprop, double* __restrict__ mo1,
                                double* __restrict__ mo_e1) {
  const int64_t per = nmo * nocc;
  const int64_t total = per * nprop;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t a = t / per, r = t - a * per;
    const int64_t p = r % nmo, i = r / nmo;
    const double b1 = f1[t] - s1[t] * e[i] + resp[t];
    if (p >= nocc) {
      mo1[t] = -b1 / (e[p] - e[i]);
    } else {
      mo_e1[p + nocc * (i + nocc * a)] = b1 + mo1[t] * (e[p] - e[i]);
    }
  }
}

// compute_dimless_cphf_rhs element-wise part (src/hessian/rscf.rs:174-178):
//   rhs[vir] = -(f1mo - s1mo e_i)[vir] / (e_a - e_i + shift),  rhs[occ] = -0.5 s1mo[occ]
__global__ void cphf_rhs_kernel(const double* __restrict__ f1, const double* __restrict__ s1,
                                const double* __restrict__ e, int64_t nmo, int64_t nocc, int64_t nprop, double shift,
                                double* __restrict__ rhs) {
  const int64_t per = nmo * nocc;
  const int64_t total = per * nprop;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = t % per;
    const int64_t p = r % nmo, i = r / nmo;
    rhs[t] = p >= nocc ? -(f1[t] - s1[t] * e[i]) / (e[p] - e[i] + shift) : -0.5 * s1[t];
  }
}

__global__ void hess_pairs_kernel(const double* __restrict__ f1, const double* __restrict__ s1,
                                  const double* __restrict__ mo1, const double* __restrict__ mo_e1,
                                  const double* __restrict__ e, int64_t nmo, int64_t nocc, int64_t nprop,
                                  double f0, double fs, double fe, double* __restrict__ G) {
  __shared__ double sh[32];
  const int64_t r = blockIdx.x % nprop, q = blockIdx.x / nprop;
  const int64_t per = nmo * nocc;
  const double* m1 = mo1 + per * r;
  const double* ff = f1 + per * q;
  const double* ss = s1 + per * q;
  const double* me = mo_e1 + nocc * nocc * r;
  double acc = 0.0;
  for (int64_t t = threadIdx.x; t < per; t += blockDim.x) {
    const int64_t p = t % nmo, i = t / nmo;
    acc += f0 * m1[t] * ff[t] - fs * m1[t] * ss[t] * e[i];
    if (p < nocc) acc -= fe * me[p + nocc * i] * ss[t];
  }
  const double s = block_sum(acc, sh);
  if (threadIdx.x == 0) G[r + nprop * q] += s;
}

__global__ void hess_assemble_kernel(const double* __restrict__ G, int64_t natm, double* __restrict__ de) {
  const int64_t np = 3 * natm;
  const int64_t total = 9 * natm * natm;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t x = t % 3, y = (t / 3) % 3, b = (t / 9) % natm, a = t / (9 * natm);
    de[t] = b <= a ? G[(x + 3 * b) + np * (y + 3 * a)] : G[(y + 3 * a) + np * (x + 3 * b)];
  }
}
}  // namespace

void launch_nonzero_flags(const double* ao, int64_t ngrids, int64_t nao, const int64_t* offsets,
                          int64_t nbatch, int* flags, cudaStream_t s) {
  if (nbatch <= 0 || nao <= 0) return;
  const int64_t blocks = nbatch * nao;
  for (int64_t b0 = 0; b0 < blocks; b0 += (int64_t)1 << 30) {
    // one launch suffices for every realistic size (grid.x < 2^31)
    nonzero_flags_kernel<<<(unsigned)blocks, kThreads, 0, s>>>(ao, ngrids, nao, offsets, nbatch, flags);
    count_launch();
    break;
  }
}

void launch_finalize(const double* f1, const double* s1, const double* resp, const double* e, int64_t nmo,
                     int64_t nocc, int64_t nprop, double* mo1, double* mo_e1, cudaStream_t s) {
  if (nmo * nocc * nprop <= 0) return;
  finalize_kernel<<<grid_for(nmo * nocc * nprop), kThreads, 0, s>>>(f1, s1, resp, e, nmo, nocc, nprop, mo1, mo_e1);
  count_launch();
}

void launch_cphf_rhs(const double* f1, const double* s1, const double* e, int64_t nmo, int64_t nocc, int64_t nprop,
                     double shift, double* rhs, cudaStream_t s) {
  if (nmo * nocc * nprop <= 0) return;
  cphf_rhs_kernel<<<grid_for(nmo * nocc * nprop), kThreads, 0, s>>>(f1, s1, e, nmo, nocc, nprop, shift, rhs);
  count_launch();
}

void launch_hess_pairs(const double* f1, const double* s1, const double* mo1, const double* mo_e1,
                       const double* e, int64_t nmo, int64_t nocc, int64_t nprop, double f0, double fs,
                       double fe, double* G, cudaStream_t s) {
  if (nprop <= 0) return;
  hess_pairs_kernel<<<(unsigned)(nprop * nprop), kThreads, 0, s>>>(f1, s1, mo1, mo_e1, e, nmo, nocc, nprop, f0,
                                                                   fs, fe, G);
  count_launch();
}

void launch_hess_assemble(const double* G, int64_t natm, double* de, cudaStream_t s) {
  if (natm <= 0) return;
  hess_assemble_kernel<<<grid_for(9 * natm * natm), kThreads, 0, s>>>(G, natm, de);
  count_launch();
}

void launch_count_nonfinite(const double* x, int64_t n, int* counter, cudaStream_t s) {
  if (n <= 0) return;
  count_nonfinite_kernel<<<grid_for(n, 2048), kThreads, 0, s>>>(x, n, counter);
  count_launch();
}

}  // namespace cphf
