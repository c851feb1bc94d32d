// Adjoint of the exact-GP marginal log-likelihood.
//
//   d mll / d theta = 1/2 tr((alpha alpha^T - Sigma^-1) dSigma/dtheta),
//   alpha = Sigma^-1 (y - m).
//
// The reference obtains this by JAX reverse-mode through slogdet and solve
// (gpjax/objectives.py:100-107 -> distributions.py:132-134 ->
// linalg/operations.py:111,164) and the vmap'd pointwise kernel
// (computations/dense.py:35).  Here Sigma^-1 = V V^T with V = L^-T is formed
// tile by tile (the LAUUM product) and never stored: each lower tile of
// Sigma^-1 is reduced at once against dK/dtheta, whose entries are
// regenerated in registers from the scaled inputs.  (Large float64 problems
// form Sigma^-1 with the split GEMM of xgemm.cuh first, and the kernel is the
// reduction alone.)  Per-tile partial sums
// go to a workspace array that a single block reduces in a fixed order, so
// the gradient is deterministic.
#include "simt_tile.cuh"
#include "xgemm.cuh"

namespace gpk {

// Number of float64 partial sums written per tile: d lengthscale terms,
// the variance term and the noise term.
__host__ __device__ inline int grad_slots(int d) { return d + 2; }

// FROM_W: V holds W = Sigma^-1 itself (lower tiles), formed beforehand on the
// tensor cores; the kernel is then the reduction alone.
template <typename T, int DMAX, typename Cfg = GemmCfg<T>, bool FROM_W = false>
__global__ void __launch_bounds__((Cfg::BM / Cfg::TM) * (Cfg::BN / Cfg::TN))
    lauum_grad_kernel(int kind, const T* __restrict__ V, int64_t ldv, int n, int d,
                      const T* __restrict__ xs, const double* __restrict__ alpha,
                      double* __restrict__ gpart, const double* __restrict__ kaptr) {
  constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK;
  constexpr int TM = Cfg::TM, TN = Cfg::TN;
  constexpr int NTX = BN / TN, NTY = BM / TM, NT = NTX * NTY;
  constexpr int WLD = BN + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // main-loop staging and the W tile share the front of shared memory
  SimtSmem<T, Cfg>& sm = *reinterpret_cast<SimtSmem<T, Cfg>*>(smem_raw);
  T* Ws = reinterpret_cast<T*>(smem_raw);
  constexpr size_t front = sizeof(SimtSmem<T, Cfg>) > sizeof(T) * BM * WLD
                               ? sizeof(SimtSmem<T, Cfg>)
                               : sizeof(T) * BM * WLD;
  T* sxi = reinterpret_cast<T*>(smem_raw + ((front + 15) & ~size_t(15)));
  T* sxj = sxi + BM * DMAX;
  T* sai = sxj + BN * DMAX;
  T* saj = sai + BM;
  double* rbuf = reinterpret_cast<double*>(
      (reinterpret_cast<uintptr_t>(saj + BN) + 15) & ~static_cast<uintptr_t>(15));

  const int t = blockIdx.x;
  int I, J;
  tri_index(t, I, J);
  const int i0 = I * BM, j0 = J * BN;
  if constexpr (FROM_W) {
    for (int e = threadIdx.x; e < BM * BN; e += NT) {
      const int r = e / BN, c = e % BN;
      Ws[r * WLD + c] = i0 + r < n && j0 + c <= i0 + r ? V[(int64_t)(i0 + r) * ldv + j0 + c] : T(0);
    }
  } else {
    int klo, khi;
    tile_krange<BM, BN, BK>(n, TRI_UPPER, TRI_UPPER, i0, j0, klo, khi);
    T acc[TM][TN];
#pragma unroll
    for (int a = 0; a < TM; ++a)
#pragma unroll
      for (int b = 0; b < TN; ++b) acc[a][b] = T(0);
    simt_tile_mma<T, Cfg>(V, ldv, n, TRI_UPPER, V, ldv, n, TRI_UPPER, i0, j0, klo, khi, sm, acc);
    // (simt_tile_mma ends with a barrier, so the staging area can be reused)
    const int tx = threadIdx.x % NTX, ty = threadIdx.x / NTX;
#pragma unroll
    for (int a = 0; a < TM; ++a)
#pragma unroll
      for (int b = 0; b < TN; ++b) Ws[(ty + a * NTY) * WLD + tx + b * NTX] = acc[a][b];
  }
  for (int e = threadIdx.x; e < BM * DMAX; e += NT) {
    int r = e / DMAX, k = e % DMAX;
    sxi[e] = (i0 + r < n && k < d) ? xs[(int64_t)(i0 + r) * d + k] : T(0);
  }
  for (int e = threadIdx.x; e < BN * DMAX; e += NT) {
    int r = e / DMAX, k = e % DMAX;
    sxj[e] = (j0 + r < n && k < d) ? xs[(int64_t)(j0 + r) * d + k] : T(0);
  }
  for (int e = threadIdx.x; e < BM; e += NT) sai[e] = (i0 + e < n) ? (T)alpha[i0 + e] : T(0);
  for (int e = threadIdx.x; e < BN; e += NT) saj[e] = (j0 + e < n) ? (T)alpha[j0 + e] : T(0);
  __syncthreads();

  const T ka = kaptr ? (T)*kaptr : T(1);  // kernel shape parameter (rational quadratic)
  // float64 accumulators: the terms cancel heavily (the variance and noise
  // sums are differences of O(n) quantities), so per-thread sums stay exact
  // to float64 while each term is formed in T
  double gl[DMAX];
#pragma unroll
  for (int k = 0; k < DMAX; ++k) gl[k] = 0.0;
  double gvar = 0.0, gnoise = 0.0;
  // consecutive threads take consecutive columns of one row
#pragma unroll 1
  for (int e = threadIdx.x; e < BM * BN; e += NT) {
    const int r = e / BN, c = e % BN;
    const int gi = i0 + r, gj = j0 + c;
    if (gi >= n || gj >= n || gj > gi) continue;
    const T w = Ws[r * WLD + c];
    const T ai = sai[r];
    const T f = (gi == gj) ? T(1) : T(2);
    const T coef = f * (ai * saj[c] - w);
    T dsq[DMAX];
    T sq = T(0);
#pragma unroll
    for (int k = 0; k < DMAX; ++k) {
      if (sizeof(T) == 8 && k >= d) continue;  // uniform: padding costs no float64 work
      const T df = sxi[r * DMAX + k] - sxj[c * DMAX + k];
      dsq[k] = df * df;
      sq += dsq[k];
    }
    T k1, c1;
    kval_dcoef<T>(kind, sq, T(1), k1, c1, ka);
    gvar += (double)(coef * k1);
    const T cc = coef * c1;
#pragma unroll
    for (int k = 0; k < DMAX; ++k)
      if (sizeof(T) == 4 || k < d) gl[k] += (double)(cc * dsq[k]);
    if (gi == gj) gnoise += (double)ai * (double)ai - (double)w;
  }
  // block reduction in float64, fixed order
  const int slots = grad_slots(d);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NW = NT / 32;
#pragma unroll
  for (int k = 0; k < DMAX; ++k) {
    if (k < d) {
      const double dv = warp_sum(gl[k]);
      if (lane == 0) rbuf[k * NW + warp] = dv;
    }
  }
  {
    const double dv = warp_sum(gvar);
    if (lane == 0) rbuf[d * NW + warp] = dv;
    const double dn = warp_sum(gnoise);
    if (lane == 0) rbuf[(d + 1) * NW + warp] = dn;
  }
  __syncthreads();
  for (int s = threadIdx.x; s < slots; s += NT) {
    double tot = 0.0;
    for (int w = 0; w < NW; ++w) tot += rbuf[s * NW + w];
    gpart[(int64_t)t * slots + s] = tot;
  }
}

template <typename T, int DMAX, typename Cfg, bool FROM_W>
static cudaError_t launch_lauum_grad(int kind, const T* V, int64_t ldv, int n, int d, const T* xs,
                                     const double* alpha, double* gpart, const double* kaptr,
                                     cudaStream_t s) {
  constexpr int BM = Cfg::BM, BN = Cfg::BN;
  constexpr int NT = (Cfg::BM / Cfg::TM) * (Cfg::BN / Cfg::TN);
  const int tiles_m = (n + BM - 1) / BM;
  const int tiles = tiles_m * (tiles_m + 1) / 2;
  const size_t front = sizeof(SimtSmem<T, Cfg>) > sizeof(T) * BM * (BN + 1)
                           ? sizeof(SimtSmem<T, Cfg>)
                           : sizeof(T) * BM * (BN + 1);
  const size_t smem = ((front + 15) & ~size_t(15)) + (size_t)(BM + BN) * DMAX * sizeof(T) +
                      (size_t)(BM + BN) * sizeof(T) + 16 +
                      (size_t)(GPK_MAX_D + 2) * (NT / 32) * sizeof(double);
  cudaFuncSetAttribute(lauum_grad_kernel<T, DMAX, Cfg, FROM_W>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  lauum_grad_kernel<T, DMAX, Cfg, FROM_W><<<tiles, NT, smem, s>>>(kind, V, ldv, n, d, xs, alpha,
                                                                  gpart, kaptr);
  return launch_status();
}

// Tile edge of the float64 form: 16 while those tiles fit about two waves of
// the chip (n <= 384), 32 up to n = 1536, 64 above (each block's float64 work
// runs at 1.7 operations per clock, so too few blocks is what a small n pays
// for).  Whole evaluation with edges 16 / 32 / 64: n = 100 270 / 273 / 375 us,
// 384 869 / 871 / 895, 1024 2018 / 1998 / 1997, 2048 4043 / 3957 / 3947.
template <typename T>
static int lauum_edge(int n) {
  if (sizeof(T) == 4) return GemmCfg<float>::BM;
  return n <= 384 ? 16 : n <= 1536 ? 32 : 64;
}

template <typename T>
int lauum_grad_tiles(int n) {
  const int e = lauum_edge<T>(n), tm = (n + e - 1) / e;
  return tm * (tm + 1) / 2;
}
template int lauum_grad_tiles<double>(int);
template int lauum_grad_tiles<float>(int);

template <typename T, bool FROM_W>
static cudaError_t lauum_dispatch(int kind, const T* V, int64_t ldv, int n, int d, const T* xs,
                                  const double* theta, int n_ls, const double* alpha,
                                  double* gpart, cudaStream_t s) {
  const double* ka = kind == GPK_RATIONAL_QUADRATIC ? theta + n_ls + 3 : nullptr;
  auto by_tile = [&](auto dmax) {
    constexpr int D = decltype(dmax)::value;
    if constexpr (sizeof(T) == 8) {
      const int e = lauum_edge<T>(n);
      if (e == 16)
        return launch_lauum_grad<T, D, GemmCfgTiny<T>, FROM_W>(kind, V, ldv, n, d, xs, alpha,
                                                               gpart, ka, s);
      if (e == 32)
        return launch_lauum_grad<T, D, GemmCfgSmall<T>, FROM_W>(kind, V, ldv, n, d, xs, alpha,
                                                                gpart, ka, s);
    }
    return launch_lauum_grad<T, D, GemmCfg<T>, FROM_W>(kind, V, ldv, n, d, xs, alpha, gpart, ka,
                                                       s);
  };
  if (sizeof(T) == 8 && d <= 4) return by_tile(std::integral_constant<int, sizeof(T) == 8 ? 4 : 8>{});
  if (d <= 8) return by_tile(std::integral_constant<int, 8>{});
  if (d <= 16) return by_tile(std::integral_constant<int, 16>{});
  if (d <= 32) return by_tile(std::integral_constant<int, 32>{});
  return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t lauum_grad(int kind, const T* V, int64_t ldv, int n, int d, const T* xs,
                       const double* theta, int n_ls, const double* alpha, double* gpart,
                       cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  return lauum_dispatch<T, false>(kind, V, ldv, n, d, xs, theta, n_ls, alpha, gpart, s);
}

cudaError_t lauum_grad_x(int kind, const double* V, int64_t ldv, int n, int d, const double* xs,
                         const double* theta, int n_ls, const double* alpha, double* gpart,
                         double* W, int64_t ldw, const XRoom& x, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  GemmProb<double> p{};
  p.A = p.B = V;
  p.lda = p.ldb = ldv;
  p.a_tri = p.b_tri = TRI_UPPER;
  p.C = W;
  p.ldc = ldw;
  p.M = p.N = p.K = n;
  p.c_lower = 1;
  p.alpha = 1.0;
  cudaError_t e = gemm_nt_x(p, 1, x, s);
  if (e != cudaSuccess) return e;
  return lauum_dispatch<double, true>(kind, W, ldw, n, d, xs, theta, n_ls, alpha, gpart, s);
}

// ---------------------------------------------------------------------------
// Residual r = diff - (K + diag_add I) alpha with K regenerated from the
// scaled inputs in T; per-chunk partial sums (RES_CHUNK columns) in T are
// accumulated in float64.  Column chunks are spread over gridDim.y and their
// partials written to rpart[y][n]; residual_finish sums them in fixed order.
// ---------------------------------------------------------------------------
constexpr int RES_ROWS = 128;
constexpr int RES_COLS = 128;
constexpr int RES_SPLIT = 16;

template <typename T, int DMAX>
__global__ void __launch_bounds__(RES_ROWS)
    residual_kernel(int kind, int n, int d, const T* __restrict__ xs,
                    const double* __restrict__ theta, int n_ls, const double* __restrict__ alpha,
                    double* __restrict__ rpart) {
  __shared__ T sx[RES_COLS][DMAX + 1];
  __shared__ T sa[RES_COLS];
  const int i = blockIdx.x * RES_ROWS + threadIdx.x;
  const T s2 = (T)theta[n_ls];
  T xi[DMAX];
#pragma unroll
  for (int k = 0; k < DMAX; ++k) xi[k] = (i < n && k < d) ? xs[(int64_t)i * d + k] : T(0);
  const int per = (n + RES_SPLIT - 1) / RES_SPLIT;
  const int cbeg = blockIdx.y * per, cend = min(n, cbeg + per);
  double accd = 0.0;
  for (int c0 = cbeg; c0 < cend; c0 += RES_COLS) {
    __syncthreads();
    for (int e = threadIdx.x; e < RES_COLS * d; e += RES_ROWS) {
      int r = e / d, k = e % d;
      sx[r][k] = (c0 + r < cend) ? xs[(int64_t)(c0 + r) * d + k] : T(0);
    }
    for (int e = threadIdx.x; e < RES_COLS; e += RES_ROWS)
      sa[e] = (c0 + e < cend) ? (T)alpha[c0 + e] : T(0);
    __syncthreads();
    const int cnt = min(RES_COLS, cend - c0);
    T part = T(0);
    for (int c = 0; c < cnt; ++c) {
      T sq = T(0);
#pragma unroll
      for (int k = 0; k < DMAX; ++k) {
        if (k < d) {
          T df = xi[k] - sx[c][k];
          sq = fma(df, df, sq);
        }
      }
      part = fma(kval<T>(kind, sq, s2, kshape<T>(kind, theta, n_ls)), sa[c], part);
    }
    accd += (double)part;
  }
  if (i < n) rpart[(int64_t)blockIdx.y * n + i] = accd;
}

__global__ void residual_finish_kernel(int n, const double* __restrict__ theta, int n_ls,
                                       double jitter, const double* __restrict__ diff,
                                       const double* __restrict__ alpha,
                                       const double* __restrict__ rpart, double* __restrict__ r) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double sd = theta[n_ls + 1];
  double s = 0.0;
  for (int y = 0; y < RES_SPLIT; ++y) s += rpart[(int64_t)y * n + i];
  s += (jitter + sd * sd) * alpha[i];
  r[i] = diff[i] - s;
}

size_t residual_scratch_doubles(int n) { return (size_t)RES_SPLIT * n; }

template <typename T>
cudaError_t residual(int kind, int n, int d, const T* xs, const double* theta, int n_ls,
                     double jitter, const double* diff, const double* alpha, double* r,
                     double* rpart, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  dim3 grid((unsigned)cdiv(n, RES_ROWS), RES_SPLIT);
  if (d <= 8)
    residual_kernel<T, 8><<<grid, RES_ROWS, 0, s>>>(kind, n, d, xs, theta, n_ls, alpha, rpart);
  else if (d <= 16)
    residual_kernel<T, 16><<<grid, RES_ROWS, 0, s>>>(kind, n, d, xs, theta, n_ls, alpha, rpart);
  else if (d <= 32)
    residual_kernel<T, 32><<<grid, RES_ROWS, 0, s>>>(kind, n, d, xs, theta, n_ls, alpha, rpart);
  else
    return cudaErrorInvalidValue;
  cudaError_t e = launch_status();
  if (e != cudaSuccess) return e;
  residual_finish_kernel<<<(int)cdiv(n, 256), 256, 0, s>>>(n, theta, n_ls, jitter, diff, alpha,
                                                           rpart, r);
  return launch_status();
}

// The residual from stored kernel values: one 64 x 64 tile (I <= J) of the
// upper triangle per block, its row sums against alpha_J and column sums
// against alpha_I: two multiply-adds an element instead of a kernel
// evaluation.  part[t][i] receives what tile row/column t contributes to row i,
// summed in order by the finishing kernel.
constexpr int RS_T = 64;
__global__ void __launch_bounds__(256)
    residual_stored_kernel(int n, const double* __restrict__ A, int64_t lda,
                           const double* __restrict__ alpha, double* __restrict__ part) {
  __shared__ double tile[RS_T][RS_T + 1];
  __shared__ double ai[RS_T], aj[RS_T], red[2][4][RS_T];
  int I, J;
  tri_index(blockIdx.x, J, I);  // I <= J
  const int i0 = I * RS_T, j0 = J * RS_T;
  const int c = threadIdx.x & 63, q = threadIdx.x >> 6;
#pragma unroll
  for (int u = 0; u < RS_T / 4; ++u) {
    const int r = q + 4 * u, gi = i0 + r, gj = j0 + c;
    tile[r][c] = gi < n && gj < n && gj > gi ? A[(int64_t)gi * lda + gj] : 0.0;
  }
  if (q == 0) ai[c] = i0 + c < n ? alpha[i0 + c] : 0.0;
  if (q == 1) aj[c] = j0 + c < n ? alpha[j0 + c] : 0.0;
  __syncthreads();
  double cs = 0.0, rs = 0.0;
#pragma unroll
  for (int u = 0; u < RS_T / 4; ++u) {
    const int k = q * (RS_T / 4) + u;
    cs = fma(tile[k][c], ai[k], cs);  // column c, rows of this quarter
    rs = fma(tile[c][k], aj[k], rs);  // row c, columns of this quarter
  }
  red[0][q][c] = cs;
  red[1][q][c] = rs;
  __syncthreads();
  if (q >= 2) return;
  const double v = (red[q][0][c] + red[q][1][c]) + (red[q][2][c] + red[q][3][c]);
  if (I == J) {
    red[q][0][c] = v;  // own slots only
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (q == 0 && j0 + c < n) part[(int64_t)I * n + j0 + c] = v + red[1][0][c];
  } else if (q == 0) {
    if (j0 + c < n) part[(int64_t)I * n + j0 + c] = v;
  } else if (i0 + c < n) {
    part[(int64_t)J * n + i0 + c] = v;
  }
}

__global__ void residual_stored_finish(int kind, int n, int nt, const double* __restrict__ theta,
                                       int n_ls, double jitter, const double* __restrict__ diff,
                                       const double* __restrict__ alpha,
                                       const double* __restrict__ part, double* __restrict__ r) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double sd = theta[n_ls + 1];
  const double kd =
      (kval<double>(kind, 0.0, theta[n_ls], kshape<double>(kind, theta, n_ls)) + jitter) + sd * sd;
  double s0 = 0.0, s1 = 0.0;
  int t = 0;
#pragma unroll 4
  for (; t + 1 < nt; t += 2) {
    s0 += part[(int64_t)t * n + i];
    s1 += part[(int64_t)(t + 1) * n + i];
  }
  if (t < nt) s0 += part[(int64_t)t * n + i];
  r[i] = diff[i] - fma(kd, alpha[i], s0 + s1);
}

cudaError_t residual_stored(int kind, int n, const double* A, int64_t lda, const double* theta,
                            int n_ls, double jitter, const double* diff, const double* alpha,
                            double* r, double* part, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int nt = (n + RS_T - 1) / RS_T;
  residual_stored_kernel<<<nt * (nt + 1) / 2, 256, 0, s>>>(n, A, lda, alpha, part);
  cudaError_t e = launch_status();
  if (e != cudaSuccess) return e;
  residual_stored_finish<<<(int)cdiv(n, 64), 64, 0, s>>>(kind, n, nt, theta, n_ls, jitter, diff,
                                                         alpha, part, r);
  return launch_status();
}

template cudaError_t lauum_grad<double>(int, const double*, int64_t, int, int, const double*,
                                        const double*, int, const double*, double*, cudaStream_t);
template cudaError_t lauum_grad<float>(int, const float*, int64_t, int, int, const float*,
                                       const double*, int, const double*, double*, cudaStream_t);
template cudaError_t residual<float>(int, int, int, const float*, const double*, int, double,
                                     const double*, const double*, double*, double*, cudaStream_t);

}  // namespace gpk
