// Gram and cross-covariance tiles generated from the inputs.
//
// Reference: DenseKernelComputation._cross_covariance builds
// K[i, j] = k(x_i, y_j) with a vmap of a vmap over the pointwise kernel
// (gpjax/kernels/computations/dense.py:32-36); gram() is cross_covariance(x, x)
// (computations/base.py:56-72).  Each pointwise kernel divides both inputs by
// the lengthscale before taking the squared distance
// (kernels/stationary/rbf.py:41-43, matern32.py:46-47, matern52.py:45-46).
// Here the inputs are scaled once (xs = x / l, or once per tile), then each
// CTA stages a panel of each side in shared memory and every thread produces
// a column strip of the output tile.
#include "gpk_internal.cuh"
#include "simt_tile.cuh"

namespace gpk {

template <typename T>
__global__ void scale_inputs_kernel(const double* __restrict__ x, int64_t ldx, int n, int d,
                                    const double* __restrict__ theta, int n_ls, T* __restrict__ xs) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (int64_t)n * d) return;
  const int i = (int)(e / d), k = (int)(e % d);
  const double l = theta[n_ls == 1 ? 0 : k];
  xs[e] = (T)(x[(int64_t)i * ldx + k] / l);
}

template <typename T>
cudaError_t scale_inputs(const double* x, int64_t ldx, int n, int d, const double* theta, int n_ls,
                         T* xs, cudaStream_t s) {
  const int64_t total = (int64_t)n * d;
  if (total == 0) return cudaSuccess;
  scale_inputs_kernel<T><<<(int)cdiv(total, 256), 256, 0, s>>>(x, ldx, n, d, theta, n_ls, xs);
  return launch_status();
}

constexpr int GT = 64;  // output tile edge

// D bounds the input dimension (coordinates past d are zero and add nothing).
template <typename T, typename TO, int D, bool LIB = false>
__global__ void __launch_bounds__(256)
    cross_cov_kernel(int kind, int n, int m, int d, const T* __restrict__ xs,
                     const T* __restrict__ ys, const double* __restrict__ theta, int n_ls, int mode,
                     double jitter, TO* __restrict__ out, int64_t ldo) {
  __shared__ T sx[GT][D + 1];
  __shared__ T sy[GT][D + 1];
  const int i0 = blockIdx.y * GT, j0 = blockIdx.x * GT;
  const T s2 = (T)theta[n_ls];
  const double sd = theta[n_ls + 1];
  if (mode >= 1 && j0 > i0 + GT - 1) {
    // strictly-upper tile of the factorisation input: zeros
    for (int e = threadIdx.x; e < GT * GT; e += blockDim.x) {
      int r = e / GT, c = e % GT;
      if (i0 + r < n && j0 + c < m) out[(int64_t)(i0 + r) * ldo + j0 + c] = TO(0);
    }
    return;
  }
  for (int e = threadIdx.x; e < GT * D; e += blockDim.x) {
    int r = e / D, k = e % D;
    sx[r][k] = (i0 + r < n && k < d) ? xs[(int64_t)(i0 + r) * d + k] : T(0);
    sy[r][k] = (j0 + r < m && k < d) ? ys[(int64_t)(j0 + r) * d + k] : T(0);
  }
  __syncthreads();
  const int c = threadIdx.x % GT;
  const int rbase = threadIdx.x / GT;  // 0..3
  const int gj = j0 + c;
  if (gj >= m) return;
  T yv[D];
#pragma unroll
  for (int k = 0; k < D; ++k) yv[k] = sy[c][k];
  for (int r = rbase; r < GT; r += 4) {
    const int gi = i0 + r;
    if (gi >= n) break;
    TO v;
    if (mode >= 1 && gj > gi) {
      v = TO(0);
    } else {
      T sq = T(0);
#pragma unroll
      for (int k = 0; k < D; ++k) {
        if (k >= d) continue;  // uniform: padding coordinates cost no float64 work
        T df = sx[r][k] - yv[k];
        sq = fma(df, df, sq);
      }
      T kv;
      if constexpr (LIB)
        kv = kval_lib(kind, sq, s2, kshape<T>(kind, theta, n_ls));
      else
        kv = kval<T>(kind, sq, s2, kshape<T>(kind, theta, n_ls));
      if (mode == 1 && gi == gj) {
        // (K + I*jitter) + I*obs_stddev^2 (objectives.py:100-103)
        double dv = ((double)kv + jitter) + sd * sd;
        v = (TO)dv;
      } else if (mode == 2 && gi == gj) {
        v = (TO)((double)kv + jitter);  // K + I*jitter (objectives.py:353-354)
      } else {
        v = (TO)kv;
      }
    }
    out[(int64_t)gi * ldo + gj] = v;
  }
}

// Mode 3, float64: Sigma's lower triangle and the kernel values above it, one
// TE x TE tile (I >= J) per block, evaluated once and stored twice (the second
// time transposed through shared memory).  TE = 32 below n = 1536: with 64 the
// float64 work of a small matrix sits in too few blocks.
template <int D, int TE>
__global__ void __launch_bounds__(256)
    gram_sym_kernel(int kind, int n, int d, const double* __restrict__ xs,
                    const double* __restrict__ theta, int n_ls, double jitter,
                    double* __restrict__ out, int64_t ldo) {
  __shared__ double sx[TE][D + 1], sy[TE][D + 1];
  __shared__ double st[TE][TE + 1];
  int I, J;
  tri_index(blockIdx.x, I, J);
  const int i0 = I * TE, j0 = J * TE;
  const double s2 = theta[n_ls], sd = theta[n_ls + 1], ka = kshape<double>(kind, theta, n_ls);
  for (int e = threadIdx.x; e < TE * D; e += 256) {
    const int r = e / D, k = e % D;
    sx[r][k] = (i0 + r < n && k < d) ? xs[(int64_t)(i0 + r) * d + k] : 0.0;
    sy[r][k] = (j0 + r < n && k < d) ? xs[(int64_t)(j0 + r) * d + k] : 0.0;
  }
  __syncthreads();
  const int c = threadIdx.x % TE, gj = j0 + c;
  double yv[D];
#pragma unroll
  for (int k = 0; k < D; ++k) yv[k] = sy[c][k];
  for (int r = threadIdx.x / TE; r < TE; r += 256 / TE) {
    const int gi = i0 + r;
    if (gi >= n || gj > gi) continue;
    double sq = 0.0;
#pragma unroll
    for (int k = 0; k < D; ++k) {
      if (k >= d) continue;
      const double df = sx[r][k] - yv[k];
      sq = fma(df, df, sq);
    }
    const double kv = kval<double>(kind, sq, s2, ka);
    st[r][c] = kv;
    out[(int64_t)gi * ldo + gj] = gi == gj ? (kv + jitter) + sd * sd : kv;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < TE * TE; e += 256) {
    const int rr = e / TE, cc = e % TE;  // element (i0 + cc, j0 + rr) at (j0 + rr, i0 + cc)
    if (i0 + cc < n && j0 + rr < i0 + cc) out[(int64_t)(j0 + rr) * ldo + i0 + cc] = st[cc][rr];
  }
}

template <typename T, typename TO>
cudaError_t cross_cov_scaled(int kind, int n, int m, int d, const T* xs, const T* ys,
                             const double* theta, int n_ls, int mode, double jitter, TO* out,
                             int64_t ldo, cudaStream_t s) {
  if (n <= 0 || m <= 0) return cudaSuccess;
  if (d > GPK_MAX_D) return cudaErrorInvalidValue;
  if constexpr (sizeof(T) == 8) {
    if (mode == 3) {
      auto sym = [&](auto dim) {
        constexpr int D = decltype(dim)::value;
        constexpr int BIG = D <= 8 ? 64 : 32;  // 64 with D > 8 exceeds static shared memory
        const int te = n < 1536 ? 32 : BIG, nt = (n + te - 1) / te;
        auto* k = te == 32 ? gram_sym_kernel<D, 32> : gram_sym_kernel<D, BIG>;
        k<<<nt * (nt + 1) / 2, 256, 0, s>>>(kind, n, d, xs, theta, n_ls, jitter, out, ldo);
      };
      if (d <= 4)
        sym(std::integral_constant<int, 4>{});
      else if (d <= 8)
        sym(std::integral_constant<int, 8>{});
      else if (d <= 16)
        sym(std::integral_constant<int, 16>{});
      else
        sym(std::integral_constant<int, 32>{});
      return launch_status();
    }
  }
  dim3 grid((unsigned)cdiv(m, GT), (unsigned)cdiv(n, GT));
  auto run = [&](auto dim) {
    cross_cov_kernel<T, TO, decltype(dim)::value><<<grid, 256, 0, s>>>(
        kind, n, m, d, xs, ys, theta, n_ls, mode, jitter, out, ldo);
  };
  if (d <= 8)
    run(std::integral_constant<int, 8>{});
  else if (d <= 16)
    run(std::integral_constant<int, 16>{});
  else
    run(std::integral_constant<int, 32>{});
  return launch_status();
}

__global__ void sigma_diag_kernel(int kind, int n, const double* __restrict__ theta, int n_ls,
                                  double jitter, double* __restrict__ dtrack) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double sd = theta[n_ls + 1];
  dtrack[i] = (kval<double>(kind, 0.0, theta[n_ls], kshape<double>(kind, theta, n_ls)) + jitter) + sd * sd;
}

cudaError_t sigma_diag_init(int kind, int n, const double* theta, int n_ls, double jitter,
                            double* dtrack, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  sigma_diag_kernel<<<(int)cdiv(n, 256), 256, 0, s>>>(kind, n, theta, n_ls, jitter, dtrack);
  return launch_status();
}

template cudaError_t scale_inputs<double>(const double*, int64_t, int, int, const double*, int,
                                          double*, cudaStream_t);
template cudaError_t scale_inputs<float>(const double*, int64_t, int, int, const double*, int,
                                         float*, cudaStream_t);
cudaError_t cross_cov_lib(int kind, int n, int m, int d, const double* xs, const double* ys,
                          const double* theta, int n_ls, int mode, double jitter, double* out,
                          int64_t ldo, cudaStream_t s) {
  if (n <= 0 || m <= 0) return cudaSuccess;
  if (d > GPK_MAX_D) return cudaErrorInvalidValue;
  const dim3 grid((unsigned)cdiv(m, GT), (unsigned)cdiv(n, GT));
  auto run = [&](auto dim) {
    cross_cov_kernel<double, double, decltype(dim)::value, true><<<grid, 256, 0, s>>>(
        kind, n, m, d, xs, ys, theta, n_ls, mode, jitter, out, ldo);
  };
  if (d <= 8)
    run(std::integral_constant<int, 8>{});
  else if (d <= 16)
    run(std::integral_constant<int, 16>{});
  else
    run(std::integral_constant<int, 32>{});
  return launch_status();
}

template cudaError_t cross_cov_scaled<double, double>(int, int, int, int, const double*,
                                                      const double*, const double*, int, int,
                                                      double, double*, int64_t, cudaStream_t);
template cudaError_t cross_cov_scaled<float, float>(int, int, int, int, const float*, const float*,
                                                    const double*, int, int, double, float*,
                                                    int64_t, cudaStream_t);

}  // namespace gpk

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
using namespace gpk;

// The public Gram / cross-covariance calls take no workspace: each block
// scales the rows of its output tile by the lengthscales itself, exactly as
// the reference's pointwise kernels do.  (Scaling per output element took 2 d
// float64 divisions for each: 0.70 ms at 3000 x 1100, d = 5.)
template <typename T, int D, int TE>
__global__ void __launch_bounds__(256)
    cross_cov_raw_kernel(int kind, int n, int m, int d, const double* __restrict__ x, int64_t ldx,
                         const double* __restrict__ y, int64_t ldy,
                         const double* __restrict__ theta, int n_ls, T* __restrict__ out,
                         int64_t ldo) {
  __shared__ T sx[TE][D + 1], sy[TE][D + 1];
  const int64_t tn = (m + TE - 1) / TE;
  const int i0 = (int)(blockIdx.x / tn) * TE, j0 = (int)(blockIdx.x % tn) * TE;
  for (int e = threadIdx.x; e < 2 * TE * D; e += 256) {
    const bool second = e >= TE * D;
    const int r = (e % (TE * D)) / D, k = e % D;
    const double l = theta[n_ls == 1 ? 0 : min(k, d - 1)];
    if (second)
      sy[r][k] = j0 + r < m && k < d ? (T)(y[(int64_t)(j0 + r) * ldy + k] / l) : T(0);
    else
      sx[r][k] = i0 + r < n && k < d ? (T)(x[(int64_t)(i0 + r) * ldx + k] / l) : T(0);
  }
  __syncthreads();
  const int c = threadIdx.x % TE, gj = j0 + c;
  if (gj >= m) return;
  const T s2 = (T)theta[n_ls], ka = kshape<T>(kind, theta, n_ls);
  T yv[D];
#pragma unroll
  for (int k = 0; k < D; ++k) yv[k] = sy[c][k];
  for (int r = threadIdx.x / TE; r < TE && i0 + r < n; r += 256 / TE) {
    T sq = T(0);
#pragma unroll
    for (int k = 0; k < D; ++k) {
      if (k >= d) continue;
      const T df = sx[r][k] - yv[k];
      sq = fma(df, df, sq);
    }
    out[(int64_t)(i0 + r) * ldo + gj] = kval<T>(kind, sq, s2, ka);
  }
}

template <typename T>
static void cross_cov_raw(int kind, int n, int m, int d, const double* x, int64_t ldx,
                          const double* y, int64_t ldy, const double* theta, int n_ls, T* out,
                          int64_t ldo, cudaStream_t s) {
  auto run = [&](auto dim, auto edge) {
    constexpr int D = decltype(dim)::value, TE = decltype(edge)::value;
    const int64_t tiles = cdiv(n, TE) * cdiv(m, TE);
    cross_cov_raw_kernel<T, D, TE><<<(unsigned)tiles, 256, 0, s>>>(kind, n, m, d, x, ldx, y, ldy,
                                                                   theta, n_ls, out, ldo);
  };
  auto by_edge = [&](auto dim) {
    // 16-wide tiles until two waves of 64-wide ones exist
    if (cdiv(n, 64) * cdiv(m, 64) >= 304)
      run(dim, std::integral_constant<int, 64>{});
    else
      run(dim, std::integral_constant<int, 16>{});
  };
  if (d <= 8)
    by_edge(std::integral_constant<int, 8>{});
  else if (d <= 16)
    by_edge(std::integral_constant<int, 16>{});
  else
    by_edge(std::integral_constant<int, 32>{});
}

__global__ void diagonal_kernel(int kind, int n, int d, const double* __restrict__ x, int64_t ldx,
                                const double* __restrict__ theta, int n_ls,
                                double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double sq = 0.0;
  for (int k = 0; k < d; ++k) {
    const double v = x[(int64_t)i * ldx + k] / theta[n_ls == 1 ? 0 : k];
    const double df = v - v;  // a NaN or an infinity stays one
    sq = fma(df, df, sq);
  }
  out[i] = kval<double>(kind, sq, theta[n_ls], kshape<double>(kind, theta, n_ls));
}

static bool valid_common(int kind, int64_t n, int d, int n_ls) {
  if (kind < GPK_RBF || kind > GPK_RATIONAL_QUADRATIC) return false;
  if (n < 0 || d <= 0 || d > GPK_MAX_D) return false;
  if (!(n_ls == 1 || n_ls == d)) return false;
  if (n > (int64_t)1 << 30) return false;
  return true;
}

extern "C" gpk_status gpk_cross_covariance(int kind, int64_t n, int64_t m, int d, const double* x,
                                           int64_t ldx, const double* y, int64_t ldy,
                                           const double* theta, int n_ls, int out_dtype, void* out,
                                           int64_t ldo, cudaStream_t stream) {
  if (!valid_common(kind, n, d, n_ls) || m < 0 || ldx < d || ldy < d || ldo < m)
    return GPK_ERR_BAD_ARG;
  if (n == 0 || m == 0) return GPK_OK;
  if (!x || !y || !theta || !out) return GPK_ERR_BAD_ARG;
  if (out_dtype == GPK_F64)
    cross_cov_raw<double>(kind, (int)n, (int)m, d, x, ldx, y, ldy, theta, n_ls, (double*)out, ldo,
                          stream);
  else if (out_dtype == GPK_F32)
    cross_cov_raw<float>(kind, (int)n, (int)m, d, x, ldx, y, ldy, theta, n_ls, (float*)out, ldo,
                         stream);
  else
    return GPK_ERR_BAD_ARG;
  GPK_LAUNCH_CHECK();
  return GPK_OK;
}

extern "C" gpk_status gpk_gram(int kind, int64_t n, int d, const double* x, int64_t ldx,
                               const double* theta, int n_ls, int out_dtype, void* out,
                               int64_t ldo, cudaStream_t stream) {
  return gpk_cross_covariance(kind, n, n, d, x, ldx, x, ldx, theta, n_ls, out_dtype, out, ldo,
                              stream);
}

extern "C" gpk_status gpk_diagonal(int kind, int64_t n, int d, const double* x, int64_t ldx,
                                   const double* theta, int n_ls, double* out,
                                   cudaStream_t stream) {
  if (!valid_common(kind, n, d, n_ls) || ldx < d) return GPK_ERR_BAD_ARG;
  if (n == 0) return GPK_OK;
  if (!x || !theta || !out) return GPK_ERR_BAD_ARG;
  diagonal_kernel<<<(int)cdiv(n, 256), 256, 0, stream>>>(kind, (int)n, d, x, ldx, theta, n_ls,
                                                         out);
  GPK_LAUNCH_CHECK();
  return GPK_OK;
}
