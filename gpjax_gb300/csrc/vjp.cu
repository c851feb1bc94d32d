// Cotangent of the cross-covariance: given G = dL/dK for K = K(x, y),
//   d theta: sum_ij G_ij dK_ij/dl_k, sum_ij G_ij dK_ij/d variance
//   d x_i = sum_j G_ij dk(x_i, y_j)/dx_i,  d y_j = sum_i G_ij dk(x_i, y_j)/dy_j
// (the reverse-mode derivative of DenseKernelComputation.cross_covariance,
// gpjax/kernels/computations/dense.py:32-36).
//
// Float64 arithmetic bounds it (1.7 operations per clock and SM), so every
// element's kernel is evaluated once and the inputs are scaled once per tile: a
// block holds a column tile and walks a strip of row tiles; column sums (d y,
// theta) stay in registers, and the elements' coefficients pass through shared
// memory to the threads that sum rows (d x).  Each column tile leaves n d partial
// row sums; past 128 MB of them the columns go in groups, whose sums are taken
// before the next begins (all at once they would be as large as G at d = 32).
// All partial sums are added in a fixed order.  Two passes that scaled and evaluated every element twice, and
// a finalisation in one block, took 1.82 ms at 3000 x 1100, d = 5.
#include <algorithm>
#include "gpk_internal.cuh"

namespace gpk {
namespace {

struct VjpShape {
  int te, tn;             // tile edge, column tiles
  int group;              // column tiles at a time
  int strips, per;        // strips of row tiles, row tiles per strip
};
constexpr int64_t VJP_ROW_BYTES = (int64_t)128 << 20;  // partial row sums held at a time

// 64-wide tiles from 256 of them (d <= 16: registers): 165 us against 187 with
// 32-wide ones at 1024 x 1024, d = 5, and 144 against 150 (d = 12), 92 against
// 89 (d = 5) at 640 x 640; 16-wide ones are no faster at any size (97 against
// 84 us at 384 x 384).  The row tiles are cut into strips that fill whole
// waves of the blocks an SM holds (by registers 3, 2 or 1), a block costing
// its tiles and about 0.15 of one more: 3000 x 1100, d = 5 took 539 us in 432
// blocks of two tiles, one wave and a 0.4, and 439 in 288 of three.
VjpShape vjp_shape(int64_t n, int64_t m, int d, bool need_x) {
  VjpShape s{};
  s.te = d <= 16 && cdiv(n, 64) * cdiv(m, 64) >= 256 ? 64 : 32;
  const int64_t tm = cdiv(n, s.te), slots = 152 * (d <= 4 ? 3 : d <= 8 ? 2 : 1);
  s.tn = (int)cdiv(m, s.te);
  if (!s.tn) return s;
  s.group = s.tn;
  if (need_x)
    s.group = (int)std::max<int64_t>(
        1, std::min<int64_t>(s.tn, VJP_ROW_BYTES / std::max<int64_t>(1, n * d * 8)));
  double best = 0.0;
  // at most about 8 waves (bounded partial sums)
  for (int64_t per = std::min(tm, cdiv(tm * s.group, 8 * slots)); per > 0 && per <= tm; ++per) {
    const int64_t strips = cdiv(tm, per);
    const double cost = (double)cdiv(strips * s.group, slots) * ((double)per + 0.15);
    if (!s.per || cost < best) {
      best = cost;
      s.per = (int)per;
      s.strips = (int)strips;
    }
    if (strips * s.group <= slots) break;  // one wave: longer strips only cost more
  }
  return s;
}

struct VjpBuf {
  // one group's: [group][n][d], [strips][its columns][d], [strips * group][d + 1];
  // theta's sums over the groups before, [d + 1]
  double *rpart, *cpart, *tpart, *tsum;
};

size_t vjp_layout(int64_t n, int64_t m, int d, bool need_x, bool need_y, void* ws, VjpBuf& b) {
  const VjpShape s = vjp_shape(n, m, d, need_x);
  double* p = static_cast<double*>(ws);
  size_t off = 0;
  auto take = [&](size_t count) {
    double* q = p ? p + off : nullptr;
    off += count;
    return q;
  };
  const int64_t cols = std::min<int64_t>(m, (int64_t)s.group * s.te);
  b.rpart = need_x ? take((size_t)s.group * n * d) : nullptr;
  b.cpart = need_y ? take((size_t)s.strips * cols * d) : nullptr;
  b.tpart = take((size_t)s.strips * s.group * (d + 1));
  b.tsum = take((size_t)d + 1);
  return off * sizeof(double) + 512;
}

template <int D, int TE>
__host__ __device__ constexpr size_t vjp_smem() {
  constexpr size_t red = (size_t)(256 / TE) * TE * D;  // column sums of the row phases
  constexpr size_t st = (size_t)TE * (TE + 4);
  return ((size_t)2 * TE * (D + 1) + (st > red ? st : red) + 8 * (D + 1)) * sizeof(double);
}

template <int D, int TE>
__global__ void __launch_bounds__(256)
    vjp_tile_kernel(int kind, int n, int m, int d, int per, int J0, int cols,
                    const double* __restrict__ x,
                    int64_t ldx, const double* __restrict__ y, int64_t ldy,
                    const double* __restrict__ theta, int n_ls, const double* __restrict__ G,
                    int64_t ldg, double* __restrict__ rpart, double* __restrict__ cpart,
                    double* __restrict__ tpart) {
  constexpr int PH = 256 / TE;  // row phases; lanes of one row in the row sums
  extern __shared__ __align__(16) double vjp_sm[];
  double* sx = vjp_sm;                   // [TE][D + 1]
  double* sy = sx + TE * (D + 1);        // [TE][D + 1]
  double* st = sy + TE * (D + 1);        // [TE][TE + 4]
  double* red = vjp_sm + vjp_smem<D, TE>() / 8 - 8 * (D + 1);
  const int J = blockIdx.x, j0 = (J0 + J) * TE;  // J: within the group
  const int c = threadIdx.x % TE, ph = threadIdx.x / TE, gj = j0 + c;
  const double ka = kshape<double>(kind, theta, n_ls);
  auto scale = [&](double* out, const double* p, int64_t ld, int o, int rows) {
    for (int e = threadIdx.x; e < TE * D; e += 256) {
      const int r = e / D, k = e % D;
      out[r * (D + 1) + k] =
          o + r < rows && k < d ? p[(int64_t)(o + r) * ld + k] / theta[n_ls == 1 ? 0 : k] : 0.0;
    }
  };
  scale(sy, y, ldy, j0, m);
  __syncthreads();
  double yv[D], al[D], az[D], av = 0.0;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    yv[k] = sy[c * (D + 1) + k];
    al[k] = az[k] = 0.0;
  }
  const int tiles = (n + TE - 1) / TE;
  const int tend = min(tiles, ((int)blockIdx.y + 1) * per);
  for (int t = blockIdx.y * per; t < tend; ++t) {
    const int i0 = t * TE;
    __syncthreads();  // the tile before is consumed
    scale(sx, x, ldx, i0, n);
    __syncthreads();
    for (int r = ph; r < TE; r += PH) {
      const int gi = i0 + r;
      double coef = 0.0;
      if (gi < n && gj < m) {
        const double g = G[(int64_t)gi * ldg + gj];
        double df[D], sq = 0.0;
#pragma unroll
        for (int k = 0; k < D; ++k) {
          if (k >= d) continue;  // uniform: padding coordinates cost no float64 work
          df[k] = sx[r * (D + 1) + k] - yv[k];
          sq = fma(df[k], df[k], sq);
        }
        double k1, c1;
        kval_dcoef<double>(kind, sq, 1.0, k1, c1, ka);
        av = fma(g, k1, av);
        coef = g * c1;
#pragma unroll
        for (int k = 0; k < D; ++k) {
          if (k >= d) continue;
          const double v = coef * df[k];
          az[k] += v;
          al[k] = fma(v, df[k], al[k]);
        }
      }
      if (rpart) st[r * (TE + 4) + c] = coef;
    }
    if (rpart) {
      __syncthreads();
      const int r = threadIdx.x / PH, sub = threadIdx.x % PH, gi = i0 + r;
      double xv[D], ar[D];
#pragma unroll
      for (int k = 0; k < D; ++k) {
        xv[k] = sx[r * (D + 1) + k];
        ar[k] = 0.0;
      }
      for (int cc = sub; cc < TE; cc += PH) {
        const double coef = st[r * (TE + 4) + cc];
#pragma unroll
        for (int k = 0; k < D; ++k)
          if (k < d) ar[k] = fma(coef, xv[k] - sy[cc * (D + 1) + k], ar[k]);
      }
#pragma unroll
      for (int k = 0; k < D; ++k) {
        if (k >= d) continue;
#pragma unroll
        for (int o = 1; o < PH; o *= 2) ar[k] += __shfl_xor_sync(0xffffffffu, ar[k], o);
        if (sub == 0 && gi < n && k < d) rpart[((int64_t)J * n + gi) * d + k] = ar[k];
      }
    }
  }
  if (cpart) {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < D; ++k) st[(ph * TE + c) * D + k] = az[k];
    __syncthreads();
    for (int e = threadIdx.x; e < TE * d; e += 256) {
      const int r = e / d, k = e % d;
      double v = 0.0;
      for (int p = 0; p < PH; ++p) v += st[(p * TE + r) * D + k];
      if (j0 + r < m) cpart[((int64_t)blockIdx.y * cols + J * TE + r) * d + k] = v;
    }
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const double v = warp_sum(al[k]);
    if (l == 0) red[w * (D + 1) + k] = v;
  }
  const double v = warp_sum(av);
  if (l == 0) red[w * (D + 1) + D] = v;
  __syncthreads();
  if (threadIdx.x <= d) {
    const int k = threadIdx.x < d ? threadIdx.x : D;
    double s = 0.0;
    for (int q = 0; q < 8; ++q) s += red[q * (D + 1) + k];
    tpart[((int64_t)blockIdx.y * gridDim.x + J) * (d + 1) + threadIdx.x] = s;
  }
}

// The sums of one group of tn column tiles (`cols` columns).  Block 0: theta, one
// warp a slot; the others: one output coordinate a thread.  Between groups tsum
// and gx hold the sums so far.
__global__ void __launch_bounds__(256)
    vjp_finalize_kernel(int n, int cols, int d, int tn, int strips, int first_group,
                        int last_group, const double* __restrict__ theta, int n_ls,
                        const double* __restrict__ rpart, const double* __restrict__ cpart,
                        const double* __restrict__ tpart, double* __restrict__ tsum,
                        double* __restrict__ gtheta, double* __restrict__ gx,
                        double* __restrict__ gy) {
  const double s2 = theta[n_ls];
  if (blockIdx.x == 0) {
    __shared__ double sl[GPK_MAX_D + 1];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    for (int k = w; k <= d; k += 8) {
      double t = 0.0;
      for (int q = l; q < tn * strips; q += 32) t += tpart[(int64_t)q * (d + 1) + k];
      t = warp_sum(t);
      if (l == 0) {
        if (!first_group) t += tsum[k];
        sl[k] = tsum[k] = t;
      }
    }
    __syncthreads();
    if (!last_group) return;
    if (n_ls > 1 && threadIdx.x < d) gtheta[threadIdx.x] = s2 * sl[threadIdx.x] / theta[threadIdx.x];
    if (threadIdx.x == 0) {
      if (n_ls == 1) {
        double a = 0.0;
        for (int k = 0; k < d; ++k) a += sl[k];
        gtheta[0] = s2 * a / theta[0];
      }
      gtheta[n_ls] = sl[d];
      gtheta[n_ls + 1] = 0.0;
      gtheta[n_ls + 2] = 0.0;
    }
    return;
  }
  int64_t e = (int64_t)(blockIdx.x - 1) * 256 + threadIdx.x;
  const int64_t nd = gx ? (int64_t)n * d : 0, md = gy ? (int64_t)cols * d : 0;
  const bool first = e < nd;
  if (!first) e -= nd;
  if (!first && e >= md) return;
  const double* p = first ? rpart : cpart;
  const int64_t stride = (int64_t)(first ? n : cols) * d;
  const int parts = first ? tn : strips;
  double t = first && !first_group ? gx[e] : 0.0;
#pragma unroll 8
  for (int q = 0; q < parts; ++q) t += p[q * stride + e];
  const double v = s2 * t / theta[n_ls == 1 ? 0 : (int)(e % d)];
  if (first)
    gx[e] = last_group ? -v : t;
  else
    gy[e] = v;
}

template <int D, int TE>
cudaError_t vjp_launch(int kind, int n, int m, int d, const VjpShape& s, int J0, int tiles,
                       int cols, const double* x, int64_t ldx, const double* y, int64_t ldy,
                       const double* theta, int n_ls, const double* G, int64_t ldg,
                       const VjpBuf& b, cudaStream_t stream) {
  constexpr size_t smem = vjp_smem<D, TE>();
  cudaFuncSetAttribute(vjp_tile_kernel<D, TE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)smem);
  vjp_tile_kernel<D, TE><<<dim3(tiles, s.strips), 256, smem, stream>>>(
      kind, n, m, d, s.per, J0, cols, x, ldx, y, ldy, theta, n_ls, G, ldg, b.rpart, b.cpart,
      b.tpart);
  return launch_status();
}

}  // namespace

size_t cross_cov_vjp_bytes(int64_t n, int64_t m, int d, bool need_x, bool need_y) {
  VjpBuf b;
  return vjp_layout(n, m, d, need_x, need_y, nullptr, b);
}

cudaError_t cross_cov_vjp(int kind, int n, int m, int d, const double* x, int64_t ldx,
                          const double* y, int64_t ldy, const double* theta, int n_ls,
                          const double* G, int64_t ldg, double* gtheta, double* gx, double* gy,
                          void* ws, cudaStream_t stream) {
  const VjpShape s = vjp_shape(n, m, d, gx != nullptr);
  VjpBuf b;
  vjp_layout(n, m, d, gx != nullptr, gy != nullptr, ws, b);
  const int groups = s.group ? (int)cdiv(s.tn, s.group) : 1;  // 1 with nothing in it for m = 0
  for (int g = 0; g < groups; ++g) {
    const int J0 = g * s.group, tiles = std::min(s.group, s.tn - J0), col0 = J0 * s.te;
    const int cols = std::min(m - col0, s.group * s.te);
    if (n > 0 && m > 0) {
      auto run = [&](auto dim) {
        constexpr int D = decltype(dim)::value;
        auto* f = s.te == 64 ? vjp_launch<D, D <= 16 ? 64 : 32> : vjp_launch<D, 32>;
        return f(kind, n, m, d, s, J0, tiles, cols, x, ldx, y, ldy, theta, n_ls, G, ldg, b, stream);
      };
      const cudaError_t e = d <= 4    ? run(std::integral_constant<int, 4>{})
                            : d <= 8  ? run(std::integral_constant<int, 8>{})
                            : d <= 16 ? run(std::integral_constant<int, 16>{})
                                      : run(std::integral_constant<int, 32>{});
      if (e != cudaSuccess) return e;
    }
    const int64_t outs = (gx ? (int64_t)n * d : 0) + (gy ? (int64_t)cols * d : 0);
    vjp_finalize_kernel<<<(unsigned)(1 + cdiv(outs, 256)), 256, 0, stream>>>(
        n, cols, d, tiles, s.strips, g == 0, g == groups - 1, theta, n_ls, b.rpart, b.cpart,
        b.tpart, b.tsum, gtheta, gx, gy ? gy + (int64_t)col0 * d : nullptr);
    const cudaError_t e = launch_status();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace gpk

using namespace gpk;

extern "C" size_t gpk_cross_covariance_vjp_workspace_bytes(int64_t n, int64_t m, int d) {
  if (n < 0 || m < 0 || d <= 0) return 256;
  // (without the x cotangents the columns go in one group: more strips' partials)
  return std::max(cross_cov_vjp_bytes(n, m, d, true, true),
                  cross_cov_vjp_bytes(n, m, d, false, true));
}

extern "C" gpk_status gpk_cross_covariance_vjp(int kind, int64_t n, int64_t m, int d,
                                               const double* x, int64_t ldx, const double* y,
                                               int64_t ldy, const double* theta, int n_ls,
                                               const double* G, int64_t ldg, double* grad_theta,
                                               double* grad_x, double* grad_y, void* workspace,
                                               size_t workspace_bytes, cudaStream_t stream) {
  if (kind < GPK_RBF || kind > GPK_RATIONAL_QUADRATIC || n < 0 || n > (int64_t)1 << 30 || d <= 0 ||
      d > GPK_MAX_D || !(n_ls == 1 || n_ls == d))
    return GPK_ERR_BAD_ARG;
  if (m < 0 || m > (int64_t)1 << 30 || ldx < d || ldy < d || ldg < m) return GPK_ERR_BAD_ARG;
  if (!theta || !grad_theta || !workspace) return GPK_ERR_BAD_ARG;
  if (workspace_bytes < gpk_cross_covariance_vjp_workspace_bytes(n, m, d)) return GPK_ERR_WORKSPACE;
  if ((n > 0 && m > 0) && (!x || !y || !G)) return GPK_ERR_BAD_ARG;
  GPK_CUDA_TRY(cross_cov_vjp(kind, (int)n, (int)m, d, x, ldx, y, ldy, theta, n_ls, G, ldg,
                             grad_theta, grad_x, grad_y, workspace, stream));
  return GPK_OK;
}
