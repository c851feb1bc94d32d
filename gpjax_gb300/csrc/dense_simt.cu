// Dense linear algebra of the float64 form and of the parts of the mixed form
// that stay off the tensor-core GEMM: a batched NT GEMM on CUDA cores with
// triangular operand masks, the blocked Cholesky (64-wide diagonal blocks and
// their panels in fixed point for float64, fixed64.cuh; trailing updates by
// the split GEMM of xgemm.cuh where the product is large enough and scratch
// for its digit planes was given, else by the CUDA-core GEMM), the recursive
// triangular inverse and triangular GEMVs.
//
// The reference reaches the same arithmetic through XLA: jnp.linalg.cholesky
// (gpjax/linalg/operations.py:54-55), jsp.linalg.solve_triangular
// (operations.py:105-107) and the LU of jnp.linalg.solve / slogdet
// (operations.py:109-111,163-165).
#include "fixed64.cuh"
#include "simt_tile.cuh"
#include "xgemm.cuh"

namespace gpk {

// ---------------------------------------------------------------------------
// Batched NT GEMM, register-tiled.
// ---------------------------------------------------------------------------
// BLOCKED (float64): sums of 16 products added in pairs up to 128, those in
// order: an error of about 20 + K / 128 roundings instead of K.
template <typename T, typename Cfg, bool BLOCKED = false>
__global__ void __launch_bounds__((Cfg::BM / Cfg::TM) * (Cfg::BN / Cfg::TN))
    gemm_nt_kernel(GemmProb<T> p) {
  constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK;
  constexpr int TM = Cfg::TM, TN = Cfg::TN;
  constexpr int NTX = BN / TN, NTY = BM / TM;
  const int z = blockIdx.z;
  const T* A = p.A + (int64_t)z * p.sA;
  const T* B = p.B + (int64_t)z * p.sB;
  T* C = p.C ? p.C + (int64_t)z * p.sC : nullptr;
  T* Ct = p.Ct ? p.Ct + (int64_t)z * p.sCt : nullptr;

  const int tilesM = (p.M + BM - 1) / BM, tilesN = (p.N + BN - 1) / BN;
  int I, J;
  const int t = blockIdx.x;
  if (p.c_lower) {
    if (t >= tilesM * (tilesM + 1) / 2) return;
    tri_index(t, I, J);
    if (J >= tilesN) return;  // a tall product's tiles right of its columns
  } else {
    if (t >= tilesM * tilesN) return;
    I = t / tilesN;
    J = t % tilesN;
  }
  const int i0 = I * BM, j0 = J * BN;
  int klo, khi;
  tile_krange<BM, BN, BK>(p.K, p.a_tri, p.b_tri, i0, j0, klo, khi);

  __shared__ SimtSmem<T, Cfg> sm;
  T acc[TM][TN];
#pragma unroll
  for (int a = 0; a < TM; ++a)
#pragma unroll
    for (int b = 0; b < TN; ++b) acc[a][b] = T(0);
  if constexpr (BLOCKED) {
    double l0[TM][TN], l1[TM][TN], l2[TM][TN], total[TM][TN];  // waiting sums of 16, 32, 64
#pragma unroll
    for (int a = 0; a < TM; ++a)
#pragma unroll
      for (int b = 0; b < TN; ++b) l0[a][b] = l1[a][b] = l2[a][b] = total[a][b] = 0.0;
    int blocks = 0;
    auto each = [&](auto f) {
#pragma unroll
      for (int a = 0; a < TM; ++a)
#pragma unroll
        for (int b = 0; b < TN; ++b) f(acc[a][b], l0[a][b], l1[a][b], l2[a][b], total[a][b]);
    };
    typedef double& R;
    simt_tile_mma<T, Cfg>(A, p.lda, p.M, p.a_tri, B, p.ldb, p.N, p.b_tri, i0, j0, klo, khi, sm, acc,
                          [&]() {
                            const int q = blocks++;
                            if (!(q & 1))
                              each([](R v, R w, R, R, R) { w = v, v = 0.0; });
                            else if (!(q & 2))
                              each([](R v, R w0, R w, R, R) { w = w0 + v, v = 0.0; });
                            else if (!(q & 4))
                              each([](R v, R w0, R w1, R w, R) { w = w1 + (w0 + v), v = 0.0; });
                            else
                              each([](R v, R w0, R w1, R w2, R t) {
                                t += w2 + (w1 + (w0 + v)), v = 0.0;
                              });
                          });
    const int q = blocks;  // what is left waiting, the small sums first
    each([q](R v, R w0, R w1, R w2, R t) {
      v = q & 1 ? w0 : 0.0;
      if (q & 2) v += w1;
      if (q & 4) v += w2;
      v += t;
    });
  } else {
    simt_tile_mma<T, Cfg>(A, p.lda, p.M, p.a_tri, B, p.ldb, p.N, p.b_tri, i0, j0, klo, khi, sm,
                          acc);
  }

  const int tx = threadIdx.x % NTX, ty = threadIdx.x / NTX;
#pragma unroll
  for (int a = 0; a < TM; ++a) {
    const int gi = i0 + ty + a * NTY;
    if (gi >= p.M) continue;
#pragma unroll
    for (int b = 0; b < TN; ++b) {
      const int gj = j0 + tx + b * NTX;
      if (gj >= p.N) continue;
      if (p.c_lower && gj > gi) continue;
      T v = p.alpha * acc[a][b];
      if (C) {
        if (p.beta != T(0)) v += p.beta * C[(int64_t)gi * p.ldc + gj];
        C[(int64_t)gi * p.ldc + gj] = v;
      }
      if (Ct) Ct[(int64_t)gj * p.ldct + gi] = v;
    }
  }
}

template <typename T, typename Cfg>
static int gemm_tiles(const GemmProb<T>& p) {
  const int tilesM = (p.M + Cfg::BM - 1) / Cfg::BM, tilesN = (p.N + Cfg::BN - 1) / Cfg::BN;
  return p.c_lower ? tilesM * (tilesM + 1) / 2 : tilesM * tilesN;
}

template <typename T, typename Cfg, bool BLOCKED>
static cudaError_t gemm_nt_cfg(const GemmProb<T>& p, int batch, cudaStream_t s) {
  constexpr int NT = (Cfg::BM / Cfg::TM) * (Cfg::BN / Cfg::TN);
  dim3 grid(gemm_tiles<T, Cfg>(p), 1, batch);
  gemm_nt_kernel<T, Cfg, BLOCKED><<<grid, NT, 0, s>>>(p);
  return launch_status();
}

constexpr int SIMT_SMALL_BELOW = 152;  // CTAs of the full-size grid (one wave)

template <typename T, bool BLOCKED>
static cudaError_t gemm_nt_tiles(const GemmProb<T>& p, int batch, cudaStream_t s) {
  if (p.M <= 0 || p.N <= 0 || batch <= 0) return cudaSuccess;
  // float64 only: the float32 form runs many independent GPs side by side
  // (batched MLL), where total work rather than one launch's latency counts.
  // Products in blocks always: their waiting sums take the registers that 64 x 64
  // tiles would need (2048^3: 18.3 ms with those, 15.1 with 32 x 32).
  if (BLOCKED ||
      (sizeof(T) == 8 && (int64_t)gemm_tiles<T, GemmCfg<T>>(p) * batch < SIMT_SMALL_BELOW)) {
    // tiles of 16 once four times as many 32 x 32 tiles still fit one wave (a
    // 36 x 36 x 64 update: 27 us with 32 x 32 tiles, 9 with 16 x 16)
    if ((int64_t)gemm_tiles<T, GemmCfgSmall<T>>(p) * batch * 4 <= SIMT_SMALL_BELOW)
      return gemm_nt_cfg<T, GemmCfgTiny<T>, BLOCKED>(p, batch, s);
    return gemm_nt_cfg<T, GemmCfgSmall<T>, BLOCKED>(p, batch, s);
  }
  return gemm_nt_cfg<T, GemmCfg<T>, BLOCKED>(p, batch, s);
}

template <typename T>
cudaError_t gemm_nt(const GemmProb<T>& p, int batch, cudaStream_t s) {
  return gemm_nt_tiles<T, false>(p, batch, s);
}

cudaError_t gemm_nt_blocked(const GemmProb<double>& p, cudaStream_t s) {
  return gemm_nt_tiles<double, true>(p, 1, s);
}

// ---------------------------------------------------------------------------
// Diagonal-block Cholesky: one CTA factors the nb x nb block at (k0, k0) in
// shared memory (unblocked right-looking, two barriers per column).  Each
// pivot's square root and reciprocal are taken once, by the thread that
// finishes that diagonal entry.  The float32 form's, and the native float64
// factor's (potrf_lower_native); the float64 objectives' block is below.
// ---------------------------------------------------------------------------
template <typename T, int NB>
__global__ void __launch_bounds__(512) potrf_diag_kernel(T* A, int64_t lda, int n, int k0,
                                                         double* logdiag, int* info,
                                                         const double* __restrict__ dtrack) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int LD = NB + 1;
  double* Dd = reinterpret_cast<double*>(smem_raw);  // float64 diagonal of the block
  double* Pv = Dd + NB;                              // float64 pivots
  T* S = reinterpret_cast<T*>(Pv + NB);
  T* col = S + NB * LD;
  T* dl = col + NB;   // L[j, j]
  T* rl = dl + NB;    // 1 / L[j, j]
  const int nb = min(NB, n - k0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  for (int e = threadIdx.x; e < nb * nb; e += blockDim.x) {
    int i = e / nb, j = e % nb;
    if (j <= i) S[i * LD + j] = A[(int64_t)(k0 + i) * lda + k0 + j];
  }
  // NaN when the pivot is negative, as in the reference; float64 square
  // root only when the factor itself is float64
  auto pivot = [&](int j) {
    const double pivd = Dd[j];
    const T ljj = sizeof(T) == 8 ? (T)sqrt(pivd) : (T)sqrtf((float)pivd);
    Pv[j] = pivd;
    dl[j] = ljj;
    rl[j] = T(1) / ljj;
  };
  for (int i = threadIdx.x; i < nb; i += blockDim.x)
    Dd[i] = dtrack ? dtrack[k0 + i] : (double)A[(int64_t)(k0 + i) * lda + k0 + i];
  __syncthreads();
  if (threadIdx.x == 0 && nb > 0) pivot(0);
  __syncthreads();
  for (int j = 0; j < nb; ++j) {
    const T rj = rl[j];
    for (int i = j + 1 + threadIdx.x; i < nb; i += blockDim.x) {
      T v = S[i * LD + j] * rj;
      S[i * LD + j] = v;
      col[i] = v;
    }
    __syncthreads();
    for (int i = j + 1 + warp; i < nb; i += nwarps) {
      const T ci = col[i];
      for (int k = j + 1 + lane; k < i; k += 32) S[i * LD + k] -= ci * col[k];
    }
    for (int i = j + 1 + threadIdx.x; i < nb; i += blockDim.x) {
      const double c = (double)col[i];
      Dd[i] -= c * c;
      if (i == j + 1) pivot(i);  // Dd[j + 1] is final after this column
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < nb; i += blockDim.x) {
    if (logdiag) logdiag[k0 + i] = 0.5 * log(Pv[i]);
    if (!(Pv[i] > 0.0)) atomicMin(info, k0 + i + 1);
  }
  for (int e = threadIdx.x; e < nb * nb; e += blockDim.x) {
    int i = e / nb, j = e % nb;
    T v = (j < i) ? S[i * LD + j] : (j == i ? dl[i] : T(0));
    A[(int64_t)(k0 + i) * lda + k0 + j] = v;
  }
}

// dtrack[r] -= sum_k P[r, k]^2 in float64 for the rows below the panel.
template <typename T>
__global__ void diag_track_kernel(const T* __restrict__ A, int64_t lda, int n, int r0, int k0,
                                  int nb, double* __restrict__ dtrack) {
  const int r = r0 + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= n) return;
  const T* row = A + (int64_t)r * lda + k0;
  double s = 0.0;
  for (int c = lane; c < nb; c += 32) {
    const double v = (double)row[c];
    s += v * v;
  }
  s = warp_sum(s);
  if (lane == 0) dtrack[r] -= s;
}

// Zeroes the strict upper triangle outside the diagonal blocks of width nb.
template <typename T>
__global__ void zero_upper_kernel(T* A, int64_t lda, int n, int nb) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (int64_t)n * n) return;
  const int i = (int)(e / n), j = (int)(e % n);
  if (j > i && (j / nb) != (i / nb)) A[(int64_t)i * lda + j] = T(0);
}

// Panel solve, float32 form: one thread per row, 128 rows per CTA, L_kk and
// the rows staged in shared memory (the float32 form serves the batched MLL,
// where many solves run side by side).
template <typename T, int NB>
__global__ void __launch_bounds__(128) trsm_rows_thread_kernel(T* A, int64_t lda, int n, int k0) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int LD = NB + 1;
  T* Ls = reinterpret_cast<T*>(smem_raw);
  T* Xs = Ls + NB * LD;
  T* rinv = Xs + 128 * LD;
  const int nb = min(NB, n - k0);
  const int r0 = k0 + nb + blockIdx.x * 128;
  const int rows = min(128, n - r0);
  if (rows <= 0) return;
  for (int e = threadIdx.x; e < nb * nb; e += blockDim.x) {
    int i = e / nb, j = e % nb;
    Ls[i * LD + j] = (j <= i) ? A[(int64_t)(k0 + i) * lda + k0 + j] : T(0);
  }
  for (int e = threadIdx.x; e < rows * nb; e += blockDim.x) {
    int r = e / nb, c = e % nb;
    Xs[r * LD + c] = A[(int64_t)(r0 + r) * lda + k0 + c];
  }
  __syncthreads();
  for (int j = threadIdx.x; j < nb; j += blockDim.x) rinv[j] = T(1) / Ls[j * LD + j];
  __syncthreads();
  if (threadIdx.x < rows) {
    T* x = Xs + threadIdx.x * LD;
    for (int j = 0; j < nb; ++j) {
      T s0 = x[j], s1 = T(0), s2 = T(0), s3 = T(0);
      const T* lj = Ls + j * LD;
      int k = 0;
      for (; k + 4 <= j; k += 4) {
        s0 -= x[k] * lj[k];
        s1 -= x[k + 1] * lj[k + 1];
        s2 -= x[k + 2] * lj[k + 2];
        s3 -= x[k + 3] * lj[k + 3];
      }
      for (; k < j; ++k) s0 -= x[k] * lj[k];
      x[j] = ((s0 + s1) + (s2 + s3)) * rinv[j];
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < rows * nb; e += blockDim.x) {
    int r = e / nb, c = e % nb;
    A[(int64_t)(r0 + r) * lda + k0 + c] = Xs[r * LD + c];
  }
}

// ---------------------------------------------------------------------------
// Float64 form of both, in fixed point (fixed64.cuh).
//
// The diagonal block: thread (row i, column group g), right-looking, in groups
// of eight columns.  The chain of 64 pivots bounds it (a reciprocal root takes
// about 290 clocks, a scaled entry 145, a product and its difference 110, a
// barrier 50): one group of threads runs the chain, the other seven apply each
// column to the rest of its group and, one column a step, the group before to
// the columns further right, so that nothing but the next group's own columns
// is waited for between groups.  (A single warp holding a whole group in
// registers needs no barriers but then issues every product itself: 65 us
// against 40.)
// ---------------------------------------------------------------------------
constexpr int FX_NB = 64;
constexpr int FX_G = 8;     // columns of a group, and groups of threads
constexpr int FX_NT = 512;  // threads: 64 rows x 8
constexpr int FX_EL = FX_NB * FX_NB / FX_NT;
__global__ void __launch_bounds__(FX_NT)
    potrf_diag_fixed_kernel(double* A, int64_t lda, int n, int k0, double* logdiag, int* info,
                            int keep_upper) {
  using namespace fx;
  pdl_wait();
  pdl_trigger();
  __shared__ long long S[FX_NB][FX_NB + 1];
  __shared__ Limbs lim[2][FX_G][FX_NB];  // this group's columns and the last one's
  __shared__ int ex[FX_NB], sbad[FX_NB], sinf[FX_NB], sdead, sany;
  const int nb = min(FX_NB, n - k0);
  const int i = threadIdx.x & 63, g = threadIdx.x >> 6;
  double av[FX_EL];  // every load in flight at once
#pragma unroll
  for (int u = 0; u < FX_EL; ++u) {
    const int e = threadIdx.x + u * FX_NT, r = e >> 6, c = e & 63;
    av[u] = r < nb && c <= r ? A[(int64_t)(k0 + r) * lda + k0 + c] : 0.0;
  }
  if (threadIdx.x < FX_NB) {
    const double a = i < nb ? A[(int64_t)(k0 + i) * lda + k0 + i] : 1.0;
    ex[i] = scale_of(a);
    sbad[i] = 0;
    sinf[i] = __double_as_longlong(a) == 0x7ff0000000000000LL;
    if (i == 0) sdead = sany = 0;
  }
  __syncthreads();
  if (threadIdx.x < FX_NB && sinf[i]) sany = 1;
#pragma unroll
  for (int u = 0; u < FX_EL; ++u) {
    const int e = threadIdx.x + u * FX_NT, r = e >> 6, c = e & 63;
    bool bad = false;
    S[r][c] = r < nb || r != c ? to_fixed(av[u], ex[r] + ex[c], bad) : ONE;  // identity past nb
    if (bad && !(r == c && sinf[r])) sbad[r] = 1;
  }
  __syncthreads();
  // an infinite variance (a noise whose square overflows) is no failure: its
  // pivot is infinite and the rest of its row and column zero
  const bool any = sany;
  if (any) {
    for (int e = threadIdx.x; e < FX_NB * FX_NB; e += FX_NT) {
      const int r = e >> 6, c = e & 63;
      if (sinf[r] || sinf[c]) S[r][c] = r == c ? ONE : 0;
    }
    __syncthreads();
  }
  // column k loses the eight columns of a group
  auto update = [&](const Limbs (&l)[FX_G][FX_NB], int k) {
    if (k >= nb || i < k) return;
    Acc a0, a1;
#pragma unroll
    for (int q = 0; q < FX_G; q += 2) {
      a0.add(l[q][i], l[q][k]);
      a1.add(l[q + 1][i], l[q + 1][k]);
    }
    S[i][k] -= a0.value() + a1.value();
  };
  // The squared norm of this row of the factor (last 64 threads): in a definite
  // matrix at most its diagonal entry, which the scale puts below 1.  A diagonal
  // entry can leave the range of [-8, 8) and come back as another number, but
  // not between two groups' looks at the norm: the row is marked before its
  // pivot's turn.
  float norm = 0.f;
  for (int c0 = 0; c0 < nb; c0 += FX_G) {
    Limbs(&cur)[FX_G][FX_NB] = lim[(c0 / FX_G) & 1];
    Limbs(&prev)[FX_G][FX_NB] = lim[((c0 / FX_G) & 1) ^ 1];
    Limbs lv{0, 0};  // this row's entry of the previous column (first 64 threads)
#pragma unroll
    for (int q = 0; q < FX_G; ++q) {
      const int j = c0 + q;
      if (g == 0) {
        long long t = S[i][j], d = S[j][j];
        const int jbad = sbad[j];
        if (q > 0) {
          const Limbs w = cur[q - 1][j];
          Acc at, ad;
          at.add(lv, w);
          ad.add(w, w);
          t -= at.value();
          d -= ad.value();
        }
        const bool good = d > 0 && !jbad;
        long long y;
        int s;
        rsqrt_fixed(good ? d : ONE, y, s);
        bool bad = false;
        const long long v = times_rsqrt(i >= j ? t : 0, y, s, bad);
        lv = limbs(v);
        cur[q][i] = lv;
        if (bad) sbad[i] = 1;
        if ((!good || bad) && i == j) {  // the rest of this group's columns mean nothing
          atomicMin(info, k0 + j + 1);
          sdead = 1;
        }
      } else {
        if (q > 0) {
          const int k = j + g;  // the group's columns after j
          if (k < c0 + FX_G && i >= k) {
            Acc acc;
            acc.add(cur[q - 1][i], cur[q - 1][k]);
            S[i][k] -= acc.value();
          }
        }
        if (c0 > 0) update(prev, c0 + FX_G + q * (FX_G - 1) + g - 1);
      }
      __syncthreads();
    }
    if (sdead) break;
    update(cur, c0 + FX_G + g);  // the next group's columns
    if (g == FX_G - 1) {
#pragma unroll
      for (int q = 0; q < FX_G; ++q) {
        const float f = (float)cur[q][i].h * 0x1p-28f;
        norm = fmaf(f, f, norm);
      }
      if (norm > 1.5f) sbad[i] = 1;
    }
    const Limbs l = cur[g][i];
    S[i][c0 + g] = ((long long)l.h << 32) + l.l;
    __syncthreads();
  }
  const bool dead = sdead != 0;  // a pivot failed
  const double nan = __longlong_as_double(0x7ff8000000000000ULL);
  const double inf = __longlong_as_double(0x7ff0000000000000ULL);
#pragma unroll 4
  for (int u = 0; u < FX_EL; ++u) {
    const int e = threadIdx.x + u * FX_NT, r = e >> 6, c = e & 63;
    if (r < nb && c < nb && !(keep_upper && c > r))
      A[(int64_t)(k0 + r) * lda + k0 + c] =
          c > r ? 0.0 : dead ? nan : any && c == r && sinf[r] ? inf : to_double(S[r][c], ex[r]);
  }
  if (logdiag && threadIdx.x < nb)
    logdiag[k0 + i] = dead ? nan : any && sinf[i] ? inf : log(to_double(S[i][i], ex[i]));
}

// Panel solve X L^T = A for 32 rows per CTA: lane = row.  One warp substitutes
// a group of four columns while the others apply the group before it to the
// columns further right; only the next group's four columns are brought up to
// date in between.  A row's scale comes from its own diagonal entry, which
// bounds every entry of the factor's row; a column's from the norm of that row
// of L.
constexpr int FX_ROWS = 32;
constexpr int FX_XLD = FX_NB + 1;
constexpr int FX_TG = 4;  // columns of a group
constexpr int FX_TW = FX_NT / 32;
constexpr size_t FX_TRSM_SMEM = (size_t)FX_NB * FX_NB * sizeof(fx::Limbs) +
                                (size_t)FX_ROWS * FX_XLD * 8 + (size_t)FX_NB * 16 +
                                FX_ROWS * 8 + (size_t)2 * FX_TG * FX_ROWS * sizeof(fx::Limbs);
__global__ void __launch_bounds__(FX_NT)
    trsm_rows_fixed_kernel(double* A, int64_t lda, int n, int k0, XSplit planes) {
  using namespace fx;
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Limbs* L = reinterpret_cast<Limbs*>(smem_raw);                   // [64][64], row j of L
  long long* X = reinterpret_cast<long long*>(L + FX_NB * FX_NB);  // [32][65]
  long long* ry = X + FX_ROWS * FX_XLD;                            // 1 / L_jj: mantissa
  int* rs = reinterpret_cast<int*>(ry + FX_NB);                    // and shift
  int* ej = rs + FX_NB;
  int* ei = ej + FX_NB;
  int* sbad = ei + FX_ROWS;
  Limbs* LX = reinterpret_cast<Limbs*>(sbad + FX_ROWS);            // [2][FX_TG][32]
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int r0 = k0 + FX_NB + blockIdx.x * FX_ROWS, rows = min(FX_ROWS, n - r0);
  constexpr int XE = FX_ROWS * FX_NB / FX_NT, LE = FX_NB / FX_TW;
  double av[XE], lv[2 * LE];  // every load in flight at once
#pragma unroll
  for (int u = 0; u < LE; ++u)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = g + FX_TW * u, k = lane + 32 * h;
      lv[2 * u + h] = k <= j ? A[(int64_t)(k0 + j) * lda + k0 + k] : 0.0;
    }
#pragma unroll
  for (int u = 0; u < XE; ++u) {
    const int e = threadIdx.x + u * FX_NT, r = e >> 6, c = e & 63;
    av[u] = r < rows ? A[(int64_t)(r0 + r) * lda + k0 + c] : 0.0;
  }
  if (threadIdx.x < FX_ROWS) {
    const int r = r0 + threadIdx.x;
    ei[threadIdx.x] = threadIdx.x < rows ? scale_of(A[(int64_t)r * lda + r]) : 0;
    sbad[threadIdx.x] = 0;
  }
#pragma unroll
  for (int u = 0; u < LE; ++u) {
    const int j = g + FX_TW * u;
    const double* a = lv + 2 * u;
    int xb[2], xm = 1;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      xb[h] = (int)((__double_as_longlong(a[h]) >> 52) & 0x7ff);
      xm = max(xm, xb[h]);
    }
    xm = __reduce_max_sync(0xffffffffu, xm);
    // squared norm over 2^(2 (xm - 1022)) from the leading bits, rounded up
    float nsq = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const unsigned top = (unsigned)(__double_as_longlong(a[h]) >> 29) & 0x7fffffu;
      const float f = xm - xb[h] < 100
                          ? __uint_as_float(((unsigned)(126 - (xm - xb[h])) << 23) | top)
                          : 0.f;
      nsq = fmaf(f, f, nsq);
    }
    nsq = warp_sum(nsq) * 1.00001f;  // below 64
    const int x2 = (int)((__float_as_uint(nsq) >> 23) & 0xff) - 126;  // nsq < 2^x2
    const int e = xm - 1022 + ((x2 + 1) >> 1);
    bool bad = false;  // a NaN of a failed block: its rows' results are not read
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      L[j * FX_NB + lane + 32 * h] = limbs(to_fixed(a[h], e, bad));
      if (lane + 32 * h == j) ry[j] = __double_as_longlong(a[h]);
    }
    if (lane == 0) ej[j] = e;
  }
  __syncthreads();
  if (threadIdx.x < FX_NB) {
    const int j = threadIdx.x;
    const unsigned long long b =
        (unsigned long long)__double_as_longlong(1.0 / __longlong_as_double(ry[j]));
    const int x = (int)((b >> 52) & 0x7ff), s = -(x - 1023 + ej[j]);
    const bool ok = x != 0x7ff && s >= -58 && s <= 1;  // not a failed block
    ry[j] = ok ? (long long)((b & 0xfffffffffffffULL) | (1ULL << 52)) << 9 : 0;
    rs[j] = ok ? s : 0;  // [1, 2) 2^61 and its shift
  }
#pragma unroll
  for (int u = 0; u < XE; ++u) {
    const int e = threadIdx.x + u * FX_NT, r = e >> 6, c = e & 63;
    bool bad = false;
    X[r * FX_XLD + c] = to_fixed(av[u], ei[r] + ej[c], bad);
    if (bad) sbad[r] = 1;
  }
  __syncthreads();
  long long* x = X + lane * FX_XLD;
  // The squared norm of the row's solved entries: below 1 in a definite matrix
  // (its scale is that of its diagonal entry).  An entry can leave the range of
  // [-8, 8) and come back as another number only in a row of norm 6 and more,
  // which is marked before.
  float norm = 0.f;
  auto solve = [&](int c0) {  // one warp: the group's four columns
    Limbs* out = LX + ((c0 / FX_TG) & 1) * FX_TG * FX_ROWS;
    long long t[FX_TG];
    bool bad = false;
#pragma unroll
    for (int q = 0; q < FX_TG; ++q) t[q] = x[c0 + q];
#pragma unroll
    for (int q = 0; q < FX_TG; ++q) {
      t[q] = times_rsqrt(t[q], ry[c0 + q], rs[c0 + q], bad);
      const Limbs l = limbs(t[q]);
      const float f = (float)l.h * 0x1p-28f;
      norm = fmaf(f, f, norm);
      out[q * FX_ROWS + lane] = l;
#pragma unroll
      for (int u = q + 1; u < FX_TG; ++u) {
        Acc acc;
        acc.add(l, L[(c0 + u) * FX_NB + c0 + q]);
        t[u] -= acc.value();
      }
    }
#pragma unroll
    for (int q = 0; q < FX_TG; ++q) x[c0 + q] = t[q];
    if (bad || norm > 2.f) sbad[lane] = 1;
  };
  auto update = [&](const Limbs (&lx)[FX_TG], int c0, int k) {  // column k loses the group at c0
    Acc acc;
#pragma unroll
    for (int q = 0; q < FX_TG; ++q) acc.add(lx[q], L[k * FX_NB + c0 + q]);
    x[k] -= acc.value();
  };
  if (g == 0) solve(0);
  __syncthreads();
  for (int c0 = 0; c0 + FX_TG < FX_NB; c0 += FX_TG) {
    const Limbs* in = LX + ((c0 / FX_TG) & 1) * FX_TG * FX_ROWS;
    Limbs lx[FX_TG];
#pragma unroll
    for (int q = 0; q < FX_TG; ++q) lx[q] = in[q * FX_ROWS + lane];
    if (g < FX_TG) update(lx, c0, c0 + FX_TG + g);  // the next group's columns
    __syncthreads();
    if (g == 0)
      solve(c0 + FX_TG);
    else
      for (int k = c0 + 2 * FX_TG + g - 1; k < FX_NB; k += FX_TW - 1) update(lx, c0, k);
    __syncthreads();
  }
  const double nan = __longlong_as_double(0x7ff8000000000000ULL);
#pragma unroll
  for (int u = 0; u < XE; ++u) {
    const int e = threadIdx.x + u * FX_NT, r = e >> 6, c = e & 63;
    if (r < rows)
      A[(int64_t)(r0 + r) * lda + k0 + c] =
          sbad[r] ? nan : to_double(X[r * FX_XLD + c], ei[r]);
  }
  // The panel's digit planes for the products that read it, at the row scale of
  // the first panel (updates only lower a diagonal entry and with it the scale).
  // A diagonal entry below half of the scale's square bounds the row by 0.71 of
  // it: there the planes take half the scale, at which their top digit stays
  // below 182 (XPER's bound) and the 55 bits reach one place further.  At the
  // whole scale the products put the noise gradient of an RBF with unit variance
  // (a diagonal of 1.01) at 1.7 times the native factor's error, median of 16
  // draws at n = 1200: 4.7e-14 against 2.7e-14, at half of it 1.8e-14.
  if (planes.planes) {
    const int r = threadIdx.x >> 4, c = (threadIdx.x & 15) * 4;
    const bool in = r < rows;  // a warp's second row may be past the last
    int* expo = planes.expo + r0 + r;
    int e0 = 0;
    if (in && k0 == 0)  // an odd exponent field: a < 2^(2 ei - 1)
      e0 = ei[r] - (int)(__double_as_longlong(A[(int64_t)(r0 + r) * lda + r0 + r]) >> 52 & 1);
    else if (in)
      e0 = *expo - 1022;
    __syncwarp();  // the row's 16 lanes have read its exponent
    if (in) {
      const bool ok = !sbad[r] && ei[r] <= e0 + 1;
      const int sh = min(62, FRAC - 55 + (ok ? e0 - ei[r] : 0));
      long long q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = (X[r * FX_XLD + c + u] + (1LL << (sh - 1))) >> sh;
      x_store_digits4(q,
                      static_cast<__half*>(planes.planes) + (int64_t)(r0 + r) * planes.ldk + k0 + c,
                      (int64_t)planes.rows * planes.ldk);
      if (c == 0 && (k0 == 0 || !ok)) *expo = ok ? e0 + 1022 : XNAN;
    }
  }
}

// Factor the 64 columns at o and the rows below (and the rows' digit planes,
// where there are any).  The kernels start while their predecessor drains.
static cudaError_t potrf_block64(double* A, int64_t lda, int n, int o, double* logdiag, int* info,
                                 bool keep_upper, const XSplit& planes, cudaStream_t s) {
  const PdlAttr attr(o > 0);  // the first follows whatever the caller did before
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1);
  cfg.blockDim = dim3(FX_NT);
  cfg.stream = s;
  cfg.attrs = const_cast<cudaLaunchAttribute*>(attr.a);
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, potrf_diag_fixed_kernel, A, lda, n, o, logdiag, info,
                     (int)keep_upper);
  cudaError_t e = launch_status();
  const int rest = n - o - FX_NB;
  if (e != cudaSuccess || rest <= 0) return e;
  cudaFuncSetAttribute(trsm_rows_fixed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)FX_TRSM_SMEM);
  const PdlAttr pdl(true);
  cfg.gridDim = dim3((rest + FX_ROWS - 1) / FX_ROWS);
  cfg.dynamicSmemBytes = FX_TRSM_SMEM;
  cfg.attrs = const_cast<cudaLaunchAttribute*>(pdl.a);
  cudaLaunchKernelEx(&cfg, trsm_rows_fixed_kernel, A, lda, n, o, planes);
  return launch_status();
}

// Panel solve, native float64: TRSM_ROWS rows per CTA (so that a short panel
// still spreads over many SMs: float64 throughput per SM is low), eliminated
// column by column by all threads: after column j is final, every later
// column c of every row takes x[c] -= (x[j] / L[j, j]) L[c, j].  The columns
// stay unscaled until the end (one barrier per column).
constexpr int TRSM_ROWS = 32;
template <typename T, int NB>
__global__ void __launch_bounds__(256) trsm_rows_kernel(T* A, int64_t lda, int n, int k0) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int LD = NB + 1;
  T* Ls = reinterpret_cast<T*>(smem_raw);
  T* Xs = Ls + NB * LD;
  T* rinv = Xs + TRSM_ROWS * LD;
  const int nb = min(NB, n - k0);
  const int r0 = k0 + nb + blockIdx.x * TRSM_ROWS;
  const int rows = min(TRSM_ROWS, n - r0);
  if (rows <= 0) return;
  for (int e = threadIdx.x; e < nb * nb; e += blockDim.x) {
    int i = e / nb, j = e % nb;
    Ls[i * LD + j] = (j <= i) ? A[(int64_t)(k0 + i) * lda + k0 + j] : T(0);
  }
  for (int e = threadIdx.x; e < rows * nb; e += blockDim.x) {
    int r = e / nb, c = e % nb;
    Xs[r * LD + c] = A[(int64_t)(r0 + r) * lda + k0 + c];
  }
  __syncthreads();
  for (int j = threadIdx.x; j < nb; j += blockDim.x) rinv[j] = T(1) / Ls[j * LD + j];
  __syncthreads();
  for (int j = 0; j + 1 < nb; ++j) {
    const int w = nb - 1 - j;  // columns j+1 .. nb-1
    const T rj = rinv[j];
    for (int e = threadIdx.x; e < rows * w; e += blockDim.x) {
      const int r = e / w, c = j + 1 + e % w;
      Xs[r * LD + c] -= (Xs[r * LD + j] * rj) * Ls[c * LD + j];
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < rows * nb; e += blockDim.x) {
    int r = e / nb, c = e % nb;
    A[(int64_t)(r0 + r) * lda + k0 + c] = Xs[r * LD + c] * rinv[c];
  }
}

// The factor in native float64 throughout (right-looking, CUDA-core updates),
// 72 us a diagonal block: for a caller's matrix (gpk_lower_cholesky) and the
// mixed collapsed bound (sgpr.cu).
cudaError_t potrf_lower_native(double* A, int64_t lda, int n, double* logdiag, int* info,
                               bool zero_upper, cudaStream_t s) {
  constexpr int NB = Blk<double>::NB;
  const size_t smem_diag = (size_t)(NB * (NB + 1) + 5 * NB) * sizeof(double);
  const size_t smem_trsm = (size_t)(NB * (NB + 1) + TRSM_ROWS * (NB + 1) + NB) * sizeof(double);
  cudaFuncSetAttribute(potrf_diag_kernel<double, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)smem_diag);
  cudaFuncSetAttribute(trsm_rows_kernel<double, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)smem_trsm);
  if (zero_upper && n > NB) {
    zero_upper_kernel<double><<<(int)cdiv((int64_t)n * n, 256), 256, 0, s>>>(A, lda, n, NB);
    cudaError_t e = launch_status();
    if (e != cudaSuccess) return e;
  }
  for (int k0 = 0; k0 < n; k0 += NB) {
    const int nb = min(NB, n - k0), rest = n - k0 - nb;
    potrf_diag_kernel<double, NB><<<1, 512, smem_diag, s>>>(A, lda, n, k0, logdiag, info, nullptr);
    cudaError_t e = launch_status();
    if (e != cudaSuccess || rest <= 0) return e;
    trsm_rows_kernel<double, NB><<<(rest + TRSM_ROWS - 1) / TRSM_ROWS, 256, smem_trsm, s>>>(
        A, lda, n, k0);
    e = launch_status();
    if (e != cudaSuccess) return e;
    GemmProb<double> p{};
    p.A = p.B = A + (int64_t)(k0 + nb) * lda + k0;
    p.C = A + (int64_t)(k0 + nb) * lda + k0 + nb;
    p.lda = p.ldb = p.ldc = lda;
    p.M = p.N = rest;
    p.K = nb;
    p.c_lower = 1;
    p.alpha = -1.0;
    p.beta = 1.0;
    e = gemm_nt<double>(p, 1, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <typename T>
cudaError_t potrf_lower(T* A, int64_t lda, int n, double* logdiag, int* info, double* dtrack,
                        bool zero_upper, cudaStream_t s, bool keep_upper) {
  constexpr int NB = Blk<T>::NB;
  constexpr bool f64 = sizeof(T) == 8;
  const size_t smem_diag = (size_t)(NB * (NB + 1) + 3 * NB) * sizeof(T) + 2 * NB * sizeof(double);
  const size_t smem_trsm = (size_t)(NB * (NB + 1) + 128 * (NB + 1) + NB) * sizeof(T);
  if constexpr (!f64) {
    cudaFuncSetAttribute(potrf_diag_kernel<T, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem_diag);
    cudaFuncSetAttribute(trsm_rows_thread_kernel<T, NB>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_trsm);
  }
  if (zero_upper && n > NB) {
    zero_upper_kernel<T><<<(int)cdiv((int64_t)n * n, 256), 256, 0, s>>>(A, lda, n, NB);
    cudaError_t e0 = launch_status();
    if (e0 != cudaSuccess) return e0;
  }
  for (int k0 = 0; k0 < n; k0 += NB) {
    const int nb = min(NB, n - k0), rest = n - k0 - nb;
    cudaError_t e;
    if constexpr (f64) {
      // its own diagonal supplies the pivots: no float64 track beside it
      e = potrf_block64(A, lda, n, k0, logdiag, info, keep_upper, XSplit{}, s);
      if (e != cudaSuccess) return e;
      if (rest <= 0) break;
    } else {
      potrf_diag_kernel<T, NB><<<1, 512, smem_diag, s>>>(A, lda, n, k0, logdiag, info, dtrack);
      e = launch_status();
      if (e != cudaSuccess) return e;
      if (rest <= 0) break;
      trsm_rows_thread_kernel<T, NB><<<(rest + 127) / 128, 128, smem_trsm, s>>>(A, lda, n, k0);
      e = launch_status();
      if (e != cudaSuccess) return e;
      if (dtrack) {
        diag_track_kernel<T><<<(int)cdiv((int64_t)rest * 32, 256), 256, 0, s>>>(
            A, lda, n, k0 + nb, k0, nb, dtrack);
        e = launch_status();
        if (e != cudaSuccess) return e;
      }
    }
    GemmProb<T> p{};
    p.A = A + (int64_t)(k0 + nb) * lda + k0;
    p.B = p.A;
    p.C = A + (int64_t)(k0 + nb) * lda + k0 + nb;
    p.lda = p.ldb = p.ldc = lda;
    p.M = p.N = rest;
    p.K = nb;
    p.c_lower = 1;
    p.alpha = T(-1);
    p.beta = T(1);
    e = gemm_nt<T>(p, 1, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Columns [o, o + w) of the float64 factor, all rows below included: the left
// half, one product that brings the right half up to date, the right half.
// The products grow with the recursion (K up to n / 2), which is what their
// tensor-core form wants; the right-looking order above rewrites the whole
// trailing matrix once per 64 columns.  They read the digit planes that the
// panel solves wrote: splitting the operands anew cost 5 to 13 us a product.
static cudaError_t potrf_rec(double* A, int64_t lda, int n, int o, int w, double* logdiag,
                             int* info, bool keep_upper, const XSplit& planes, cudaStream_t s) {
  constexpr int NB = Blk<double>::NB;
  if (w <= NB) return potrf_block64(A, lda, n, o, logdiag, info, keep_upper, planes, s);
  int h = NB;
  while (2 * h < w) h *= 2;
  cudaError_t e = potrf_rec(A, lda, n, o, h, logdiag, info, keep_upper, planes, s);
  if (e != cudaSuccess) return e;
  GemmProb<double> p{};
  p.C = A + (int64_t)(o + h) * lda + o + h;
  p.ldc = lda;
  p.M = n - o - h;
  p.N = w - h;
  p.K = h;
  p.c_lower = 1;
  p.alpha = -1.0;
  p.beta = 1.0;
  XSplit x = planes;
  x.row0 = o + h;
  x.col0 = o;
  e = xgemm_run(p, x, x, 1, info, s, true);
  if (e != cudaSuccess) return e;
  return potrf_rec(A, lda, n, o + h, w - h, logdiag, info, keep_upper, planes, s);
}

cudaError_t potrf_lower_x(double* A, int64_t lda, int n, double* logdiag, int* info,
                          bool zero_upper, const XRoom& planes, cudaStream_t s, bool keep_upper) {
  // without room for digit planes every product is a CUDA-core one
  if (planes.bytes < xsplit_bytes(n, n))
    return potrf_lower<double>(A, lda, n, logdiag, info, nullptr, zero_upper, s, keep_upper);
  constexpr int NB = Blk<double>::NB;
  if (zero_upper && n > NB) {
    zero_upper_kernel<double><<<(int)cdiv((int64_t)n * n, 256), 256, 0, s>>>(A, lda, n, NB);
    cudaError_t e = launch_status();
    if (e != cudaSuccess) return e;
  }
  return potrf_rec(A, lda, n, 0, n, logdiag, info, keep_upper, xsplit_at(planes.mem, n, n), s);
}

// ---------------------------------------------------------------------------
// Triangular inverse.  Leaves: every nb x nb diagonal block inverted by
// column-parallel forward substitution (one CTA per block).  Then pairs of
// sibling blocks are merged level by level:
//   [L11 0; L21 L22]^-1 = [M11 0; -M22 L21 M11, M22]
// as two batched NT GEMMs per level.  M (lower) and V = M^T (upper) are both
// kept row-major so that every product reads K-contiguous operands.
// ---------------------------------------------------------------------------
template <typename T, int NB>
__global__ void __launch_bounds__(NB) trtri_diag_kernel(const T* L, int64_t ldl, int n, T* M,
                                                        int64_t ldm, T* V, int64_t ldv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int LD = NB + 1;
  T* Ls = reinterpret_cast<T*>(smem_raw);
  T* Ms = Ls + NB * LD;
  T* ri = Ms + NB * LD;  // 1 / L[i, i], one division per row
  const int k0 = blockIdx.x * NB;
  const int nb = min(NB, n - k0);
  for (int e = threadIdx.x; e < nb * nb; e += blockDim.x) {
    int i = e / nb, j = e % nb;
    Ls[i * LD + j] = (j <= i) ? L[(int64_t)(k0 + i) * ldl + k0 + j] : T(0);
  }
  __syncthreads();
  if (threadIdx.x < nb) ri[threadIdx.x] = T(1) / Ls[threadIdx.x * LD + threadIdx.x];
  __syncthreads();
  const int c = threadIdx.x;
  if (c < nb) {
    for (int i = 0; i < c; ++i) Ms[i * LD + c] = T(0);
    Ms[c * LD + c] = ri[c];
    for (int i = c + 1; i < nb; ++i) {
      T s0 = T(0), s1 = T(0);
      const T* li = Ls + i * LD;
      int k = c;
      for (; k + 2 <= i; k += 2) {
        s0 += li[k] * Ms[k * LD + c];
        s1 += li[k + 1] * Ms[(k + 1) * LD + c];
      }
      if (k < i) s0 += li[k] * Ms[k * LD + c];
      Ms[i * LD + c] = -(s0 + s1) * ri[i];
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nb * nb; e += blockDim.x) {
    int i = e / nb, j = e % nb;
    M[(int64_t)(k0 + i) * ldm + k0 + j] = Ms[i * LD + j];
    V[(int64_t)(k0 + i) * ldv + k0 + j] = Ms[j * LD + i];
  }
}

// The float64 leaf: right-looking forward substitution on the identity, all
// threads on every step (row k final, the rows below lose L[i, k] / L[k, k]
// times it).  One thread per column, as above, is a chain of dependent
// products: 130 us; this one issues each product once: 35 us.
template <int NB>
__global__ void __launch_bounds__(256)
    trtri_diag64_kernel(const double* L, int64_t ldl, int n, double* M, int64_t ldm, double* V,
                        int64_t ldv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int LD = NB + 1;
  double* Ls = reinterpret_cast<double*>(smem_raw);
  double* Ms = Ls + NB * LD;
  double* ri = Ms + NB * LD;  // 1 / L[i, i]
  const int k0 = blockIdx.x * NB;
  const int nb = min(NB, n - k0);
#pragma unroll 8
  for (int u = 0; u < NB * NB / 256; ++u) {
    const int e = threadIdx.x + u * 256, i = e / NB, j = e % NB;
    Ls[i * LD + j] = (i < nb && j <= i) ? L[(int64_t)(k0 + i) * ldl + k0 + j] : 0.0;
    Ms[i * LD + j] = i == j ? 1.0 : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < nb) ri[threadIdx.x] = 1.0 / Ls[threadIdx.x * LD + threadIdx.x];
  __syncthreads();
  for (int e = threadIdx.x; e < NB * NB; e += 256) {
    const int i = e / NB, j = e % NB;
    if (j < i && i < nb) Ls[i * LD + j] *= ri[j];
  }
  __syncthreads();
  for (int k = 0; k + 1 < nb; ++k) {
    const int w = k + 1, total = (nb - w) * w;
    const float inv = 1.f / (float)w;
    for (int e = threadIdx.x; e < total; e += 256) {
      const int r = (int)(((float)e + 0.5f) * inv);  // e / w
      const int i = w + r, c = e - r * w;
      Ms[i * LD + c] = fma(-Ls[i * LD + k], Ms[k * LD + c], Ms[i * LD + c]);
    }
    __syncthreads();
  }
#pragma unroll 4
  for (int u = 0; u < NB * NB / 256; ++u) {
    const int e = threadIdx.x + u * 256, i = e / NB, j = e % NB;
    if (i >= nb || j >= nb) continue;
    M[(int64_t)(k0 + i) * ldm + k0 + j] = Ms[i * LD + j] * ri[i];
    V[(int64_t)(k0 + i) * ldv + k0 + j] = Ms[j * LD + i] * ri[j];
  }
}

template <typename T>
static cudaError_t trtri_merge(const T* L, int64_t ldl, T* M, int64_t ldm, T* V, int64_t ldv,
                               T* scratch, int o, int b, int b2, int count, const XRoom& x,
                               cudaStream_t s) {
  // count pairs starting at offset o, each [b | b2], pair stride 2b.
  const int64_t step = 2 * (int64_t)b;
  GemmProb<T> p{};
  // T_p^T = (L21 M11)^T ; T[i,j] = sum_c L21[i,c] V11[j,c]
  p.A = L + (int64_t)(o + b) * ldl + o;
  p.lda = ldl;
  p.sA = step * ldl + step;
  p.B = V + (int64_t)o * ldv + o;
  p.ldb = ldv;
  p.sB = step * ldv + step;
  p.b_tri = TRI_UPPER;
  p.C = nullptr;
  p.Ct = scratch;
  p.ldct = b2;
  p.sCt = (int64_t)b * b;
  p.M = b2;
  p.N = b;
  p.K = b;
  p.alpha = T(1);
  p.beta = T(0);
  cudaError_t e = gemm_nt_room<T>(p, count, x, s);
  if (e != cudaSuccess) return e;
  // M21 = -M22 T ; M21[i,j] = sum_c M22[i,c] TT[j,c]; also V12 = M21^T
  GemmProb<T> q{};
  q.A = M + (int64_t)(o + b) * ldm + o + b;
  q.lda = ldm;
  q.sA = step * ldm + step;
  q.a_tri = TRI_LOWER;
  q.B = scratch;
  q.ldb = b2;
  q.sB = (int64_t)b * b;
  q.C = M + (int64_t)(o + b) * ldm + o;
  q.ldc = ldm;
  q.sC = step * ldm + step;
  q.Ct = V + (int64_t)o * ldv + o + b;
  q.ldct = ldv;
  q.sCt = step * ldv + step;
  q.M = b2;
  q.N = b;
  q.K = b2;
  q.alpha = T(-1);
  q.beta = T(0);
  return gemm_nt_room<T>(q, count, x, s);
}

template <typename T>
cudaError_t trtri_lower(const T* L, int64_t ldl, int n, T* M, int64_t ldm, T* V, int64_t ldv,
                        T* scratch, const XRoom& x, cudaStream_t s, bool native) {
  constexpr int NB = Blk<T>::NB;
  const size_t smem = (size_t)(2 * NB * (NB + 1) + NB) * sizeof(T);
  const int nblk = (n + NB - 1) / NB;
  if (sizeof(T) == 8 && !native) {
    cudaFuncSetAttribute(trtri_diag64_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem);
    trtri_diag64_kernel<NB><<<nblk, 256, smem, s>>>((const double*)L, ldl, n, (double*)M, ldm,
                                                    (double*)V, ldv);
  } else {
    cudaFuncSetAttribute(trtri_diag_kernel<T, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem);
    trtri_diag_kernel<T, NB><<<nblk, NB, smem, s>>>(L, ldl, n, M, ldm, V, ldv);
  }
  cudaError_t e = launch_status();
  if (e != cudaSuccess) return e;
  for (int b = NB; b < n; b *= 2) {
    // pairs at offsets p*2b whose second block starts before n
    const int npairs = (int)((n - b + 2 * (int64_t)b - 1) / (2 * (int64_t)b));
    int full = 0;
    for (int q = 0; q < npairs; ++q)
      if ((int64_t)q * 2 * b + 2 * b <= n) ++full;
    if (full > 0) {
      e = trtri_merge<T>(L, ldl, M, ldm, V, ldv, scratch, 0, b, b, full, x, s);
      if (e != cudaSuccess) return e;
    }
    if (full < npairs) {
      const int o = full * 2 * b;
      const int b2 = n - o - b;
      e = trtri_merge<T>(L, ldl, M, ldm, V, ldv, scratch + (int64_t)full * b * b, o, b, b2, 1, x,
                         s);
      if (e != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

// ---------------------------------------------------------------------------
// GEMVs, float64 accumulation; one warp per row.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void gemv_tri_kernel(const T* __restrict__ A, int64_t ld, int n, int lower,
                                const double* __restrict__ x, double* __restrict__ y,
                                double alpha, int accumulate) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= n) return;
  const int i = warp;
  const int c0 = lower ? 0 : i, c1 = lower ? i + 1 : n;
  const T* row = A + (int64_t)i * ld;
  double s = 0.0;
  for (int c = c0 + lane; c < c1; c += 32) s += (double)row[c] * x[c];
  s = warp_sum(s);
  if (lane == 0) y[i] = accumulate ? y[i] + alpha * s : alpha * s;
}

template <typename T>
cudaError_t gemv_tri(const T* Tri, int64_t ld, int n, bool lower, const double* x, double* y,
                     double alpha, bool accumulate, cudaStream_t s) {
  const int threads = 256;
  const int blocks = (int)cdiv((int64_t)n * 32, threads);
  gemv_tri_kernel<T><<<blocks, threads, 0, s>>>(Tri, ld, n, lower ? 1 : 0, x, y, alpha,
                                                accumulate ? 1 : 0);
  return launch_status();
}

template <typename T>
__global__ void gemv_dense_kernel(const T* __restrict__ A, int64_t ld, int rows, int cols,
                                  const double* __restrict__ x, double* __restrict__ y) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= rows) return;
  const T* row = A + (int64_t)warp * ld;
  double s = 0.0;
  for (int c = lane; c < cols; c += 32) s += (double)row[c] * x[c];
  s = warp_sum(s);
  if (lane == 0) y[warp] = s;
}

template <typename T>
cudaError_t gemv_dense(const T* A, int64_t ld, int rows, int cols, const double* x, double* y,
                       cudaStream_t s) {
  const int threads = 256;
  const int blocks = (int)cdiv((int64_t)rows * 32, threads);
  gemv_dense_kernel<T><<<blocks, threads, 0, s>>>(A, ld, rows, cols, x, y);
  return launch_status();
}

#define GPK_INST(T)                                                                             \
  template cudaError_t gemm_nt<T>(const GemmProb<T>&, int, cudaStream_t);                       \
  template cudaError_t potrf_lower<T>(T*, int64_t, int, double*, int*, double*, bool,          \
                                      cudaStream_t, bool);                                           \
  template cudaError_t trtri_lower<T>(const T*, int64_t, int, T*, int64_t, T*, int64_t, T*,     \
                                      const XRoom&, cudaStream_t, bool);                        \
  template cudaError_t gemv_tri<T>(const T*, int64_t, int, bool, const double*, double*, double, \
                                   bool, cudaStream_t);                                         \
  template cudaError_t gemv_dense<T>(const T*, int64_t, int, int, const double*, double*,      \
                                     cudaStream_t);
GPK_INST(double)
GPK_INST(float)
#undef GPK_INST

}  // namespace gpk
