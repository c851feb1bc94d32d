// Split float64 GEMM (xgemm.cuh): digit planes, the tcgen05 kernel, dispatch.
#include <cuda_fp16.h>
#include <climits>
#include "tile_order.cuh"
#include "tc_ptx.cuh"
#include "xgemm.cuh"

namespace gpk {
namespace {

using namespace tc;

constexpr int XG = 8;             // digit-sum groups p + q = 2 .. 9
constexpr int XN = 64;            // output tile columns
constexpr int XK = 32;            // K elements per stage (64-byte rows, 64B swizzle)
constexpr int XSTAGES = 2;
constexpr int XA_PLANE = BM * XK * 2, XB_PLANE = XN * XK * 2;
constexpr int XSTAGE_BYTES = XP * (XA_PLANE + XB_PLANE);
constexpr int XTHREADS = 320;     // w0 TMA, w1 MMA + TMEM, w2..w9 epilogue
constexpr int XEPI_WARPS = 8, XEPI_THREADS = XEPI_WARPS * 32;
constexpr int XHC = XN / 2;       // accumulator columns of one epilogue thread
constexpr int XTLD = XN + 1;      // staged tile row stride (doubles)
// Multiply-adds from which a product whose operands are split first beats the
// CUDA-core tiles: 7e6 (192^3) 39 us against 23, 8.4e6 34 against 45 (512 x 128
// x 128) and 63 against 53 (128 x 128 x 512), 1.7e7 (256^3) 43 against 86.
// Marginal likelihood with the line at 5e5 / 8e6 / 1.6e7 / 3.2e7: n = 384
// 860 / 757 / 745 / 816 us, n = 1024 1979 / 1930 / 1955 / 1955 us.
constexpr double XMIN_MULTS = 8e6;
constexpr int XMAX_K = 1 << 18;   // the drained 64-bit sums stay below K * 2^41

// K slices summed by one accumulator before it is drained: a group holds up to
// 7 products of digits up to 128 x 128, two of them with a top digit, which in
// the factor's planes reaches 182: (4 * 32) (5 * 128^2 + 2 * 182 * 128) < 2^24.
constexpr int XPER = 4;

struct XCtl {
  uint64_t full[XSTAGES], empty[XSTAGES];
  uint64_t tfull[XG], tempty[XG];
  uint64_t mdone;
  uint32_t tmem;
  int abort_flag;
  int eb[XN];  // column row-exponents of this tile
};

struct XParams {
  int M, N, K, a_tri, b_tri, c_lower, tiles_m, tiles_n;
  int a_row0, a_col0, b_row0, b_col0;  // origins inside the tensor maps
  const int* ea;
  const int* eb;
  double *C, *Ct;
  int64_t ldc, ldct, sC, sCt;
  double alpha, beta;
  int alpha_mode, beta_mode;  // 0: general; 1: alpha 1 / beta 0; 2: alpha -1 / beta 1
  int* info;                  // a wait that ran out makes it -1 (may be null)
  long long test_stall;       // self-test (0: off): cycles that the MMA warp first waits on a
                              // barrier nothing arrives at
};

// (hi * 2^32 + lo) * 2^e rounded to float64, in integer arithmetic (this
// part's float64 units would take longer than the products of a short K): a
// 64-bit head and a 32-bit tail, |hi| < 2^58.
__device__ __forceinline__ double x_round(long long hi, long long lo, int e) {
  long long h = hi + (lo >> 32);
  unsigned t = (unsigned)lo;
  const unsigned long long sign = (unsigned long long)h & 0x8000000000000000ULL;
  if (h < 0) {  // negate the pair
    h = ~h + (t == 0);
    t = 0u - t;
  }
  if (h == 0) {  // below 2^32 units: the tail is the head
    if (t == 0) return 0.0;
    h = t;
    t = 0;
    e -= 32;
  }
  const int lz = __clzll(h);
  unsigned long long top = (unsigned long long)h << lz;
  unsigned rest = 0;
  if (lz >= 32) {
    top |= (unsigned long long)t << (lz - 32);
  } else {
    top |= ((unsigned long long)t << lz) >> 32;
    rest = t << lz;
  }
  unsigned long long r = top >> 11;
  const unsigned rem = (unsigned)top & 0x7ff;
  if (rem > 0x400 || (rem == 0x400 && (rest != 0 || (r & 1)))) ++r;
  const int biased = 63 + 32 - lz + e + 1023;
  if (biased >= 1 && biased <= 2046)
    return __longlong_as_double((long long)(sign | (((unsigned long long)(biased - 1) << 52) + r)));
  const double v = scalbn((double)r, 63 + 32 - lz + e - 52);
  return sign ? -v : v;
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int w,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(w), "r"(smem_u32(bar))
      : "memory");
}

// One 128 x 64 output tile per CTA: all seven planes of both operands of a
// 32-wide K slice are staged together (84 KB, 2 stages), so each staged byte
// feeds up to seven products; the eight group accumulators fill the 512 TMEM
// columns.  The drain of a group overlaps the MMAs of the other seven.
__global__ void __launch_bounds__(XTHREADS, 1)
    xgemm_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
                 const __grid_constant__ XParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  XCtl* ctl = reinterpret_cast<XCtl*>(ring + XSTAGES * XSTAGE_BYTES);
  double* otile = reinterpret_cast<double*>(ring);  // output tile, reuses the operand ring
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int z = blockIdx.z;
  int I, J;
  tile_of(blockIdx.x, p.c_lower, p.tiles_m, p.tiles_n, XN, I, J);
  const int i0 = I * BM, j0 = J * XN;
  int klo = 0, khi = p.K;
  if (p.a_tri == TRI_LOWER) khi = min(khi, i0 + BM);
  if (p.a_tri == TRI_UPPER) klo = max(klo, i0);
  if (p.b_tri == TRI_LOWER) khi = min(khi, j0 + XN);
  if (p.b_tri == TRI_UPPER) klo = max(klo, j0);
  klo = (klo / XK) * XK;
  const int nk = khi > klo ? (khi - klo + XK - 1) / XK : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < XSTAGES; ++s) {
      mbar_init(&ctl->full[s], 1);
      mbar_init(&ctl->empty[s], 1);
    }
    for (int g = 0; g < XG; ++g) {
      mbar_init(&ctl->tfull[g], 1);
      mbar_init(&ctl->tempty[g], XEPI_WARPS);
    }
    mbar_init(&ctl->mdone, 1);
    ctl->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&ctl->tmem)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_trigger();
  const uint32_t tmem = ctl->tmem;
  volatile int* abort_flag = &ctl->abort_flag;

  if (warp == 0) {
    if (lane == 0) {
      int issued = 0;
      for (int kc = 0; kc < nk; ++kc) {
        const int s = kc % XSTAGES;
        if (kc >= XSTAGES &&
            !mbar_wait(&ctl->empty[s], ((kc / XSTAGES) - 1) & 1, abort_flag, nullptr, kWaitCycles))
          break;
        uint8_t* st = ring + s * XSTAGE_BYTES;
        mbar_expect_tx(&ctl->full[s], XSTAGE_BYTES);
        tma_load_3d(st, &ta, p.a_col0 + klo + kc * XK, p.a_row0 + z * p.M + i0, 0, &ctl->full[s]);
        tma_load_3d(st + XP * XA_PLANE, &tb, p.b_col0 + klo + kc * XK, p.b_row0 + z * p.N + j0, 0,
                    &ctl->full[s]);
        ++issued;
      }
      for (int kc = max(0, issued - XSTAGES); kc < issued; ++kc)
        mbar_wait_own(&ctl->full[kc % XSTAGES], (kc / XSTAGES) & 1, kWaitCycles);
    }
  } else if (warp == 1) {
    // The whole warp runs this loop and an elected lane issues: with the
    // stage unrolled and the tensor memory base broadcast, the descriptors
    // stay in uniform registers.  From inside a one-lane branch the moves into
    // them took longer than the MMAs (4096^3: 4.8 ms; this form 3.7 ms).
    constexpr uint32_t idesc = idesc_f16(BM, XN);
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const bool leader = elect_one();
    bool ok = true, issued_mma = false;
    if (p.test_stall)
      ok = __all_sync(0xffffffffu, mbar_wait(&ctl->mdone, 0, abort_flag, nullptr, p.test_stall));
    auto chunk = [&](int kc, const int s) {
      ok = __all_sync(0xffffffffu, mbar_wait(&ctl->full[s], (kc / XSTAGES) & 1, abort_flag,
                                             nullptr, kWaitCycles));
      if (!ok) return;
      tc_fence_after();
      const uint32_t sb = smem_u32(ring) + (uint32_t)s * XSTAGE_BYTES;
      const uint64_t da = sdesc<64>(sb), db = sdesc<64>(sb + XP * XA_PLANE);
      // two groups at a time, their MMAs alternating; a group's accumulator is
      // waited for only when its turn comes
      const bool first = kc % XPER == 0, last = kc % XPER == XPER - 1 || kc == nk - 1;
#pragma unroll
      for (int pr = 0; pr < XG / 2; ++pr) {
        if (first && kc > 0) {
          const uint32_t ph = ((kc / XPER) - 1) & 1;
          ok = mbar_wait(&ctl->tempty[2 * pr], ph, abort_flag, nullptr, kWaitCycles) &&
               mbar_wait(&ctl->tempty[2 * pr + 1], ph, abort_flag, nullptr, kWaitCycles);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) return;
          tc_fence_after();
        }
        issued_mma = true;
        if (!leader) continue;
#pragma unroll
        for (int t = 0; t < 2 * XP; ++t) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            // group gi (planes counted from 0): pa + pb = gi, both in [0, XP)
            const int gi = 2 * pr + h, lo = gi < XP ? 0 : gi - XP + 1, hi = gi < XP ? gi : XP - 1;
            if (t >= 2 * (hi - lo + 1)) continue;
            const int pa = lo + t / 2, pb = gi - pa, k4 = t & 1;
            mma_f16(tm + (uint32_t)(gi * XN), da + (uint64_t)(pa * (XA_PLANE >> 4) + 2 * k4),
                    db + (uint64_t)(pb * (XB_PLANE >> 4) + 2 * k4), idesc,
                    t == 0 && first ? 0u : 1u);
          }
        }
        if (last) {
          mma_commit(&ctl->tfull[2 * pr]);
          mma_commit(&ctl->tfull[2 * pr + 1]);
        }
      }
      if (leader) mma_commit(&ctl->empty[s]);
    };
    static_assert(XSTAGES * XSTAGE_BYTES >= BM * (XTLD + XN) * 8, "both output tiles fit the ring");
    static_assert(XSTAGES == 2, "the stage is a compile-time constant of each call below");
    for (int kc = 0; kc < nk && ok; kc += 2) {
      chunk(kc, 0);
      if (ok && kc + 1 < nk) chunk(kc + 1, 1);
    }
    if (!ok && issued_mma) {  // MMAs already issued finish before TMEM is freed
      if (leader) mma_commit(&ctl->mdone);
      mbar_wait_own(&ctl->mdone, 0, kWaitCycles);
    }
    __syncwarp();
  } else {
    const int q = warp & 3, ew = warp - 2;
    const int hcol = (ew >> 2) * XHC;
    const int r = q * 32 + lane, gi0 = i0 + r;
    const int et = threadIdx.x - 64;
    if (et < XN) ctl->eb[et] = j0 + et < p.N ? p.eb[(int64_t)z * p.N + j0 + et] : 1;
    const int ea = gi0 < p.M ? p.ea[(int64_t)z * p.M + gi0] : 1;
    long long hi[XHC], lo[XHC];
#pragma unroll
    for (int c = 0; c < XHC; ++c) hi[c] = lo[c] = 0;
    bool have = true;
    for (int kc = 0; kc < nk && have; ++kc) {
#pragma unroll
      for (int g = 0; g < XG; ++g) {
        constexpr int per = XPER;
        if (!have || !(kc % per == per - 1 || kc == nk - 1)) continue;
        have = __all_sync(0xffffffffu, mbar_wait(&ctl->tfull[g], (kc / per) & 1, abort_flag,
                                                 nullptr, kWaitCycles));
        if (!have) continue;
        tc_fence_after();
        const uint32_t tg = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(g * XN + hcol);
        auto take = [&](const uint32_t (&v)[16], int c0) {
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const int d = __float2int_rn(__uint_as_float(v[c]));
            if (g < 4)
              hi[c0 + c] += (long long)d * (1 << (8 * (g < 4 ? 3 - g : 0)));
            else
              lo[c0 + c] += (long long)d * (1 << (8 * (g < 4 ? 0 : 7 - g)));
          }
        };
        uint32_t v0[16];
        tmem_ld16_nowait(tg, v0);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        take(v0, 0);
        uint32_t v1[16];
        tmem_ld16_nowait(tg + 16, v1);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&ctl->tempty[g]))
                       : "memory");
        take(v1, 16);
      }
    }
    const double nan = __longlong_as_double(0x7ff8000000000000ULL);
    const double beta = p.beta;
    const int bm = p.beta_mode;
    double* C = p.C ? p.C + (int64_t)z * p.sC : nullptr;
    double* Ct = p.Ct ? p.Ct + (int64_t)z * p.sCt : nullptr;
    auto inside = [&](int rr, int cc) {
      const int gi = i0 + rr, gj = j0 + cc;
      return gi < p.M && gj < p.N && !(p.c_lower && gj > gi);
    };
    asm volatile("bar.sync 1, %0;" ::"r"(XEPI_THREADS) : "memory");  // ring free, eb staged
    // A wait that ran out (its flag is set ahead of the barrier, and with every
    // sum drained no wait is left to run out): the tile is NaN through alpha, for
    // copies still under way may land on what is staged below.
    const bool failed = *abort_flag != 0;
    const int am = failed ? 0 : p.alpha_mode;
    const double alpha = failed ? nan : p.alpha;
    if (failed && et == 0 && p.info) atomicMin(p.info, -1);
    // the old C tile comes into the other half of the ring while the sums are
    // rounded (2.5 us of loads otherwise)
    double* ctile = otile + BM * XTLD;
    if (C && bm != 1) {
#pragma unroll 4
      for (int e = et; e < BM * XN; e += XEPI_THREADS) {
        const int rr = e / XN, cc = e % XN;
        if (inside(rr, cc))
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(ctile + e)),
                       "l"(C + (int64_t)(i0 + rr) * p.ldc + j0 + cc)
                       : "memory");
      }
    }
#pragma unroll
    for (int c = 0; c < XHC; ++c) {
      const int eb = ctl->eb[hcol + c];
      const bool bad = ea == XNAN || eb == XNAN;
      otile[r * XTLD + hcol + c] = bad ? nan : x_round(hi[c], lo[c], ea + eb - 2 * 1022 - 70);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    asm volatile("bar.sync 1, %0;" ::"r"(XEPI_THREADS) : "memory");
    // integer modes: a float64 comparison per element runs at the float64 rate
    auto scaled = [&](double v) {
      if (am == 1) return v;
      if (am == 2)
        return __longlong_as_double(__double_as_longlong(v) ^ (long long)0x8000000000000000ULL);
      return alpha * v;
    };
    if (C) {
#pragma unroll 8
      for (int e = et; e < BM * XN; e += XEPI_THREADS) {
        const int rr = e / XN, cc = e % XN;
        if (!inside(rr, cc)) continue;
        double v = scaled(otile[rr * XTLD + cc]);
        if (bm == 2)
          v += ctile[e];
        else if (bm == 0)
          v = fma(beta, ctile[e], v);
        C[(int64_t)(i0 + rr) * p.ldc + j0 + cc] = v;
      }
    }
    if (Ct) {
      for (int e = et; e < BM * XN; e += XEPI_THREADS) {
        const int cc = e / BM, rr = e % BM;
        if (inside(rr, cc)) Ct[(int64_t)(j0 + cc) * p.ldct + i0 + rr] = scaled(otile[rr * XTLD + cc]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512)
                 : "memory");
  }
}

// ---------------------------------------------------------------------------
// Digit planes
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool x_outside(int tri, int r, int c) {
  return (tri == TRI_LOWER && c > r) || (tri == TRI_UPPER && c < r);
}
__device__ __forceinline__ int x_expo(double a) {
  const int x = (int)((__double_as_longlong(a) >> 52) & 0x7ff);
  return x > 1 ? x : 1;
}

// The digits of four float64 elements at row exponent X.
__device__ __forceinline__ void x_digits4(const double (&a)[4], int X, __half* dst, int64_t plane) {
  long long q[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(a[u]);
    const int xb = (int)((b >> 52) & 0x7ff), s = X - (xb > 1 ? xb : 1);
    const unsigned long long m = (b & 0xfffffffffffffULL) | (xb ? 1ULL << 52 : 0ULL);
    const long long v = s <= 2 ? (long long)(m << (2 - s))
                               : (s < 57 ? (long long)((m + (1ULL << (s - 3))) >> (s - 2)) : 0LL);
    q[u] = (long long)b < 0 ? -v : v;
  }
  x_store_digits4(q, dst, plane);
}

// One warp per row (and, CHUNKED, per XCHUNK columns of it): the row's largest
// exponent, then its digits.  Long rows are cut into chunks so that a few of
// them still fill the chip; their exponents come from xexpo_kernel.
constexpr int XCHUNK = 1024;
template <bool CHUNKED>
__global__ void __launch_bounds__(256)
    xsplit_kernel(const double* __restrict__ src, int64_t ld, int64_t stride, int rows, int K,
                  int ldk, int tri, int total, __half* __restrict__ planes,
                  int* __restrict__ expo) {
  pdl_wait();
  pdl_trigger();
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= total) return;
  const int z = row / rows, r = row % rows;
  const double* a = src + z * stride + (int64_t)r * ld;
  const int c0 = CHUNKED ? blockIdx.y * XCHUNK : 0, c1 = CHUNKED ? min(ldk, c0 + XCHUNK) : ldk;
  int X = 1;
  if (CHUNKED) {
    X = expo[row];
  } else {
    for (int c = lane; c < K; c += 32)
      if (!x_outside(tri, r, c)) X = max(X, x_expo(a[c]));
    X = __reduce_max_sync(0xffffffffu, X);
    if (lane == 0) expo[row] = X;
  }
  const int64_t plane = (int64_t)total * ldk;
  __half* out = planes + (int64_t)row * ldk;
  for (int c = c0 + 4 * lane; c < c1; c += 128) {
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      v[u] = c + u < K && X != XNAN && !x_outside(tri, r, c + u) ? a[c + u] : 0.0;
    x_digits4(v, X, out + c, plane);
  }
}

__global__ void __launch_bounds__(256)
    xexpo_kernel(const double* __restrict__ src, int64_t ld, int64_t stride, int rows, int K,
                 int tri, int total, int* __restrict__ expo) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= total) return;
  const int z = row / rows, r = row % rows;
  const double* a = src + z * stride + (int64_t)r * ld;
  const int c0 = blockIdx.y * XCHUNK, c1 = min(K, c0 + XCHUNK);
  int X = 1;
#pragma unroll 4
  for (int c = c0 + lane; c < c1; c += 32)
    if (!x_outside(tri, r, c)) X = max(X, x_expo(a[c]));
  X = __reduce_max_sync(0xffffffffu, X);
  if (lane == 0) atomicMax(&expo[row], X);
}

bool x_map(CUtensorMap* m, const XSplit& x, int box_rows) {
  const cuuint64_t dims[3] = {(cuuint64_t)x.ldk, (cuuint64_t)x.rows, (cuuint64_t)XP};
  const cuuint64_t strides[2] = {(cuuint64_t)x.ldk * 2, (cuuint64_t)x.ldk * 2 * x.rows};
  const cuuint32_t box[3] = {(cuuint32_t)XK, (cuuint32_t)box_rows, (cuuint32_t)XP};
  return tc_encode_map(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, x.planes, dims, strides, box,
                       CU_TENSOR_MAP_SWIZZLE_64B);
}

}  // namespace

static int x_ldk(int64_t K) { return (int)((K + XK - 1) / XK * XK); }

size_t xsplit_bytes(int64_t rows, int64_t K) {
  return (((size_t)rows * x_ldk(K) * 2 * XP + 255) & ~size_t(255)) +
         (((size_t)rows * sizeof(int) + 255) & ~size_t(255));
}

XSplit xsplit_at(void* mem, int64_t rows, int64_t K) {
  XSplit x;
  x.rows = (int)rows;
  x.K = (int)K;
  x.ldk = x_ldk(K);
  x.planes = mem;
  x.expo = reinterpret_cast<int*>(static_cast<char*>(mem) +
                                  (((size_t)rows * x.ldk * 2 * XP + 255) & ~size_t(255)));
  return x;
}

cudaError_t xsplit_run(const double* src, int64_t ld, int64_t stride, int rows, int K, int tri,
                       int batch, const XSplit& out, cudaStream_t s) {
  const int total = rows * batch;
  if (total <= 0 || K <= 0) return cudaSuccess;
  const unsigned gx = (unsigned)cdiv(total, 8);
  __half* planes = static_cast<__half*>(out.planes);
  // 1024 columns: below, one pass per row has both reads in L1; above, rows
  // alone are too few warps
  if (out.ldk <= XCHUNK) {
    xsplit_kernel<false><<<gx, 256, 0, s>>>(src, ld, stride, rows, K, out.ldk, tri, total, planes,
                                            out.expo);
    return launch_status();
  }
  const dim3 grid(gx, (unsigned)cdiv(out.ldk, XCHUNK));
  cudaError_t e = cudaMemsetAsync(out.expo, 0, (size_t)total * sizeof(int), s);
  if (e != cudaSuccess) return e;
  xexpo_kernel<<<grid, 256, 0, s>>>(src, ld, stride, rows, K, tri, total, out.expo);
  e = launch_status();
  if (e != cudaSuccess) return e;
  xsplit_kernel<true><<<grid, 256, 0, s>>>(src, ld, stride, rows, K, out.ldk, tri, total, planes,
                                           out.expo);
  return launch_status();
}

cudaError_t xgemm_run(const GemmProb<double>& p, const XSplit& A, const XSplit& B, int batch,
                      int* info, cudaStream_t s, bool pdl, long long test_stall) {
  if (p.M <= 0 || p.N <= 0 || batch <= 0) return cudaSuccess;
  if (p.K > XMAX_K) return cudaErrorInvalidValue;
  CUtensorMap ma, mb;
  if (!x_map(&ma, A, BM) || !x_map(&mb, B, XN)) return cudaErrorInvalidValue;
  XParams q{};
  q.M = p.M;
  q.N = p.N;
  q.K = p.K;
  q.a_tri = p.a_tri;
  q.b_tri = p.b_tri;
  q.c_lower = p.c_lower;
  q.tiles_m = (p.M + BM - 1) / BM;
  q.tiles_n = (p.N + XN - 1) / XN;
  q.a_row0 = A.row0;
  q.a_col0 = A.col0;
  q.b_row0 = B.row0;
  q.b_col0 = B.col0;
  q.ea = A.expo + A.row0;
  q.eb = B.expo + B.row0;
  q.C = p.C;
  q.Ct = p.Ct;
  q.ldc = p.ldc;
  q.ldct = p.ldct;
  q.sC = p.sC;
  q.sCt = p.sCt;
  q.alpha = p.alpha;
  q.beta = p.beta;
  q.alpha_mode = p.alpha == 1.0 ? 1 : p.alpha == -1.0 ? 2 : 0;
  q.beta_mode = p.beta == 0.0 ? 1 : p.beta == 1.0 ? 2 : 0;
  q.info = info;
  q.test_stall = test_stall;
  const size_t smem = 1024 + (size_t)XSTAGES * XSTAGE_BYTES + sizeof(XCtl);
  cudaFuncSetAttribute(xgemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const PdlAttr attr(pdl);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tile_count(q.c_lower, q.tiles_m, q.tiles_n, XN), 1, batch);
  cfg.blockDim = dim3(XTHREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = const_cast<cudaLaunchAttribute*>(attr.a);
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, xgemm_kernel, ma, mb, q);
  return launch_status();
}

cudaError_t gemm_nt_x(const GemmProb<double>& p, int batch, const XRoom& x, cudaStream_t s) {
  if (p.M <= 0 || p.N <= 0 || batch <= 0) return cudaSuccess;
  // B's rows are the first of A's (a symmetric update): one split serves both
  const bool front = p.A == p.B && p.lda == p.ldb && p.a_tri == p.b_tri && p.N <= p.M &&
                     (batch == 1 || (p.N == p.M && p.sA == p.sB));
  const size_t na = xsplit_bytes((int64_t)p.M * batch, p.K);
  const size_t nb = front ? 0 : xsplit_bytes((int64_t)p.N * batch, p.K);
  const double outs = (double)p.M * p.N - (p.c_lower ? 0.5 * p.N * p.N : 0.0);
  const double mults = outs * p.K * batch;
  if (!x.mem || na + nb > x.bytes || p.K > XMAX_K || p.K < XK || mults < XMIN_MULTS ||
      (int64_t)p.M * batch > INT_MAX / 2 || (int64_t)p.N * batch > INT_MAX / 2)
    return gemm_nt<double>(p, batch, s);
  const XSplit A = xsplit_at(x.mem, (int64_t)p.M * batch, p.K);
  cudaError_t e = xsplit_run(p.A, p.lda, p.sA, p.M, p.K, p.a_tri, batch, A, s);
  if (e != cudaSuccess) return e;
  XSplit B = A;
  if (!front) {
    B = xsplit_at(static_cast<char*>(x.mem) + na, (int64_t)p.N * batch, p.K);
    e = xsplit_run(p.B, p.ldb, p.sB, p.N, p.K, p.b_tri, batch, B, s);
    if (e != cudaSuccess) return e;
  }
  return xgemm_run(p, A, B, batch, x.info, s, true);  // follows a split kernel
}

size_t xroom_factor_bytes(int64_t n) {
  if (n <= 128) return 0;  // at most two blocks
  int64_t b = 64;
  while (2 * b < n) b *= 2;
  // a product of the factor or of a merge level reads at most n rows in all, of
  // at most b elements each
  return xsplit_bytes(n + 64, b) + 512;
}

size_t xroom_fit(size_t base, size_t want) {
  return base + want <= ((size_t)190 << 30) ? want : 0;
}

}  // namespace gpk

// ---------------------------------------------------------------------------
// Self-test of the bounded waits: one product whose MMA warp waits 20M cycles
// on a barrier that nothing arrives on.
// ---------------------------------------------------------------------------
using namespace gpk;

constexpr int kSelfTestN = 256, kSelfTestK = 128;

extern "C" size_t gpk_selftest_split_wait_timeout_workspace_bytes(void) {
  return (size_t)kSelfTestN * kSelfTestK * sizeof(double) + 512 +
         xsplit_bytes(kSelfTestN, kSelfTestK);
}

extern "C" gpk_status gpk_selftest_split_wait_timeout(double* C, int* info, void* workspace,
                                                      size_t workspace_bytes,
                                                      cudaStream_t stream) {
  if (!C || !info || !workspace ||
      workspace_bytes < gpk_selftest_split_wait_timeout_workspace_bytes())
    return GPK_ERR_BAD_ARG;
  const uintptr_t base = (reinterpret_cast<uintptr_t>(workspace) + 255) & ~uintptr_t(255);
  double* A = reinterpret_cast<double*>(base);
  const size_t bytes = (size_t)kSelfTestN * kSelfTestK * sizeof(double);
  GPK_CUDA_TRY(cudaMemsetAsync(A, 0, bytes, stream));
  const XSplit x = xsplit_at(reinterpret_cast<void*>(base + bytes), kSelfTestN, kSelfTestK);
  GPK_CUDA_TRY(xsplit_run(A, kSelfTestK, 0, kSelfTestN, kSelfTestK, TRI_NONE, 1, x, stream));
  GemmProb<double> p{};
  p.C = C;
  p.ldc = kSelfTestN;
  p.M = p.N = kSelfTestN;
  p.K = kSelfTestK;
  p.alpha = 1.0;
  GPK_CUDA_TRY(xgemm_run(p, x, x, 1, info, stream, false, 20000000LL));
  return GPK_OK;
}
