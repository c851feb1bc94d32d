// Float64 NT GEMM on the float16 tensor cores by error-free splitting.
//
//   C[i, j] = alpha * sum_k A[i, k] B[j, k] (+ beta C[i, j]),  float64 in and out
//
// Each operand row is scaled by a power of two above its largest element and
// rounded to 55 fraction bits, which seven signed 8-bit digits hold exactly
// (integers in [-128, 128], stored as float16).  The products of digit planes
// p and q are integers; those with p + q = g share one float32 accumulator in
// tensor memory, whose partial sums stay below 2^24 and are therefore exact
// (Ozaki, Ogita, Oishi and Rump, "Error-free transformations of matrix
// multiplication by using fast routines of matrix multiplication", Numerical
// Algorithms 59, 2012).  The accumulators are drained into 64-bit integers and
// the finished sum is rounded to float64 once.  What is left out is the
// rounding of an element below 2^-56 of its row's scale and the digit products
// with p + q > 9, below 2^-62 of the two scales each; a float64 loop over k
// rounds at every step.  Measured largest error over the product of the two
// rows' norms, against extended precision: 1.8e-17 (a float64 library GEMM
// 2.1e-16) at K = 512, 7.4e-18 (1.1e-16) at K = 4000 on normal data, 6e-17
// (1.2e-14) on constant rows at K = 2048.  It is a bound of norms: an element 2^-56 below its row's
// largest is lost, which the objectives' operands bear and a caller's need not
// (gpk_gemm_f64 and gpk_solve_triangular therefore run native float64).
//
// This part has 1.7 float64 multiply-adds per clock and SM (measured: a warp
// instruction every 19 clocks); the 34 float16 products this takes run at
// 4096.
#pragma once
#include <cuda_fp16.h>
#include "gpk_internal.cuh"

namespace gpk {

// One split operand: seven planes of rows x ldk float16 digits and the biased
// exponent of each row's scale (a row holding a NaN or an infinity is marked
// and makes its outputs NaN).
struct XSplit {
  void* planes;
  int* expo;
  int rows, K, ldk;
  int row0 = 0, col0 = 0;  // origin of the operand inside the planes (col0 a multiple of 8)
};
constexpr int XP = 7;        // digit planes
constexpr int XNAN = 0x7ff;  // row exponent of a row with a NaN or an infinity

// The digits of four elements (integers of 55 fraction bits at the row's
// scale), one 8-byte store of float16s per plane.  An integer d in [-128, 128]
// (the top digit of the factor's planes: [-182, 182]) becomes a float16 through the bit pattern of 1536 + d (unit spacing there),
// less 1536: no conversion instruction.
__device__ __forceinline__ void x_store_digits4(long long (&q)[4], __half* dst, int64_t plane) {
  const __half2 base = __halves2half2(__ushort_as_half(0x6600), __ushort_as_half(0x6600));
#pragma unroll
  for (int p = XP - 1; p >= 0; --p) {
    int d[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      d[u] = p ? (int)((q[u] + 128) & 255) - 128 : (int)q[u];
      q[u] = (q[u] - d[u]) >> 8;
    }
    uint32_t w[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t bits = (uint32_t)(0x6600 + d[2 * h]) | ((uint32_t)(0x6600 + d[2 * h + 1]) << 16);
      const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&bits), base);
      w[h] = *reinterpret_cast<const uint32_t*>(&v);
    }
    *reinterpret_cast<uint2*>(dst + p * plane) = make_uint2(w[0], w[1]);
  }
}

// Bytes of the planes and exponents of `rows` rows of K elements.
size_t xsplit_bytes(int64_t rows, int64_t K);
// Places an XSplit in `mem` (256-byte aligned, xsplit_bytes of room).
XSplit xsplit_at(void* mem, int64_t rows, int64_t K);

// Digits of a row-major float64 operand; `tri` zeroes the elements outside the
// triangle (never read).  Batch z covers rows [z * rows, (z + 1) * rows) of
// the split, read from src + z * stride.
cudaError_t xsplit_run(const double* src, int64_t ld, int64_t stride, int rows, int K, int tri,
                       int batch, const XSplit& out, cudaStream_t s);

// The product of two split operands with p's shape, triangles, outputs, alpha
// and beta (p.A, p.B and their strides are not read).  Operand rows of batch z
// start at z * p.M in A and z * p.N in B.  A wait that runs out makes its tile
// NaN and *info -1.  pdl: launched as a programmatic dependent of the kernel
// before it in the stream.  (test_stall: the self-test's.)
cudaError_t xgemm_run(const GemmProb<double>& p, const XSplit& A, const XSplit& B, int batch,
                      int* info, cudaStream_t s, bool pdl = false, long long test_stall = 0);

// gemm_nt<double> with room for the split form: splits A and B (once when B is
// the front of A's rows) and multiplies on the tensor cores where that is the
// faster form, on the CUDA cores otherwise.
cudaError_t gemm_nt_x(const GemmProb<double>& p, int batch, const XRoom& x, cudaStream_t s);

// The same for either type: float32 products always run on the CUDA cores.
template <typename T>
cudaError_t gemm_nt_room(const GemmProb<T>& p, int batch, const XRoom& x, cudaStream_t s) {
  if constexpr (sizeof(T) == 8)
    return gemm_nt_x(p, batch, x, s);
  else
    return gemm_nt<T>(p, batch, s);
}

// Room for every product of an n x n triangular inverse (trtri_lower), 0 for
// sizes whose products all run on the CUDA cores.
size_t xroom_factor_bytes(int64_t n);
// `want` bytes of room, or 0 where a workspace of `base` bytes would grow past
// what the card can hold beside the caller's data.
size_t xroom_fit(size_t base, size_t want);

}  // namespace gpk
