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
// rounds at every step.  Measured largest error over |a_i| |b_j|, against
// extended precision: 4.1e-17 (a float64 library GEMM 2.1e-16) at K = 512,
// 2.5e-17 (1.1e-16) at K = 4000 on normal data, 6e-17 (1.2e-14) on constant
// rows at K = 2048.
//
// This part has 1.7 float64 multiply-adds per clock and SM (measured: a warp
// instruction every 19 clocks); the 34 float16 products this takes run at
// 4096.
#pragma once
#include "gpk_internal.cuh"

namespace gpk {

// One split operand: seven planes of rows x ldk float16 digits and the biased
// exponent of each row's scale (a row holding a NaN or an infinity is marked
// and makes its outputs NaN).
struct XSplit {
  void* planes;
  int* expo;
  int rows, K, ldk;
};

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
// start at z * p.M in A and z * p.N in B.
cudaError_t xgemm_run(const GemmProb<double>& p, const XSplit& A, const XSplit& B, int batch,
                      cudaStream_t s);

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

// Room for every product of an n x n factorisation and inverse (potrf_lower_x,
// trtri_lower), 0 for sizes whose products all run on the CUDA cores.
size_t xroom_factor_bytes(int64_t n);
// `want` bytes of room, or 0 where a workspace of `base` bytes would grow past
// what the card can hold beside the caller's data.
size_t xroom_fit(size_t base, size_t want);

}  // namespace gpk
