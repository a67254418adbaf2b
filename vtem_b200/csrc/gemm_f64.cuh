// FP64 GEMM on the float64 tensor-core path, used by the plain float64
// path: C[m, n] = alpha * sum_k A(m, k) B(n, k) + beta * C[m, n]
// with arbitrary element strides, so one kernel serves the RF projection
// (video x RFs), the synthesis (H x spatial functions) and the small
// cross-weight products.
#pragma once
#include "common.cuh"

namespace vtb {

struct GemmF64Args {
    int M, N, K;
    const double* A;
    int64_t a_m, a_k;   // strides of A(m, k)
    const double* B;
    int64_t b_n, b_k;   // strides of B(n, k)
    double* C;
    int64_t c_m, c_n;   // strides of C(m, n)
    double alpha, beta;
};

// C(m, n) = alpha sum_k A(m, k) B(n, k) + beta C(m, n) on `s` (gemm_f64.cu).
int gemm_f64(const GemmF64Args& p, cudaStream_t s);

// C = A^2 + beta A for symmetric A (N x N, rows of lda doubles), C exactly
// symmetric: the tiles of one triangle computed, written to both (gemm_f64.cu).
int square_f64(int N, const double* A, int64_t lda, double beta, double* C, int64_t ldc, cudaStream_t s);

}  // namespace vtb
