// Float64 Kronecker Gram of the coefficient-space decoder (kron_gram.cu).
#pragma once
#include "common.cuh"

namespace vtb {

// M[(s,m),(s',m')] = sum_n d[n][s] conj(d[n][s']) W_n[m][m'] (N neurons, Ks
// spatial indices, Hermitian Kt x Kt W_n), M column-major, Hermitian, full.
int kron_gram_f64(const double2* d, int N, int Ks, const double2* Wn, int Kt, double2* M, int64_t ldm, cudaStream_t s);

}  // namespace vtb
