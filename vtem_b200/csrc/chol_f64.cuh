// Float64 tile Cholesky of one or two systems (chol_f64.cu).
#pragma once
#include <cstdint>

#include "common.cuh"

namespace vtb {

struct Chol64System {
    double* A;           // column-major, lower factor in place; 16-byte aligned columns are the fast form
    int64_t ld;
    int K;
    double* x;           // right-hand side; y = L^-1 b after chol64_factor
    void* work;          // chol64_bytes(K), 256-byte aligned
    int32_t* status;     // 0, 1 (pivot), 2 (spread * rcond >= 1), 3 (a wait ran out) or -1 (chol64_solve's check)
    double* pivots;      // (min, max) squared pivots, may be null
    double rcond;
};

constexpr int kChol64Phases = 6;      // at most

int64_t chol64_bytes(int K);
int chol64_factor(const Chol64System* systems, int n, cudaStream_t s);   // n = 1 or 2, factorised side by side
// x <- the triangular solves one after another, forward and backward in turn, `phases` of them;
// check: status 0 becomes -1 where a diagonal tile is ill conditioned
int chol64_solve(const Chol64System& system, bool backward_first, int phases, bool check, cudaStream_t s);

}  // namespace vtb
