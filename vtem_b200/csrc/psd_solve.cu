// Pseudoinverse solve of a positive semidefinite system of low rank.
//
// The plain decoder's Gram G (n x n) has the rank of the Dirichlet space, a
// fraction of n in any window that samples it well, and its eigenvalues below
// that rank are rounding noise.  solve_eq_sym's eigendecomposition of G
// (solve.cu) then spends 4/3 n^3 operations, most of them in a chain of n
// matrix-vector products, to find a null space it drops.  Here instead
//   G = L L^T,  L n x r,  by Cholesky with pivoting down to rounding noise,
//   B = L^T L (r x r, the nonzero eigenvalues of G),
//   c = G L B^-3 L^T q,  refined: c += L B^-3 L^T (G (q - G c)),
// which is the reference's truncated pseudoinverse exactly when the rule
// s > rcond * s_0 drops the noise and keeps the rest.  Both are tested.
// B - rcond * |B|_inf I has a Cholesky factorisation: every eigenvalue of B
// passes the rule.  The remainder E = G - L L^T is below it: by its trace, which
// decides for a semidefinite G, and, as an indefinite one can hide from its
// diagonal, by |E v| for kPcProbes pseudo-random vectors v.  That part is
// probabilistic: an eigenvalue e of E above the rule passes when its eigenvector
// is nearly orthogonal to every v, |<v, u>| below 0.05 rule / e, under one
// chance in 25 a vector.  The vectors' magnitudes vary and their seed is taken
// from G, so that no pattern of entries cancels in all of them (signs alone miss
// a four-cycle of +-a on rows of zero diagonal).  Anything else is left to the
// eigendecomposition: *accepted = 0, G untouched.
//
// In exact arithmetic G L B^-3 L^T = L B^-2 L^T = G^+.  The range of the computed
// L is off that of G by about sqrt(n k) eps |diag G| / s_r (the sums of k products
// behind every column), several times the error of an eigenvector.  A product
// with G returns the solution to G's own range, and takes the part of the
// residual outside it away, at an error of eps |G| each.  One refinement does
// until the condition number nears 1e7; more are taken while the last was above
// kPcConverged, and a solve that does not settle is refused.  Relative error of c
// against the known solution, for the spectra 1..1/cond of n = 1900, r = 261 and a q
// outside the range: by L B^-2 L^T refined with q - G c 1.3e-13 at cond = 1e2 and
// 1.1e-9 at 1e6, here 8.6e-15 and 5.4e-11, by the eigendecomposition 9.7e-15 and
// 1.4e-10.  It costs 0.1 ms of 1.0 at that size, 2 of 21 at n = 24000.
//
// Pivots are taken kPcB at a time: candidates are the largest remaining
// diagonal entries of kPcB strided groups of indices, their columns of the
// Schur complement come from one product (C = G(:, cand) - L L(cand, :)^T, the
// float64 GEMM), and a pivoted Cholesky of the candidates' own block accepts
// those that stay above a hundredth of the largest diagonal (for a
// semidefinite matrix any order of such pivots is stable: entries of L are
// bounded by the square root of the diagonal).  So the chain is one of
// r / kPcB small launches instead of r global searches.  k, the columns so
// far, lives on the device (accepted counts vary); the product runs over the
// host's upper bound, the columns beyond k being zero.
//
// B and the shifted B are factorised side by side by the float64 tile Cholesky
// and B^-3 applied in one launch of its triangular solves (two library
// factorisations and eight library solves took 447 us of 1002 at r = 261).
// Measured at n = 1900, r = 261 (the small configuration): 21.0 ms with the
// eigendecomposition, 1.0 ms here; n = 24000, r = 1921: 6.9 s and 21 ms.  What a
// refusal costs: a matrix of full rank whose spectrum is flat, or an indefinite
// one, goes after the second step (by the trace its columns have taken), 0.1 ms
// of 3.3 at n = 300 and of 28 at n = 2000; one whose eigenvalues decay over five
// decades only at n/2 columns, 0.4 of 3.3 and 2.0 of 27.5.
#include <algorithm>
#include <cmath>
#include <cstddef>

#include "chol_f64.cuh"
#include "common.cuh"
#include "gemm_f64.cuh"

namespace vtb {

constexpr int kPcB = 32;               // candidates (and at most as many pivots) per step
constexpr int kPcMaxRank = 3072;       // columns the workspace holds at most
constexpr int kPcProbes = 3;            // vectors the remainder is tried on
constexpr int kPcSweeps = 8;            // refinements at most
// a refinement of this size (of |c|) leaves its square; one that is still above
// kPcSettled when they no longer shrink is not rounding (condition numbers reach
// 1 / rcond <= 1.1e10)
constexpr double kPcConverged = 1e-8, kPcSettled = 1e-5;
constexpr double kPcKeep = 0.01;       // accepted pivots, relative to the largest remaining diagonal
// pivots end here, relative to G's largest diagonal entry: the noise left by
// the updates is mostly below 1e-13 (1.4e-14 absolute at n = 2000, r = 800), but
// at n = 24000, r = 1921 one clip in ten had an entry above 1024 eps, took it as
// a pivot and was refused (6.9 s for 19 ms).  Over 190 matrices of n = 1900 to 24000 the largest entry
// left was 1960 eps, none was refused.
// What lies between is judged with the remainder, whose test is far
// stricter than this line.
constexpr double kPcTol = 4096 * 2.220446049250313e-16;

struct PcState {
    int k, nacc, done, bad;            // columns; accepted in this step; 1 finished, 2 out of columns; indefinite
    int cand[kPcB], order[kPcB];       // candidate rows (-1: none); accepted candidates in pivot order
    double maxd0, tol, dmax;           // largest diagonal entry of G; stop below; largest remaining
    double trace0;                     // of G
    double R[kPcB * kPcB];             // factor of the accepted block, row-major lower
    double trace;                      // of the remainder G - L L^T
    double probe, norm;                // largest |G v - L L^T v|_2 of the probes; |B|_inf
    double ratio;                      // |last refinement| / |c|
    int info[2];
};

__device__ __forceinline__ double warp_max(double v) {
    for (int o = 16; o; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// d = diag(G), the tolerance, zero state (one block)
__global__ void __launch_bounds__(1024) pc_init_kernel(const double* __restrict__ G, int64_t ld, int n,
                                                       double* __restrict__ d, PcState* __restrict__ st) {
    __shared__ double sm[32], ts[32];
    double m = 0.0, tr = 0.0;
    bool neg = false;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double v = G[(int64_t)i * ld + i];
        d[i] = v;
        m = fmax(m, v);
        tr += v;
        neg |= !(v >= 0.0);
    }
    m = warp_max(m);
    for (int o = 16; o; o >>= 1) tr += __shfl_xor_sync(0xffffffffu, tr, o);
    if ((threadIdx.x & 31) == 0) {
        sm[threadIdx.x >> 5] = m;
        ts[threadIdx.x >> 5] = tr;
    }
    const int any = __syncthreads_or(neg);
    if (threadIdx.x == 0) {
        for (int w = 1; w < 32; ++w) {
            m = fmax(m, sm[w]);
            tr += ts[w];
        }
        st->trace0 = tr;
        st->k = st->nacc = st->done = 0;
        st->bad = any || !(m > 0.0) || !(m < 1e300);
        st->maxd0 = m;
        st->tol = kPcTol * m;
        st->dmax = m;
        st->probe = st->norm = st->ratio = 0.0;
        st->info[0] = st->info[1] = 0;
    }
}

// the columns accepted last join k; candidates of the next step and their rows of L (32 warps, warp = group)
__global__ void __launch_bounds__(1024) pc_select_kernel(double* __restrict__ d, int n, const double* __restrict__ L,
                                                         int64_t ldl, int cols, int used, double* __restrict__ LP,
                                                         PcState* __restrict__ st) {
    __shared__ double smax[32], smin[32], ssum[32];
    __shared__ int s_done;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double best = -1.0, low = 0.0, sum = 0.0;
    int at = -1;
    for (int i = w + 32 * lane; i < n; i += 1024) {
        const double v = d[i];
        sum += v;
        low = fmin(low, v);
        if (v > best) {
            best = v;
            at = i;
        }
    }
    for (int o = 16; o; o >>= 1) {
        const double b2 = __shfl_xor_sync(0xffffffffu, best, o), l2 = __shfl_xor_sync(0xffffffffu, low, o);
        const int a2 = __shfl_xor_sync(0xffffffffu, at, o);
        low = fmin(low, l2);
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (b2 > best || (b2 == best && a2 >= 0 && (at < 0 || a2 < at))) {
            best = b2;
            at = a2;
        }
    }
    if (lane == 0) {
        smax[w] = best;
        smin[w] = low;
        ssum[w] = sum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = smax[0], l = smin[0];
        for (int k = 1; k < 32; ++k) {
            m = fmax(m, smax[k]);
            l = fmin(l, smin[k]);
            sum += ssum[k];
        }
        const int k = st->k + st->nacc;
        st->k = k;
        st->nacc = 0;
        st->dmax = m;
        if (l < -16.0 * st->tol) st->bad = 1;
        if (!st->done) {
            if (!(m > st->tol)) st->done = 1;
            else if (k + kPcB > cols) st->done = 2;
            // columns taken largest first reduce the trace less and less, so the
            // rank is at least k over the share of the trace they have taken
            else if (k > 0 && (double)k * st->trace0 > 0.55 * n * (st->trace0 - sum)) st->done = 2;
        }
        s_done = st->done || st->bad;
        smax[0] = m;
    }
    __syncthreads();
    const bool use = !s_done && at >= 0 && best > st->tol && best >= kPcKeep * smax[0];
    if (lane == 0) st->cand[w] = use ? at : -1;
    for (int j = lane; j < used; j += 32) LP[(int64_t)w * ldl + j] = use ? L[(int64_t)at * ldl + j] : 0.0;
}

// C[i][j] = G(i, cand_j), from G's lower triangle
__global__ void __launch_bounds__(256) pc_gather_kernel(const double* __restrict__ G, int64_t ld, int n,
                                                        double* __restrict__ C, const PcState* __restrict__ st) {
    const int j = threadIdx.x & 31;
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= n) return;
    const int c = st->cand[j];
    C[(int64_t)i * kPcB + j] = c < 0 ? 0.0 : __ldg(G + (int64_t)max(i, c) * ld + min(i, c));
}

// Pivoted Cholesky of the candidates' block (one warp, lane = candidate): the
// column of each pivot is formed when it is taken, from the lane's own entries
// of L (registers) and the pivot's (shared memory), and pivots are ranked by
// one integer reduction (the diagonal entry's float bits above the lane's
// number; their exact order does not matter).
__global__ void __launch_bounds__(32) pc_factor_kernel(const double* __restrict__ C, PcState* __restrict__ st) {
    __shared__ double S[kPcB][kPcB + 1], Lc[kPcB][kPcB + 1];   // the block; Lc[j][row]
    const int r = threadIdx.x;
    const int mine = st->cand[r];
    const double floor_ = fmax(st->tol, kPcKeep * st->dmax);
    double rows[kPcB];
#pragma unroll
    for (int c = 0; c < kPcB; ++c) {
        const int row = __shfl_sync(0xffffffffu, mine, c);
        rows[c] = row >= 0 && mine >= 0 ? C[(int64_t)row * kPcB + r] : 0.0;
    }
#pragma unroll
    for (int c = 0; c < kPcB; ++c) S[c][r] = rows[c];
    __syncwarp();
    bool left = mine >= 0;
    double diag = S[r][r];
    double l[kPcB];
    int a = 0, at = -1;                                      // at: this lane's place in the pivot order
#pragma unroll
    for (int j = 0; j < kPcB; ++j) {
        l[j] = 0.0;
        if (a == j) {
            const unsigned key = left && diag >= floor_ ? (__float_as_uint((float)diag) & ~31u) | (unsigned)r : 0u;
            const unsigned best = __reduce_max_sync(0xffffffffu, key);
            if (best >= 32u) {
                const int p = best & 31u;
                const double inv = 1.0 / sqrt(__shfl_sync(0xffffffffu, diag, p));
                double v0 = S[p][r], v1 = 0.0;
#pragma unroll
                for (int t = 0; t < j; t += 2) {
                    v0 = fma(-l[t], Lc[t][p], v0);
                    if (t + 1 < j) v1 = fma(-l[t + 1], Lc[t + 1][p], v1);
                }
                l[j] = r == p ? diag * inv : left ? (v0 + v1) * inv : 0.0;
                if (r == p) {
                    left = false;
                    at = j;
                }
                diag = fma(-l[j], l[j], diag);
                Lc[j][r] = l[j];
                if (r == 0) st->order[j] = p;
                a = j + 1;
                __syncwarp();
            }
        }
    }
    // R[t][j]: entry of pivot t in column j
    if (at >= 0) {
#pragma unroll
        for (int j = 0; j < kPcB; ++j)
            if (j <= at) st->R[at * kPcB + j] = l[j];
    }
    if (r == 0) st->nacc = a;
}

// the accepted columns of L: every row of C substituted through R; d less their
// squares.  Thread = row; rows enter and leave through shared memory, so that
// global memory sees whole rows of 256 bytes.
__global__ void __launch_bounds__(64) pc_update_kernel(const double* __restrict__ C, int n, double* __restrict__ L,
                                                       int64_t ldl, double* __restrict__ d,
                                                       const PcState* __restrict__ st) {
    __shared__ double R[kPcB][kPcB];
    __shared__ double tile[2][32][kPcB + 1];
    __shared__ double inv[kPcB];
    __shared__ int ord[kPcB], piv[kPcB];
    const int a = st->nacc, k = st->k;
    if (a == 0) return;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i0 = blockIdx.x * 64 + 32 * w, i = i0 + lane;
    for (int e = threadIdx.x; e < kPcB * kPcB; e += 64) {
        const int t = e / kPcB, j = e % kPcB;
        R[t][j] = t < a && j <= t ? st->R[e] : 0.0;
    }
    if (threadIdx.x < kPcB) {
        const int t = threadIdx.x;
        inv[t] = t < a ? 1.0 / st->R[t * kPcB + t] : 0.0;
        ord[t] = t < a ? st->order[t] : 0;
        piv[t] = t < a ? st->cand[st->order[t]] : -1;
    }
#pragma unroll 8
    for (int r = 0; r < 32; ++r) tile[w][r][lane] = i0 + r < n ? C[(int64_t)(i0 + r) * kPcB + lane] : 0.0;
    __syncthreads();
    double x[kPcB];
#pragma unroll
    for (int t = 0; t < kPcB; ++t) x[t] = t < a ? tile[w][lane][ord[t]] : 0.0;
    int own = kPcB;                        // row i is the own-th pivot: its later entries are zero by construction
#pragma unroll
    for (int t = 0; t < kPcB; ++t)
        if (piv[t] == i) own = t;
    double s = 0.0;
#pragma unroll
    for (int t = 0; t < kPcB; ++t) {
        if (t > own) x[t] = 0.0;
        x[t] *= inv[t];
        s = fma(x[t], x[t], s);
#pragma unroll
        for (int j = t + 1; j < kPcB; ++j) x[j] = fma(-R[j][t], x[t], x[j]);
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < kPcB; ++t) tile[w][lane][t] = x[t];
    __syncwarp();
    if (lane < a)
#pragma unroll 8
        for (int r = 0; r < 32; ++r)
            if (i0 + r < n) L[(int64_t)(i0 + r) * ldl + k + lane] = tile[w][r][lane];
    if (i < n) d[i] = own < kPcB ? 0.0 : d[i] - s;
}

// y_b = A^T x_b (row-major A, n x r), b < gridDim.y: block of 32 columns x 32 row groups
__global__ void __launch_bounds__(1024) pc_gemv_t_kernel(const double* __restrict__ A, int64_t ld, int n, int r,
                                                        const double* __restrict__ x, double* __restrict__ y) {
    __shared__ double part[32][33];
    const int c = blockIdx.x * 32 + (threadIdx.x & 31), g = threadIdx.x >> 5;
    const double* xv = x + (int64_t)blockIdx.y * n;
    double s0 = 0.0, s1 = 0.0;
    if (c < r) {
        int i = g;
        for (; i + 32 < n; i += 64) {
            s0 = fma(A[(int64_t)i * ld + c], xv[i], s0);
            s1 = fma(A[(int64_t)(i + 32) * ld + c], xv[i + 32], s1);
        }
        if (i < n) s0 = fma(A[(int64_t)i * ld + c], xv[i], s0);
    }
    part[g][threadIdx.x & 31] = s0 + s1;
    __syncthreads();
    if (g == 0 && c < r) {
        double t = 0.0;
        for (int k = 0; k < 32; ++k) t += part[k][threadIdx.x & 31];
        y[(int64_t)blockIdx.y * r + c] = t;
    }
}

// y_b = A x_b, one warp a row
__global__ void __launch_bounds__(256) pc_gemv_kernel(const double* __restrict__ A, int64_t ld, int n, int r,
                                                      const double* __restrict__ x, double* __restrict__ y) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= n) return;
    const double* xv = x + (int64_t)blockIdx.y * r;
    double s = 0.0;
    for (int j = lane; j < r; j += 32) s = fma(A[(int64_t)i * ld + j], xv[j], s);
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    double* q = y + (int64_t)blockIdx.y * n + i;
    if (lane == 0) *q = s;
}

// y_b = G x_b from G's lower triangle, b < NV: the part left of the diagonal
// by rows (one warp each) into y, then the part below it by columns added.
// Columns: few blocks at the small configuration (n = 1780), so each takes
// kPcCols of them and loads kPcRows rows at a time: 13 us (20 for four vectors),
// against 57 with 32 columns a block and one row at a time.
constexpr int kPcCols = 16, kPcRows = 8;

template <int NV>
__global__ void __launch_bounds__(256) pc_symv_rows_kernel(const double* __restrict__ G, int64_t ld, int n,
                                                           const double* __restrict__ x, double* __restrict__ y) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= n) return;
    const double* row = G + (int64_t)i * ld;
    double s[NV] = {};
    for (int j = lane; j <= i; j += 32) {
        const double g = row[j];
#pragma unroll
        for (int b = 0; b < NV; ++b) s[b] = fma(g, x[(int64_t)b * n + j], s[b]);
    }
#pragma unroll
    for (int b = 0; b < NV; ++b) {
        for (int o = 16; o; o >>= 1) s[b] += __shfl_xor_sync(0xffffffffu, s[b], o);
        if (lane == 0) y[(int64_t)b * n + i] = s[b];
    }
}

template <int NV>
__global__ void __launch_bounds__(512) pc_symv_cols_kernel(const double* __restrict__ G, int64_t ld, int n,
                                                           const double* __restrict__ x, double* __restrict__ y) {
    constexpr int groups = 512 / kPcCols;
    __shared__ double part[NV][groups][kPcCols + 1];
    const int q = threadIdx.x % kPcCols, c = blockIdx.x * kPcCols + q, g = threadIdx.x / kPcCols;
    double s[NV] = {};
    if (c < n)
        for (int i0 = blockIdx.x * kPcCols + g; i0 < n; i0 += groups * kPcRows) {
            double v[kPcRows];
#pragma unroll
            for (int k = 0; k < kPcRows; ++k) {
                const int i = i0 + groups * k;
                v[k] = i > c && i < n ? G[(int64_t)i * ld + c] : 0.0;
            }
#pragma unroll
            for (int k = 0; k < kPcRows; ++k) {
                const int i = min(i0 + groups * k, n - 1);
#pragma unroll
                for (int b = 0; b < NV; ++b) s[b] = fma(v[k], x[(int64_t)b * n + i], s[b]);
            }
        }
#pragma unroll
    for (int b = 0; b < NV; ++b) part[b][g][q] = s[b];
    __syncthreads();
    if (g < NV && c < n) {
        double t = 0.0;
        for (int k = 0; k < groups; ++k) t += part[g][k][q];
        y[(int64_t)g * n + c] += t;
    }
}

// the probes: entries of either sign and magnitudes 0.5 to 1.5, from the splitmix64
// generator (Steele, Lea, Flood 2014) seeded by G's trace and largest diagonal entry
__global__ void pc_probes_kernel(double* __restrict__ v, int n, const PcState* __restrict__ st) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kPcProbes * n) return;
    unsigned long long z = (unsigned long long)__double_as_longlong(st->trace0) ^
                           ((unsigned long long)__double_as_longlong(st->maxd0) << 1);
    z += 0x9e3779b97f4a7c15ull * (unsigned long long)(i + 1);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    z ^= z >> 31;
    const double m = 0.5 + (double)(z >> 12) * 0x1p-52;
    v[i] = z & 1 ? m : -m;
}

// res = q - y
__global__ void pc_residual_kernel(const double* __restrict__ q, const double* __restrict__ y, double* __restrict__ res,
                                   int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) res[i] = q[i] - y[i];
}

// c += v, st->ratio = |v| / |c| (one block)
__global__ void __launch_bounds__(1024) pc_correct_kernel(double* __restrict__ c, const double* __restrict__ v, int n,
                                                          PcState* __restrict__ st) {
    __shared__ double sm[32], tm[32];
    double s = 0.0, t = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double u = c[i] + v[i];
        c[i] = u;
        s = fma(v[i], v[i], s);
        t = fma(u, u, t);
    }
    for (int o = 16; o; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    if ((threadIdx.x & 31) == 0) {
        sm[threadIdx.x >> 5] = s;
        tm[threadIdx.x >> 5] = t;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 32; ++w) {
            s += sm[w];
            t += tm[w];
        }
        st->ratio = s > 0.0 ? sqrt(s / t) : s;       // 0 for q = 0, NaN stays
    }
}

// st->probe = the largest |y_b - z_b|_2 (raised to it; one block per probe),
// st->trace = sum of |d|
__global__ void __launch_bounds__(1024) pc_probe_kernel(const double* __restrict__ y, const double* __restrict__ z,
                                                        const double* __restrict__ d, int n, PcState* __restrict__ st) {
    __shared__ double sm[32], tm[32];
    y += (int64_t)blockIdx.x * n;
    z += (int64_t)blockIdx.x * n;
    double s = 0.0, t = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        s = fma(y[i] - z[i], y[i] - z[i], s);
        t += fabs(d[i]);
    }
    for (int o = 16; o; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    if ((threadIdx.x & 31) == 0) {
        sm[threadIdx.x >> 5] = s;
        tm[threadIdx.x >> 5] = t;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 32; ++w) {
            s += sm[w];
            t += tm[w];
        }
        // (non-negative doubles, and a NaN above them, order like their bits)
        atomicMax(reinterpret_cast<unsigned long long*>(&st->probe),
                  (unsigned long long)__double_as_longlong(fabs(sqrt(s))));
        if (blockIdx.x == 0) st->trace = t;
    }
}

// |B|_inf by rows into the state (a maximum of non-negative doubles orders like their bits)
__global__ void __launch_bounds__(256) pc_norm_kernel(const double* __restrict__ B, int r, int ldb,
                                                      PcState* __restrict__ st) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= r) return;
    double s = 0.0;
    for (int j = lane; j < r; j += 32) s += fabs(B[(int64_t)i * ldb + j]);
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0)
        atomicMax(reinterpret_cast<unsigned long long*>(&st->norm), (unsigned long long)__double_as_longlong(s));
}

__global__ void pc_shift_kernel(const double* __restrict__ B, int r, int ldb, double rcond,
                                const PcState* __restrict__ st, double* __restrict__ B2) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= (int64_t)r * ldb) return;
    B2[e] = e % ldb < r ? B[e] - (e / ldb == e % ldb ? rcond * st->norm : 0.0) : 0.0;
}

struct PsdWork {
    PcState* st;
    double *d, *L, *LP, *C, *B, *B2, *v, *y, *t, *z;
    void *wk, *wk2;
    int64_t ldl, bytes;
    int cols;
};

// columns the factor may take: half of n (beyond it the eigendecomposition is
// the better one), at most kPcMaxRank, and kPcB of slack
static int psd_cols(int n) { return (std::min(n / 2, kPcMaxRank) + 2 * kPcB - 1) / kPcB * kPcB; }

static PsdWork psd_work(int n, char* base) {
    PsdWork w;
    int64_t off = 0;
    auto take = [&](int64_t doubles) {
        char* p = base + off;
        off += (doubles * 8 + 255) & ~(int64_t)255;
        return reinterpret_cast<double*>(p);
    };
    w.cols = psd_cols(n);
    w.ldl = w.cols;
    w.st = reinterpret_cast<PcState*>(take((sizeof(PcState) + 7) / 8));
    w.d = take(n);
    w.L = take((int64_t)n * w.ldl);
    w.LP = take((int64_t)kPcB * w.ldl);
    w.C = take((int64_t)n * kPcB);
    w.B = take((int64_t)w.cols * w.cols);
    w.B2 = take((int64_t)w.cols * w.cols);
    w.v = take((1 + kPcProbes) * (int64_t)n);
    w.y = take((1 + kPcProbes) * (int64_t)n);
    w.t = take(kPcProbes * (int64_t)w.cols);
    w.z = take(w.cols);
    w.wk = take(chol64_bytes(w.cols) / 8);
    w.wk2 = take(chol64_bytes(w.cols) / 8);
    w.bytes = off;
    return w;
}

}  // namespace vtb

using namespace vtb;

VTB_API int vtb_solve_psd_workspace(int n, int64_t* bytes) {
    VTB_CHECK_ARG(n > 0 && bytes);
    *bytes = psd_work(n, nullptr).bytes;
    return VTB_OK;
}

VTB_API int vtb_solve_psd(const double* G, int64_t ld, const double* q, double* c, int n, double rcond, void* work,
                          int64_t work_bytes, int32_t* kept, int32_t* accepted, void* stream) {
    VTB_CHECK_ARG(n > 0 && ld >= n && G && q && c && work && accepted && ((uintptr_t)work & 255) == 0);
    *accepted = 0;
    if (!(rcond >= 100.0 * kPcTol) || !(rcond < 1.0)) return VTB_OK;   // the rule would keep noise
    int st = VTB_OK;
    const PsdWork w = psd_work(n, reinterpret_cast<char*>(work));
    VTB_CHECK_ARG(work_bytes >= w.bytes);
    cudaStream_t s = as_stream(stream);
    VTB_CUDA_TRY(cudaMemsetAsync(w.L, 0, (size_t)n * w.ldl * 8, s));
    pc_init_kernel<<<1, 1024, 0, s>>>(G, ld, n, w.d, w.st);
    struct {
        int k, nacc, done, bad;
    } host = {0, 0, 0, 0};
    constexpr int kCheck = 4;              // steps between looks at the state
    const int most = 2 * (w.cols / kPcB) + kCheck;
    for (int step = 0; step < most && !host.done && !host.bad; ++step) {
        const int cols = std::min(step * kPcB, w.cols);      // k is at most this
        pc_select_kernel<<<1, 1024, 0, s>>>(w.d, n, w.L, w.ldl, w.cols, cols, w.LP, w.st);
        pc_gather_kernel<<<ceil_div(n, 8), 256, 0, s>>>(G, ld, n, w.C, w.st);
        if (cols) {
            const GemmF64Args g{n, kPcB, cols, w.L, w.ldl, 1, w.LP, w.ldl, 1, w.C, kPcB, 1, -1.0, 1.0};
            st = gemm_f64(g, s);
            if (st) return st;
        }
        pc_factor_kernel<<<1, 32, 0, s>>>(w.C, w.st);
        pc_update_kernel<<<ceil_div(n, 64), 64, 0, s>>>(w.C, n, w.L, w.ldl, w.d, w.st);
        if (step % kCheck == 1 || step + 1 == most) {   // the first look as soon as the trace can refuse
            VTB_CUDA_TRY(cudaMemcpyAsync(&host, w.st, sizeof(host), cudaMemcpyDeviceToHost, s));
            VTB_CUDA_TRY(cudaStreamSynchronize(s));
        }
    }
    st = launch_status();
    if (st) return st;
    if (host.done != 1 || host.bad || host.k < 1) return VTB_OK;
    const int r = host.k, ldb = r + (r & 1);      // columns on 16 bytes
    const GemmF64Args gb{r, r, n, w.L, 1, w.ldl, w.L, 1, w.ldl, w.B, ldb, 1, 1.0, 0.0};
    st = gemm_f64(gb, s);
    if (st) return st;
    pc_norm_kernel<<<ceil_div((int64_t)r * 32, 256), 256, 0, s>>>(w.B, r, ldb, w.st);
    pc_shift_kernel<<<ceil_div((int64_t)r * ldb, 256), 256, 0, s>>>(w.B, r, ldb, rcond, w.st, w.B2);
    int* info = reinterpret_cast<int*>(reinterpret_cast<char*>(w.st) + offsetof(PcState, info));
    // B for the solves, and B - rcond |B| I for the rule (its right-hand side, 0, is not used)
    const Chol64System sys[2] = {{w.B, ldb, r, w.t, w.wk, info, nullptr, 0.0},
                                 {w.B2, ldb, r, w.z, w.wk2, info + 1, nullptr, 0.0}};
    VTB_CUDA_TRY(cudaMemsetAsync(w.z, 0, (size_t)r * 8, s));
    // y = L B^-3 L^T x; the first time with the factorisation, which leaves the first forward solve done
    auto apply = [&](const double* x, double* y, bool first) -> int {
        pc_gemv_t_kernel<<<dim3(ceil_div(r, 32), 1), 1024, 0, s>>>(w.L, w.ldl, n, r, x, w.t);
        const int f = first ? chol64_factor(sys, 2, s) : VTB_OK;
        if (f) return f;
        const int g = chol64_solve(sys[0], first, first ? 5 : 6, false, s);
        if (g) return g;
        pc_gemv_kernel<<<dim3(ceil_div((int64_t)n * 32, 256), 1), 256, 0, s>>>(w.L, w.ldl, n, r, w.t, y);
        return VTB_OK;
    };
    const int rows_grid = ceil_div((int64_t)n * 32, 256), cols_grid = ceil_div(n, kPcCols);
    auto product = [&](const double* x, double* y) {
        pc_symv_rows_kernel<1><<<rows_grid, 256, 0, s>>>(G, ld, n, x, y);
        pc_symv_cols_kernel<1><<<cols_grid, 512, 0, s>>>(G, ld, n, x, y);
    };
    if ((st = apply(q, w.v, true))) return st;
    // one pass over G for c and the probes
    constexpr int nv = 1 + kPcProbes;
    pc_probes_kernel<<<ceil_div((int64_t)kPcProbes * n, 256), 256, 0, s>>>(w.v + n, n, w.st);
    pc_symv_rows_kernel<nv><<<rows_grid, 256, 0, s>>>(G, ld, n, w.v, w.y);
    pc_symv_cols_kernel<nv><<<cols_grid, 512, 0, s>>>(G, ld, n, w.v, w.y);
    pc_gemv_t_kernel<<<dim3(ceil_div(r, 32), kPcProbes), 1024, 0, s>>>(w.L, w.ldl, n, r, w.v + n, w.t);
    pc_gemv_kernel<<<dim3(rows_grid, kPcProbes), 256, 0, s>>>(w.L, w.ldl, n, r, w.t, w.v + n);
    pc_probe_kernel<<<kPcProbes, 1024, 0, s>>>(w.y + n, w.v + n, w.d, n, w.st);
    VTB_CUDA_TRY(cudaMemcpyAsync(c, w.y, (size_t)n * 8, cudaMemcpyDeviceToDevice, s));
    PcState end;
    double last = 1.0;
    for (int sweep = 0; sweep < kPcSweeps; ++sweep) {
        product(c, w.v);
        pc_residual_kernel<<<ceil_div(n, 256), 256, 0, s>>>(q, w.v, w.y, n);
        product(w.y, w.v);
        if ((st = apply(w.v, w.y, false))) return st;
        pc_correct_kernel<<<1, 1024, 0, s>>>(c, w.y, n, w.st);
        VTB_CUDA_TRY(cudaMemcpyAsync(&end, w.st, sizeof(end), cudaMemcpyDeviceToHost, s));
        if (sweep == 0 && kept) VTB_CUDA_TRY(cudaMemcpyAsync(kept, w.st, 4, cudaMemcpyDeviceToDevice, s));
        VTB_CUDA_TRY(cudaStreamSynchronize(s));
        st = launch_status();
        if (st) return st;
        if (end.info[0] != 0 || end.info[1] != 0 || !(end.ratio > kPcConverged) || end.ratio > 0.5 * last) break;
        last = end.ratio;
    }
    // the remainder against the rule, with s_0 at least the largest diagonal entry and |B|_inf / sqrt(r)
    const double rule = rcond * std::max(end.maxd0, end.norm / std::sqrt((double)r));
    if (end.info[0] != 0 || end.info[1] != 0 || !(end.ratio <= kPcSettled)) return VTB_OK;
    if (!(end.trace <= 0.1 * rule) || !(end.probe <= 0.05 * rule)) return VTB_OK;
    *accepted = 1;
    return VTB_OK;
}
