// Float64 Cholesky solve of ONE symmetric positive definite system (the real
// form of the float64 decoder's coefficient system), M x = b.
//
// At K = 979 the library's factorisation is bound by its chain of panel steps
// (459 us for 0.3 GFLOP) and its two triangular solves by theirs (155 us).
// Here one cooperative launch factorises in 32 x 32 tiles (T = ceil(K/32)) as
// a data-flow graph, with the right-hand side as one more tile row (row T, one
// row used): its tiles become y = L^-1 b on the way.
//
//   CTA 0 ("diagonal"), step k = 0..T-1: the panel [A_kk; I] -> [L_kk; L_kk^-T]
//     in blocks of 8 columns (warp 0 factorises the 8 x 8 blocks and solves the
//     32 rows of a column block, warps 1-2 apply the rank-8 updates, warp 3
//     waits for the next two tiles and fetches them); publishes L_kk^-1; the
//     sub-diagonal tile L_{k+1,k} = A_{k+1,k} L_kk^-T; the next diagonal tile's
//     last update.
//   CTAs 1.. ("workers"): for tile (I, J) the updates A_IJ -= sum_k' L_Ik' L_Jk'^T
//     (accumulators in registers), then for I >= J + 2 the product with the
//     published L_JJ^-T; sub-diagonal and diagonal tiles receive all updates
//     but the last.
//
// Tasks are ordered by the step whose outputs they need (group g: the tiles
// (I, g) for I = g+2..T, the sub-diagonal (g+2, g+1) and the diagonal
// (g+2, g+2), pre-updated through g) and dealt round-robin; each CTA runs its
// tasks in that order.  A task depends on earlier tasks and on diagonal steps
// that depend on earlier groups only, so with every CTA resident (cooperative
// launch) the graph cannot deadlock.  Products run on the float64 tensor path
// (mma m8n8k4); tiles in shared memory have columns of 36 doubles, which makes
// every fragment read conflict-free.  Every wait is bounded: after the limit
// the call is marked aborted (flag 3) and all CTAs return.
//
// The triangular solves are a second launch, one CTA per block row: the partial
// sums over the blocks before stay in registers, so only the last block's
// product, one reduction and the product with L_JJ^-1 lie between two
// hand-offs; the hand-off is the value itself (readers poll the words, which
// start as all ones).  Several solves, forward and backward in turn, run in one
// launch, each reading the words of the one before.
//
// Bound: latency, the workers' more than the panel's: of a step's 16,000 cycles at
// K = 979 the panel takes 9,000, and a tile passes two publications and two
// products of workers between the steps that produce its operands and the one
// that needs it.  Factor and solves, cuSOLVER -> here (us): K = 261 201 -> 98, 979
// 595 -> 269, 1921 1129 -> 552, 3001 1747 -> 1024.  Columns that do not start
// on 16 bytes are loaded entry by entry (679 us at 979).  Two and one CTAs per SM:
// 271 and 289 us at 979, 1375 and 2246 at 3001; warp 3 publishing and writing
// instead of taking a share of the products: 283 us at 979.
#include "chol_f64.cuh"

#include <algorithm>

namespace vtb {

constexpr int kDT = 32;
constexpr int kDL = 36;                 // doubles per tile column in shared memory
constexpr int kDE = kDT * kDL;
constexpr int kDThreads = 128;
constexpr unsigned kDSpin = 1u << 20;
constexpr int kDPerSM = 4;

struct DCholCtx {
    double* A;
    int64_t ld;
    int K, T;
    double* x;           // b on entry, y = L^-1 b when done
    double* Dinv;        // T tiles: (L_kk^-1)[c][t] at c*32 + t
    unsigned* flag;      // (T + 1) * T: 1 = worker part done, 2 = tile final
    int* abort_word;
    int32_t* status;
    double* piv;
    double rcond;
    unsigned limit;
};

struct DCholSmem {
    double a[2][kDE];    // worker: L_Ik' (double buffer); diagonal CTA: current and next diagonal tile
    double b[2][kDE];    // worker: L_Jk' (double buffer), then L_JJ^-1; diagonal CTA: L_kk^-T, sub-diagonal tile
    double x[kDE];       // worker: the task's tile
    double rinv[kDT];
    int ok;
};

__device__ __forceinline__ unsigned d_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void d_release(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}

// one thread: until *f1 >= v1 and *f2 >= v2 (f2 may be null); false once the call is aborted
__device__ __forceinline__ bool d_poll(const DCholCtx& c, const unsigned* f1, unsigned v1, const unsigned* f2,
                                       unsigned v2) {
    for (unsigned it = 0;; ++it) {
        const unsigned a = d_acquire(f1), b = f2 ? d_acquire(f2) : v2;
        if (a >= v1 && b >= v2) return true;
        if (it > c.limit || *(volatile int*)c.abort_word != 0) {
            atomicExch(c.abort_word, 1);
            atomicMax(c.status, 3);
            return false;
        }
    }
}

__device__ bool d_wait(const DCholCtx& c, const unsigned* f1, unsigned v1, const unsigned* f2, unsigned v2, int* s_ok) {
    __syncthreads();
    if (threadIdx.x == 0) *s_ok = d_poll(c, f1, v1, f2, v2);
    __syncthreads();
    return *s_ok != 0;
}

__device__ __forceinline__ void d_cp16(double* dst, const double* src) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void d_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void d_cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// element (r, j) of tile (I, J) in global memory; the identity beyond K, the
// right-hand side in row 0 of tile row T
__device__ __forceinline__ double d_entry(const DCholCtx& c, int I, int J, int r, int j) {
    const int gc = J * kDT + j;
    if (I == c.T) return r == 0 && gc < c.K ? __ldcg(c.x + gc) : 0.0;
    const int gr = I * kDT + r;
    if (gr < c.K && gc < c.K) return __ldcg(c.A + (int64_t)gc * c.ld + gr);
    return gr == gc ? 1.0 : 0.0;
}

__device__ __forceinline__ bool d_wide(const DCholCtx& c, int I, int J) {
    return I < c.T && (I + 1) * kDT <= c.K && (J + 1) * kDT <= c.K && (c.ld & 1) == 0 && ((uintptr_t)c.A & 15) == 0;
}

// tile (I, J) into shared memory by n threads; one cp.async group per call
__device__ __forceinline__ void d_load(const DCholCtx& c, double* s, int I, int J, int tid, int n) {
    if (d_wide(c, I, J)) {
        const double* g = c.A + (int64_t)J * kDT * c.ld + I * kDT;
        for (int e = tid; e < kDT * kDT / 2; e += n) {
            const int j = e >> 4, r = (e & 15) * 2;
            d_cp16(s + j * kDL + r, g + j * c.ld + r);
        }
    } else {
        for (int e = tid; e < kDT * kDT; e += n) s[(e >> 5) * kDL + (e & 31)] = d_entry(c, I, J, e & 31, e >> 5);
    }
    d_commit();
}

// the tile in shared memory to (I, J) (a diagonal tile's lower triangle only)
__device__ __forceinline__ void d_store(const DCholCtx& c, const double* s, int I, int J, int tid, int n) {
    for (int e = tid; e < kDT * kDT; e += n) {
        const int j = e >> 5, r = e & 31;
        const int gc = J * kDT + j, gr = I * kDT + r;
        const double v = s[j * kDL + r];
        if (I == c.T) {
            if (r == 0 && gc < c.K) __stcg(c.x + gc, v);
        } else if (gr < c.K && gc < c.K && (I != J || r >= j)) {
            __stcg(c.A + (int64_t)gc * c.ld + gr, v);
        }
    }
}

__device__ __forceinline__ void d_mma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// rows 8w..8w+7 of acc -= P Q^T (Q[n][k] at k*36 + n) or, TRI, acc += P Q^T with
// Q lower triangular and k contiguous (Q[n][k] at n*36 + k); columns 8j.. for j < nj.
// Lane l holds row l / 4, columns 2 (l % 4) + {0, 1} of each 8 x 8 block.  The
// product is summed by itself and then subtracted: taken off the tile one k at a
// time, every one of K terms is rounded to the tile's own size, and the solve's
// error was up to twice the library's (windows of K = 221 and 261: 1.1 to 2.3 times
// it; summed apart 0.3 to 1.0 times, at the same speed).
template <bool TRI>
__device__ __forceinline__ void d_product(double (&acc)[4][2], const double* P, const double* Q, int w, int nj) {
    const int lane = threadIdx.x & 31, lo = lane & 3, hi = lane >> 2;
    double t[4][2] = {};
#pragma unroll
    for (int kk = 0; kk < kDT; kk += 4) {
        const double p = P[(kk + lo) * kDL + 8 * w + hi];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (TRI ? kk < 8 * j + 8 : j < nj)
                d_mma(t[j], p, TRI ? Q[(8 * j + hi) * kDL + kk + lo] : Q[(kk + lo) * kDL + 8 * j + hi]);
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) acc[j][e] = TRI ? acc[j][e] + t[j][e] : acc[j][e] - t[j][e];
}

__device__ __forceinline__ void d_acc_to(const double (&acc)[4][2], double* s, int w, int nj = 4) {
    const int lane = threadIdx.x & 31, lo = lane & 3, hi = lane >> 2;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (j < nj) {
            s[(8 * j + 2 * lo) * kDL + 8 * w + hi] = acc[j][0];
            s[(8 * j + 2 * lo + 1) * kDL + 8 * w + hi] = acc[j][1];
        }
}

// ------------------------------------------------------------------ the panel
// the 8 x 8 diagonal block bb of S in one warp, every lane on its own copy
__device__ __forceinline__ void d_potrf8(double* S, double* rinv, int bb, double& pmin, double& pmax, int& bad,
                                         int nvalid) {
    const int o = 8 * bb;
    double a[8][8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
            const double2 v = *reinterpret_cast<const double2*>(S + (o + j) * kDL + o + i);
            a[i][j] = v.x;
            a[i + 1][j] = v.y;
        }
    double rs[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        double p = a[j][j];
        if (!(p > 0.0)) {
            bad = 1;
            p = 1.0;
        }
        if (o + j < nvalid) {
            pmin = fmin(pmin, p);
            pmax = fmax(pmax, p);
        }
        rs[j] = rsqrt(p);
#pragma unroll
        for (int i = j; i < 8; ++i) a[i][j] *= rs[j];
#pragma unroll
        for (int q = j + 1; q < 8; ++q)
#pragma unroll
            for (int i = q; i < 8; ++i) a[i][q] = fma(-a[i][j], a[q][j], a[i][q]);
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
        for (int i = 0; i < 8; i += 2)
            *reinterpret_cast<double2*>(S + (o + j) * kDL + o + i) =
                make_double2(i >= j ? a[i][j] : 0.0, i + 1 >= j ? a[i + 1][j] : 0.0);
        rinv[o + j] = rs[j];
    }
    __syncwarp();
}

// row r of column block bb of X: x <- x L_bb^-T
__device__ __forceinline__ void d_subst8(double* X, const double* L, const double* rinv, int bb, int r) {
    const int o = 8 * bb;
    double x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = X[(o + j) * kDL + r];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        double v = x[j];
#pragma unroll
        for (int t = 0; t < j; ++t) v = fma(-x[t], L[(o + t) * kDL + o + j], v);
        x[j] = v * rinv[o + j];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) X[(o + j) * kDL + r] = x[j];
}

// the 8 x 8 block at rows r0, columns c0 of X -= X[r0.., o..o+7] L[c0.., o..o+7]^T (one warp)
__device__ __forceinline__ void d_patch(double* X, const double* L, int r0, int c0, int o) {
    const int lane = threadIdx.x & 31, lo = lane & 3, hi = lane >> 2;
    double* d0 = X + (c0 + 2 * lo) * kDL + r0 + hi;
    double acc[2] = {0.0, 0.0};
#pragma unroll
    for (int kk = 0; kk < 8; kk += 4) d_mma(acc, X[(o + kk + lo) * kDL + r0 + hi], L[(o + kk + lo) * kDL + c0 + hi]);
    d0[0] -= acc[0];
    d0[kDL] -= acc[1];
}

__device__ __forceinline__ void d_panel_sync() { asm volatile("bar.sync 1, 96;" ::: "memory"); }

// S <- L (zeros above the diagonal of each 8 x 8 block), E <- L^-T, by warps 0-2
__device__ __forceinline__ void d_panel(double* S, double* E, double* rinv, double& pmin, double& pmax, int& bad,
                                        int nvalid) {
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    if (w == 0) {
        d_potrf8(S, rinv, 0, pmin, pmax, bad, nvalid);
    } else {
        for (int e = tid - 32; e < kDT * kDT; e += 64) E[(e >> 5) * kDL + (e & 31)] = (e >> 5) == (e & 31) ? 1.0 : 0.0;
    }
    d_panel_sync();
    for (int bb = 0; bb < 4; ++bb) {
        const int o = 8 * bb, c0 = o + 8, nd = kDT - c0;
        if (w == 0) {
            // the rows of S below the block, then rows 0..c0-1 of E (the others hold 0 in it)
            const bool srow = lane < nd;
            d_subst8(srow ? S : E, S, rinv, bb, srow ? c0 + lane : lane - nd);
        }
        d_panel_sync();
        if (bb == 3) break;
        if (w == 0) {
            d_patch(S, S, c0, c0, o);
            __syncwarp();
            d_potrf8(S, rinv, bb + 1, pmin, pmax, bad, nvalid);
        } else {
            // blocks of columns c0..: E's rows 0..c0-1 and S's below the next diagonal block
            int q = w - 1;
            for (int cb = bb + 1; cb < 4; ++cb)
                for (int rb = 0; rb < 4; ++rb) {
                    const bool ep = rb <= bb, sp = rb >= cb && !(rb == bb + 1 && cb == bb + 1);
                    if (!ep && !sp) continue;
                    if (q == 0) d_patch(ep ? E : S, S, 8 * rb, 8 * cb, o);
                    q ^= 1;
                }
        }
        d_panel_sync();
    }
}

// ------------------------------------------------------------------ roles
__device__ void d_diagonal(const DCholCtx& c, DCholSmem& sm) {
    const int T = c.T, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    double pmin = 1.7e308, pmax = 0.0;
    int bad = 0, cur = 0;
    double* E = sm.b[0];
    double* X = sm.b[1];
    d_load(c, sm.a[0], 0, 0, tid, kDThreads);
    d_cp_wait<0>();
    __syncthreads();
    for (int k = 0; k < T; ++k) {
        double* D = sm.a[cur];
        double* Y = sm.a[cur ^ 1];
        const bool more = k + 1 < T;
        if (w == 3) {
            // the next two tiles: their updates through k-1 need no more than step k-1
            int ok = 1;
            if (lane == 0 && k > 0)
                ok = d_poll(c, c.flag + (k + 1) * T + k, 1u, more ? c.flag + (k + 1) * T + k + 1 : nullptr, 1u);
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (lane == 0) sm.ok = ok;
            // a shuffle exchanges registers only: this barrier orders every lane's
            // loads of the two tiles after lane 0's acquire
            __syncwarp();
            if (ok) {
                d_load(c, X, k + 1, k, lane, 32);
                if (more) d_load(c, Y, k + 1, k + 1, lane, 32);
                d_cp_wait<0>();
            }
        } else {
            d_panel(D, E, sm.rinv, pmin, pmax, bad, c.K - k * kDT);
            double* g = c.Dinv + (int64_t)k * kDT * kDT;
            for (int e = tid; e < kDT * kDT / 2; e += 96) {
                const int j = e >> 4, r = (e & 15) * 2;
                __stcg(reinterpret_cast<double2*>(g + j * kDT + r), *reinterpret_cast<const double2*>(E + j * kDL + r));
            }
            d_panel_sync();
            if (tid == 0) d_release(c.flag + k * T + k, 2u);
        }
        __syncthreads();
        if (!sm.ok) break;
        double out[4][2] = {};
        d_product<true>(out, X, E, w, 4);
        __syncthreads();
        d_acc_to(out, X, w);
        __syncthreads();
        d_store(c, X, k + 1, k, tid, kDThreads);
        if (more) {
            double acc[4][2];
            const int lo = lane & 3, hi = lane >> 2;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                acc[j][0] = Y[(8 * j + 2 * lo) * kDL + 8 * w + hi];
                acc[j][1] = Y[(8 * j + 2 * lo + 1) * kDL + 8 * w + hi];
            }
            d_product<false>(acc, X, X, w, w + 1);
            d_acc_to(acc, Y, w, w + 1);
        }
        __syncthreads();
        // by warp 3, whose next work is a wait
        if (tid == 96) d_release(c.flag + (k + 1) * T + k, 2u);
        if (w == 3) d_store(c, D, k, k, lane, 32);
        __syncwarp();
        cur ^= 1;
        // warp 3 reads D (its tile of the step after next) until its next load into it
    }
    if (tid == 0) {
        int f = 0;
        if (bad) f = 1;
        else if (pmax / pmin * c.rcond >= 1.0) f = 2;
        if (f) atomicMax(c.status, f);
        if (c.piv) {
            c.piv[0] = pmin;
            c.piv[1] = pmax;
        }
    }
}

__host__ __device__ __forceinline__ int d_group(int T, int g) { return T - g - 1 + (g + 2 <= T) + (g + 2 <= T - 1); }

__device__ bool d_task(const DCholCtx& c, DCholSmem& sm, int I, int J, int type) {
    const int T = c.T, tid = threadIdx.x, w = tid >> 5, lane = tid & 31, lo = lane & 3, hi = lane >> 2;
    const int kend = type == 0 ? J : I - 1;      // updates k' < kend
    double acc[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) acc[j][e] = d_entry(c, I, J, 8 * w + hi, 8 * j + 2 * lo + e);
    auto fi = [&](int k) { return c.flag + I * T + k; };
    auto fj = [&](int k) -> const unsigned* { return I != J ? c.flag + J * T + k : nullptr; };
    auto fetch = [&](int k) {
        d_load(c, sm.a[k & 1], I, k, tid, kDThreads);
        if (I != J) d_load(c, sm.b[k & 1], J, k, tid, kDThreads);
        else d_commit();
    };
    if (kend > 0) {
        if (!d_wait(c, fi(0), 2u, fj(0), 2u, &sm.ok)) return false;
        fetch(0);
    }
    for (int k = 0; k < kend; ++k) {
        bool next = false;
        if (k + 1 < kend) {
            // the next operands, if they are there, arrive during this product
            __syncthreads();
            if (tid == 0) {
                const unsigned a = d_acquire(fi(k + 1)), b = I != J ? d_acquire(fj(k + 1)) : 2u;
                sm.ok = a >= 2u && b >= 2u;
            }
            __syncthreads();
            next = sm.ok != 0;
            if (next) fetch(k + 1);
        }
        if (next) d_cp_wait<2>();
        else d_cp_wait<0>();
        __syncthreads();
        d_product<false>(acc, sm.a[k & 1], I != J ? sm.b[k & 1] : sm.a[k & 1], w, 4);
        if (k + 1 < kend && !next) {
            if (!d_wait(c, fi(k + 1), 2u, fj(k + 1), 2u, &sm.ok)) return false;
            fetch(k + 1);
        }
    }
    __syncthreads();
    d_acc_to(acc, sm.x, w);
    if (type == 0) {
        if (!d_wait(c, c.flag + J * T + J, 2u, nullptr, 2u, &sm.ok)) return false;
        const double* g = c.Dinv + (int64_t)J * kDT * kDT;
        for (int e = tid; e < kDT * kDT / 2; e += kDThreads) d_cp16(sm.b[0] + (e >> 4) * kDL + (e & 15) * 2, g + 2 * e);
        d_commit();
        d_cp_wait<0>();
        __syncthreads();
        double out[4][2] = {};
        d_product<true>(out, sm.x, sm.b[0], w, 4);
        __syncthreads();
        d_acc_to(out, sm.x, w);
    }
    __syncthreads();
    d_store(c, sm.x, I, J, tid, kDThreads);
    __syncthreads();
    if (tid == 0) d_release(c.flag + I * T + J, type == 0 ? 2u : 1u);
    return true;
}

struct DCholPair {
    DCholCtx c[2];
    int split;           // CTAs of the first system
};

// one system's CTAs: rank 0 the diagonal, the others workers
__device__ __forceinline__ void d_system(const DCholCtx& c, DCholSmem& sm, int rank, int ctas) {
    if (rank == 0) {
        d_diagonal(c, sm);
        return;
    }
    const int W = ctas - 1;
    int t = rank - 1, first = 0;      // tasks before group g
    for (int g = 0; g <= c.T - 2; ++g) {
        const int n = d_group(c.T, g), n0 = c.T - g - 1;
        for (; t < first + n; t += W) {
            const int q = t - first;
            const bool ok = q < n0 ? d_task(c, sm, g + 2 + q, g, 0)
                                   : q == n0 ? d_task(c, sm, g + 2, g + 1, 1) : d_task(c, sm, g + 2, g + 2, 2);
            if (!ok) return;
        }
        first += n;
    }
}

__global__ void __launch_bounds__(kDThreads, kDPerSM) chol64_kernel(DCholCtx c) {
    extern __shared__ __align__(16) uint8_t d_smem[];
    d_system(c, *reinterpret_cast<DCholSmem*>(d_smem), blockIdx.x, gridDim.x);
}

__global__ void __launch_bounds__(kDThreads, kDPerSM) chol64_pair_kernel(const __grid_constant__ DCholPair pair) {
    extern __shared__ __align__(16) uint8_t d_smem[];
    const bool second = (int)blockIdx.x >= pair.split;
    d_system(pair.c[second], *reinterpret_cast<DCholSmem*>(d_smem), blockIdx.x - (second ? pair.split : 0),
             second ? gridDim.x - pair.split : pair.split);
}

// ------------------------------------------------------------------ triangular solves
constexpr unsigned long long kDEmpty = 0xffffffffffffffffull;   // no result has these bits (see the store)

// the word at p once it is written
__device__ __forceinline__ double d_value(const DCholCtx& c, const unsigned long long* p) {
    const volatile unsigned long long* src = p;
    unsigned long long v = *src;
    for (unsigned it = 0; v == kDEmpty; v = *src)
        if (++it > c.limit || *(volatile int*)c.abort_word != 0) {
            atomicExch(c.abort_word, 1);
            atomicMax(c.status, 3);
            break;
        }
    return __longlong_as_double((long long)v);
}

// The factor and the solves multiply by the inverses of the diagonal tiles, which
// is as exact as substituting while the tiles are well conditioned: the same steps
// on the host have 0.6 to 1.0 times the error of LAPACK's solve at a Skeel
// condition number of 300 (the largest of any tile), 1.4 to 2 at 700, 3 to 5 (once
// 56) at 10,000.  Windows that the pivot test accepts at the default rcond have 5
// to 200.  Past the line the caller is told (status -1) and solves with the
// library.
constexpr double kDSkeel = 256.0;

// the Skeel condition number | |L_JJ^-1| |L_JJ| |_inf by one warp: true above the line
__device__ __forceinline__ bool d_skeel(const DCholCtx& c, int J) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, t = J * kDT + lane;
    const double* D = c.Dinv + (int64_t)J * kDT * kDT + lane * kDT;
    double rows = t < c.K ? 0.0 : 1.0, s = 0.0;
    if (t < c.K)
        for (int j = 0; j <= lane; ++j) rows += fabs(__ldcg(c.A + (int64_t)(J * kDT + j) * c.ld + t));
    for (int k = 0; k < kDT; ++k) s = fma(fabs(__ldcg(D + k)), __shfl_sync(full, rows, k), s);
    return __any_sync(full, s > kDSkeel);
}

// Phase p of np: block J's solution into out (and, in the last phase, x); in
// is the phase before, null for x itself.
__global__ void __launch_bounds__(kDThreads) chol64_solve_kernel(DCholCtx c, unsigned long long* words, int backward,
                                                                 int np, int check) {
    __shared__ double s_v[kDT], s_p[4][kDT];
    const unsigned full = 0xffffffffu;
    const int T = c.T, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    for (int p = 0; p < np; ++p, backward ^= 1) {
        unsigned long long* out = words + (int64_t)p * T * kDT;
        const unsigned long long* in = p ? out - (int64_t)T * kDT : nullptr;
        auto rhs = [&](int i) -> double { return in ? d_value(c, in + i) : i < c.K ? __ldcg(c.x + i) : 0.0; };
        for (int b = blockIdx.x; b < T; b += gridDim.x) {
            const int J = backward ? T - 1 - b : b;
            // the tile's condition number while the block would wait, or, for the first blocks, after their hand-off
            auto skeel = [&](bool now) {
                if (check && p == 0 && w == 3 && now && d_skeel(c, J) && lane == 0) atomicCAS(c.status, 0, -1);
            };
            skeel(b >= 8);
            // L_JJ^-1: lane = its column t of the rows 8w.. (backward), its row of the columns 8w.. (forward)
            const double* D = c.Dinv + (int64_t)J * kDT * kDT;
            double di[8], l[8], acc[8] = {};
#pragma unroll
            for (int q = 0; q < 8; ++q) di[q] = __ldcg(backward ? D + (8 * w + q) * kDT + lane : D + lane * kDT + 8 * w + q);
            const int other = backward ? T - 1 : 0, last = backward ? J + 1 : J - 1, step = backward ? -1 : 1;
            const int n = b;                       // blocks before J in this order
            auto fetch = [&](int I) {              // backward: tile (I, J); forward: tile (J, I)
                const int gr = (backward ? I : J) * kDT + lane, gc0 = (backward ? J : I) * kDT + 8 * w;
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    l[q] = gr < c.K && gc0 + q < c.K ? __ldcg(c.A + (int64_t)(gc0 + q) * c.ld + gr) : 0.0;
            };
            if (n) fetch(other);
            for (int k = 0, I = other; k < n; ++k, I += step) {
                if (backward) {                    // acc[q]: this row's part of column 8w + q
                    const double xv = d_value(c, out + I * kDT + lane);
#pragma unroll
                    for (int q = 0; q < 8; ++q) acc[q] = fma(l[q], xv, acc[q]);
                } else {                           // acc[q]: row `lane`, column 8w + q
                    const double xv = d_value(c, out + I * kDT + 8 * w + (lane & 7));
#pragma unroll
                    for (int q = 0; q < 8; ++q) acc[q] = fma(l[q], __shfl_sync(full, xv, q), acc[q]);
                }
                if (I != last) fetch(I + step);
            }
            if (backward) {
                // sums over the warp's lanes: 8 columns -> lane 4q holds column q
#pragma unroll
                for (int h = 4; h >= 1; h >>= 1) {
                    const bool up = lane & (h * 4);
#pragma unroll
                    for (int q = 0; q < h; ++q) {
                        const double give = up ? acc[q] : acc[q + h], keep = up ? acc[q + h] : acc[q];
                        acc[q] = keep + __shfl_xor_sync(full, give, h * 4);
                    }
                }
                acc[0] += __shfl_xor_sync(full, acc[0], 2);
                acc[0] += __shfl_xor_sync(full, acc[0], 1);
                if ((lane & 3) == 0) {
                    const int j = 8 * w + (lane >> 2);
                    s_v[j] = rhs(J * kDT + j) - acc[0];
                }
                __syncwarp();
            } else {
                s_p[w][lane] = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
                __syncthreads();
                if (lane < 8) {                    // each warp the entries it reads below
                    const int j = 8 * w + lane;
                    s_v[j] = rhs(J * kDT + j) - ((s_p[0][j] + s_p[1][j]) + (s_p[2][j] + s_p[3][j]));
                }
                __syncthreads();
            }
            double p0 = 0.0, p1 = 0.0;
#pragma unroll
            for (int q = 0; q < 8; q += 2) {
                p0 = fma(di[q], s_v[8 * w + q], p0);
                p1 = fma(di[q + 1], s_v[8 * w + q + 1], p1);
            }
            s_p[w][lane] = p0 + p1;
            __syncthreads();
            if (w == 0) {
                const double r = (s_p[0][lane] + s_p[1][lane]) + (s_p[2][lane] + s_p[3][lane]);
                unsigned long long bits = (unsigned long long)__double_as_longlong(r);
                if (bits == kDEmpty) bits = 0x7ff8000000000000ull;
                *reinterpret_cast<volatile unsigned long long*>(out + J * kDT + lane) = bits;
                if (p + 1 == np && J * kDT + lane < c.K) c.x[J * kDT + lane] = r;
            }
            skeel(b < 8);
            __syncthreads();
        }
    }
}

static int64_t d_al(int64_t b) { return (b + 255) & ~(int64_t)255; }

// [Dinv][flags][abort word 256][words of the solves' phases]
int64_t chol64_bytes(int K) {
    if (K <= 0) return 0;
    const int64_t T = ceil_div(K, kDT);
    return d_al(T * kDT * kDT * 8) + d_al((T + 1) * T * 4) + 256 + d_al(kChol64Phases * T * kDT * 8);
}

static DCholCtx d_context(const Chol64System& y) {
    DCholCtx c;
    c.A = y.A;
    c.ld = y.ld;
    c.K = y.K;
    c.T = ceil_div(y.K, kDT);
    c.x = y.x;
    char* p = reinterpret_cast<char*>(y.work);
    c.Dinv = reinterpret_cast<double*>(p);
    p += d_al((int64_t)c.T * kDT * kDT * 8);
    c.flag = reinterpret_cast<unsigned*>(p);
    c.abort_word = reinterpret_cast<int*>(p + d_al((int64_t)(c.T + 1) * c.T * 4));
    c.status = y.status;
    c.piv = y.pivots;
    c.rcond = y.rcond;
    c.limit = wait_limit(kDSpin);
    return c;
}

static int d_resident(const void* kernel, size_t smem, int* nsm, int* per_sm) {
    int dev = 0, coop = 0;
    VTB_CUDA_TRY(cudaGetDevice(&dev));
    VTB_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    VTB_CUDA_TRY(cudaDeviceGetAttribute(nsm, cudaDevAttrMultiProcessorCount, dev));
    VTB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    VTB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kernel, kDThreads, smem));
    return coop && *per_sm >= 1 ? VTB_OK : VTB_CUDA_ERR;
}

int chol64_factor(const Chol64System* systems, int n, cudaStream_t s) {
    const size_t sm = sizeof(DCholSmem);
    int nsm = 0, per_sm = 0;
    const void* kernel = n == 1 ? (const void*)chol64_kernel : (const void*)chol64_pair_kernel;
    const int st = d_resident(kernel, sm, &nsm, &per_sm);
    if (st) return st;
    const int room = std::min(per_sm, kDPerSM) * nsm / n;
    DCholPair pair = {};
    int ctas[2] = {0, 0};
    for (int i = 0; i < n; ++i) {
        DCholCtx& c = pair.c[i];
        c = d_context(systems[i]);
        int tasks = 0;
        for (int g = 0; g <= c.T - 2; ++g) tasks += d_group(c.T, g);
        ctas[i] = 1 + std::max(1, std::min(room - 1, tasks));
        VTB_CUDA_TRY(cudaMemsetAsync(c.status, 0, 4, s));
        VTB_CUDA_TRY(cudaMemsetAsync(c.flag, 0, (size_t)(d_al((int64_t)(c.T + 1) * c.T * 4) + 256), s));
    }
    pair.split = ctas[0];
    void* args[] = {n == 1 ? (void*)&pair.c[0] : (void*)&pair};
    VTB_CUDA_TRY(cudaLaunchCooperativeKernel(kernel, dim3(ctas[0] + ctas[1]), dim3(kDThreads), args, sm,
                                             s));
    return launch_status();
}

int chol64_solve(const Chol64System& system, bool backward_first, int phases, bool check, cudaStream_t s) {
    int nsm = 0, per_sm = 0;
    const int st = d_resident((const void*)chol64_solve_kernel, 0, &nsm, &per_sm);
    if (st) return st;
    DCholCtx c = d_context(system);
    unsigned long long* words = reinterpret_cast<unsigned long long*>(reinterpret_cast<char*>(c.abort_word) + 256);
    VTB_CUDA_TRY(cudaMemsetAsync(words, 0xff, (size_t)phases * c.T * kDT * 8, s));
    int first = backward_first, look = check;
    void* args[] = {(void*)&c, (void*)&words, (void*)&first, (void*)&phases, (void*)&look};
    VTB_CUDA_TRY(cudaLaunchCooperativeKernel((void*)chol64_solve_kernel, dim3(std::min(c.T, per_sm * nsm)),
                                             dim3(kDThreads), args, 0, s));
    return launch_status();
}

}  // namespace vtb

using namespace vtb;

VTB_API int64_t vtb_sym_chol_solve_bytes(int K) { return chol64_bytes(K); }

VTB_API int vtb_sym_chol_solve(double* M, int64_t ld, int K, double* x, double rcond, void* work, int64_t work_bytes,
                               int32_t* flag, double* pivots, void* stream) {
    VTB_CHECK_ARG(K > 0 && ld >= K && M && x && work && flag);
    VTB_CHECK_ARG(work_bytes >= chol64_bytes(K) && ((uintptr_t)work & 255) == 0);
    const Chol64System y{M, ld, K, x, work, flag, pivots, rcond};
    const int st = chol64_factor(&y, 1, as_stream(stream));
    return st ? st : chol64_solve(y, true, 1, true, as_stream(stream));
}
