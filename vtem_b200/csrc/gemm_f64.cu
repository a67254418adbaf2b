// Float64 GEMM on the float64 tensor-core path (declared in gemm_f64.cuh).
//
// Bound: the float64 rate, 37.1 TFLOP/s measured for mma m8n8k4 (FMAs alone
// 34.5).  The products are exact float64 FMAs; what the instruction saves
// against a register tile of FMAs is operand traffic: a warp reads MT + NT
// doubles per lane from shared memory for MT x NT products of 8 x 8 x 4.
// Operands arrive by cp.async in ST slabs of 16 k, each operand kept in
// the order in which it is contiguous (k fastest: [row][k], else [k][row]),
// with row strides of 4 mod 16 doubles so that every fragment read is free of
// bank conflicts; 16-byte copies where bases and strides allow, else 8-byte.
// Measured: 10000 x 1024 x 4096 (the GPU configuration's projection) 2.50 ms,
// 33.6 TFLOP/s (7.8 ms, 10.7 with a 4 x 4 register tile per thread of FMAs);
// 2000 x 128 x 1024 27 us (131).  Four warps of 32 x 32 each and three CTAs
// per SM; eight warps of 32 x 16: 2.57 ms; 128 x 64 tiles: 2.77; 96 x 96: 2.69.
#include "gemm_f64.cuh"

#include <cooperative_groups.h>

namespace vtb {

constexpr int kBK = 16, kGemmThreads = 128;

template <int BYTES>
__device__ __forceinline__ void cp_async_fill(double* dst, const double* src, int valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(valid) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(valid) : "memory");
}

// c (16 x 8) += a (16 x 4) b (4 x 8): a lane holds rows lane/4 and lane/4 + 8
// and k = lane%4 of a, column lane/4 of b (the k8 and k16 forms and m8n8k4
// ran at the same rate in this kernel)
__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double b) {
    asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a0), "d"(a1), "d"(b));
}

// How a kernel uses its grid: one CTA a tile; a cluster of gridDim.z CTAs
// sharing a tile's k range; or C = A A^T + beta A (A square and symmetric),
// the tiles of the lower triangle computed and written twice.
enum { kWhole = 0, kSplit = 1, kSym = 2 };

// One operand's slab: ROWS x kBK, KF: k fastest.  V doubles a copy.
template <int ROWS, bool KF, int V>
struct Slab {
    static constexpr int kLd = KF ? kBK + 4 : ROWS + 4;
    static constexpr int kDoubles = KF ? ROWS * kLd : kBK * kLd;
    // element (r, k)
    static __device__ __forceinline__ int at(int r, int k) { return KF ? r * kLd + k : k * kLd + r; }
    static constexpr int kPer = KF ? kBK / V : ROWS / V;         // copies per contiguous run
    static constexpr int kCopies = ROWS * kBK / V;
    static constexpr int kMine = (kCopies + kGemmThreads - 1) / kGemmThreads;
    const double* src[kMine];   // this thread's copies of the next slab
    int valid[kMine];           // bytes inside the operand along its rows (k is cut at the last slab)
    int64_t step;
    const double* base;

    __device__ __forceinline__ void init(const double* X, int64_t x_r, int64_t x_k, int r0, int k0, int R) {
        base = X;
        step = x_k * kBK;
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
            const int e = i * kGemmThreads + threadIdx.x;
            const int r = KF ? e / kPer : (e % kPer) * V, k = KF ? (e % kPer) * V : e / kPer;
            const int left = KF ? (r0 + r < R ? V : 0) : min(max(R - r0 - r, 0), V);
            src[i] = left > 0 ? X + (int64_t)(r0 + r) * x_r + (int64_t)(k0 + k) * x_k : X;
            valid[i] = 8 * left;
        }
    }
    // issue the slab whose first k is k0, of K
    __device__ __forceinline__ void load(double* s, int k0, int K) {
        const bool whole = k0 + kBK <= K;
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
            const int e = i * kGemmThreads + threadIdx.x;
            if (kCopies % kGemmThreads != 0 && e >= kCopies) break;
            const int r = KF ? e / kPer : (e % kPer) * V, k = KF ? (e % kPer) * V : e / kPer;
            int v = valid[i];
            const double* q = src[i];
            if (!whole) {
                const int left = max(K - k0 - k, 0);
                v = KF ? min(v, 8 * left) : (left > 0 ? v : 0);
                if (v == 0) q = base;
            }
            cp_async_fill<8 * V>(s + at(r, k), q, v);
            if (valid[i]) src[i] += step;
        }
    }
};

template <int BM, int BN, int WR, int WC, int ST, bool AKF, bool BKF, int V, int MODE>
__global__ void __launch_bounds__(kGemmThreads, 3) gemm_f64_kernel(GemmF64Args p) {
    constexpr bool SPLIT = MODE == kSplit;
    if (MODE == kSym && blockIdx.x > blockIdx.y) return;   // the mirror of a tile below the diagonal
    using SA = Slab<BM, AKF, V>;
    using SB = Slab<BN, BKF, V>;
    constexpr int MT = BM / WR / 16, NT = BN / WC / 8;
    static_assert(WR * WC * 32 == kGemmThreads && MT * WR * 16 == BM && NT * WC * 8 == BN, "warp tiling");
    extern __shared__ __align__(16) double gemm_sm[];
    double* sa = gemm_sm;
    double* sb = gemm_sm + ST * SA::kDoubles;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int wm = (w % WR) * (BM / WR), wn = (w / WR) * (BN / WC);
    // the CTA's part of k: slabs k_lo .. nk - 1
    const int slabs = (p.K + kBK - 1) / kBK, splits = SPLIT ? gridDim.z : 1;
    const int k_lo = SPLIT ? (int)((int64_t)slabs * blockIdx.z / splits) : 0;
    const int nk = SPLIT ? (int)((int64_t)slabs * (blockIdx.z + 1) / splits) : slabs;
    const int fr = lane >> 2, fk = lane & 3;
    double acc[MT][NT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 4; ++h) acc[i][j][h] = 0.0;
    SA la;
    SB lb;
    la.init(p.A, p.a_m, p.a_k, m0, k_lo * kBK, p.M);
    lb.init(p.B, p.b_n, p.b_k, n0, k_lo * kBK, p.N);
    auto load = [&](int kb, int st) {
        if (kb < nk) {
            la.load(sa + st * SA::kDoubles, kb * kBK, p.K);
            lb.load(sb + st * SB::kDoubles, kb * kBK, p.K);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (int s = 0; s < ST - 1; ++s) load(k_lo + s, s);
    int cur = 0, nxt = ST - 1;   // the ring's places of the slab in use and of the next to be issued
    for (int kb = k_lo; kb < nk; ++kb) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(ST - 2) : "memory");
        __syncthreads();   // slab kb has arrived for every thread; slab kb - 1 has been read by every warp
        load(kb + ST - 1, nxt);
        const double* a = sa + cur * SA::kDoubles;
        const double* b = sb + cur * SB::kDoubles;
        nxt = cur;
        cur = cur + 1 == ST ? 0 : cur + 1;
#pragma unroll
        for (int k = 0; k < kBK; k += 4) {
            double fa[MT][2], fb[NT];
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) fa[i][h] = a[SA::at(wm + 16 * i + 8 * h + fr, k + fk)];
#pragma unroll
            for (int j = 0; j < NT; ++j) fb[j] = b[SB::at(wn + 8 * j + fr, k + fk)];
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int j = 0; j < NT; ++j) dmma(acc[i][j], fa[i][0], fa[i][1], fb[j]);
        }
    }
    auto store = [&](int gm, int gn, double x) {
        if (gm >= p.M || gn >= p.N) return;
        double* c = p.C + (int64_t)gm * p.c_m + (int64_t)gn * p.c_n;
        double v = p.alpha * x;
        if (p.beta != 0.0) v += p.beta * *c;
        *c = v;
    };
    if constexpr (!SPLIT) {
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const int gm = m0 + wm + 16 * i + 8 * (h >> 1) + fr, gn = n0 + wn + 8 * j + 2 * fk + (h & 1);
                    if constexpr (MODE == kSym) {
                        if (gm >= p.M || gn >= p.N) continue;
                        // the addend last: with it first, every one of N terms is rounded to its size
                        const double v = fma(p.beta, p.A[(int64_t)gm * p.a_m + gn], acc[i][j][h]);
                        p.C[(int64_t)gm * p.c_m + gn] = v;
                        if (m0 != n0) p.C[(int64_t)gn * p.c_m + gm] = v;
                    } else {
                        store(gm, gn, acc[i][j][h]);
                    }
                }
    } else {
        // the cluster's partial tiles, each in its CTA's shared memory, added in
        // rank order; CTA r takes the r-th part of the tile, consecutive threads
        // along the contiguous dimension of C
        namespace cg = cooperative_groups;
        cg::cluster_group cluster = cg::this_cluster();
        constexpr int kLdT = BN + 1;
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int h = 0; h < 4; ++h)
                    gemm_sm[(wm + 16 * i + 8 * (h >> 1) + fr) * kLdT + wn + 8 * j + 2 * fk + (h & 1)] = acc[i][j][h];
        cluster.sync();
        const int part = BM * BN / splits;
        for (int e = blockIdx.z * part + threadIdx.x; e < (int)(blockIdx.z + 1) * part; e += kGemmThreads) {
            const int m = p.c_m == 1 ? e % BM : e / BN, n = p.c_m == 1 ? e / BM : e % BN;
            double v = 0.0;
            for (int r = 0; r < splits; ++r) v += cluster.map_shared_rank(gemm_sm, r)[m * kLdT + n];
            store(m0 + m, n0 + n, v);
        }
        cluster.sync();   // the partial tiles stay valid until every CTA has read them
    }
}

template <int BM, int BN, int WR, int WC, int ST, bool AKF, bool BKF, int V>
static int launch_tile(const GemmF64Args& p, int splits, cudaStream_t s) {
    constexpr size_t sm = (size_t)ST * (Slab<BM, AKF, V>::kDoubles + Slab<BN, BKF, V>::kDoubles) * sizeof(double);
    static_assert(sm >= BM * (BN + 1) * sizeof(double), "a partial tile fits the slabs");
    auto kernel = splits > 1 ? gemm_f64_kernel<BM, BN, WR, WC, ST, AKF, BKF, V, kSplit>
                             : gemm_f64_kernel<BM, BN, WR, WC, ST, AKF, BKF, V, kWhole>;
    VTB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ceil_div(p.N, BN), ceil_div(p.M, BM), splits);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {1, 1, (unsigned)splits};
    cfg.attrs = at;
    cfg.numAttrs = splits > 1 ? 1 : 0;
    VTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p));
    return launch_status();
}

// Tile and split of k.  An SM works through its tiles at one rate whatever
// their shape, so the time goes with (CTAs per SM, rounded up) x (a CTA's
// products), plus a tenth for 32 x 32 tiles (twice the operand traffic:
// 5000 x 777 x 2304 takes 616 us with them, 595 with 64 x 64) and two fifths
// for a split k (the exchange of partial tiles: 2000 x 128 x 1024 takes 38 us
// with 64 x 64 tiles split in two, 27 with whole 32 x 32 tiles).  Where even
// the small tiles leave SMs without one, up to kMaxSplit CTAs of a cluster
// share a tile's k range, at least four slabs each and at most one CTA per SM
// in all.  101 x 128 x 1024: 54 us (64 x 64), 23 (32 x 32), 13 (split in eight).
constexpr int kMaxSplit = 8;

static int split_of(int64_t tiles, int slabs) {
    int s = 1;
    while (s < kMaxSplit && tiles * s * 2 <= kNumSMs && slabs >= 4 * s * 2) s *= 2;
    return s;
}

template <bool AKF, bool BKF, int V>
static int launch_layout(const GemmF64Args& p, cudaStream_t s) {
    const int slabs = ceil_div(p.K, kBK);
    const int64_t t64 = (int64_t)ceil_div(p.M, 64) * ceil_div(p.N, 64);
    const int64_t t32 = (int64_t)ceil_div(p.M, 32) * ceil_div(p.N, 32);
    const int s64 = split_of(t64, slabs), s32 = split_of(t32, slabs);
    // CTAs per SM x a CTA's share of a tile
    auto cost = [](int64_t tiles, int split, double unit) {
        return (double)((tiles * split + kNumSMs - 1) / kNumSMs) * unit / split * (split > 1 ? 1.4 : 1.0);
    };
    if (cost(t32, s32, 1.1) < cost(t64, s64, 4.0) && ceil_div(p.M, 32) <= 65535)
        return launch_tile<32, 32, 2, 2, 4, AKF, BKF, V>(p, s32, s);
    return launch_tile<64, 64, 2, 2, 3, AKF, BKF, V>(p, s64, s);
}

int gemm_f64(const GemmF64Args& p, cudaStream_t s) {
    if (p.M <= 0 || p.N <= 0) return VTB_OK;
    if (ceil_div(p.M, 64) > 65535) return VTB_BAD_ARG;
    const bool akf = p.a_k == 1, bkf = p.b_k == 1;
    // 16-byte copies: the fast dimension contiguous, the other stride and the base on 16 bytes
    auto wide = [](const double* x, int64_t fast, int64_t slow) {
        return fast == 1 && slow % 2 == 0 && ((uintptr_t)x & 15) == 0;
    };
    const bool v2 = wide(p.A, akf ? p.a_k : p.a_m, akf ? p.a_m : p.a_k) &&
                    wide(p.B, bkf ? p.b_k : p.b_n, bkf ? p.b_n : p.b_k);
    if (akf && bkf) return v2 ? launch_layout<true, true, 2>(p, s) : launch_layout<true, true, 1>(p, s);
    if (akf) return v2 ? launch_layout<true, false, 2>(p, s) : launch_layout<true, false, 1>(p, s);
    if (bkf) return v2 ? launch_layout<false, true, 2>(p, s) : launch_layout<false, true, 1>(p, s);
    return v2 ? launch_layout<false, false, 2>(p, s) : launch_layout<false, false, 1>(p, s);
}

template <int T, int ST, int V>
static int launch_sym(const GemmF64Args& p, cudaStream_t s) {
    constexpr size_t sm = (size_t)2 * ST * Slab<T, true, V>::kDoubles * sizeof(double);
    auto kernel = gemm_f64_kernel<T, T, 2, 2, ST, true, true, V, kSym>;
    VTB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    kernel<<<dim3(ceil_div(p.N, T), ceil_div(p.M, T)), kGemmThreads, sm, s>>>(p);
    return launch_status();
}

int square_f64(int N, const double* A, int64_t lda, double beta, double* C, int64_t ldc, cudaStream_t s) {
    if (N <= 0) return VTB_OK;
    if (ceil_div(N, 32) > 65535) return VTB_BAD_ARG;
    const GemmF64Args p{N, N, N, A, lda, 1, A, lda, 1, C, ldc, 1, 1.0, beta};
    const bool v2 = lda % 2 == 0 && ((uintptr_t)A & 15) == 0;
    // 64 x 64 tiles come three CTAs to an SM in waves of 444; up to a few waves
    // the ragged last one costs more than the small tiles' operand traffic
    // (N = K = 1921, 496 tiles: 384 us; 1891 tiles of 32 x 32: 285 us)
    const int64_t t = ceil_div(N, 64);
    if (t * (t + 1) / 2 < 12 * kNumSMs) return v2 ? launch_sym<32, 4, 2>(p, s) : launch_sym<32, 4, 1>(p, s);
    return v2 ? launch_sym<64, 3, 2>(p, s) : launch_sym<64, 3, 1>(p, s);
}

}  // namespace vtb
