// RNN (gradient-flow) decoder in the coefficient space.
//
// The reference's rnn3 (vtem/neural_network.py:15-99) runs, from c = 0,
// steps+1 updates c <- c + dt*alpha*(q - G c) on the n x n spike Gram
// G = Phi Phi^H.  The reconstruction only uses a = Phi^H c, and
//     Phi^H c_{i+1} = Phi^H c_i + dt*alpha*(Phi^H q - Phi^H Phi Phi^H c_i),
// so a_{i+1} = a_i + dt*alpha*(b - M a_i) with M = Phi^H Phi, b = Phi^H q:
// the same iterates, on the K x K system instead of n x n (1921 instead of
// ~25k at the GPU configuration).  In the real form (realsys.cu) this is
// x <- x + dt*alpha*(br - Mr x), float64 like the reference.
//
// Two forms.  vtb_rnn_coeff_work, which the decoder uses, squares the update's
// map first and takes what is left of the updates with the matrix in registers
// (further down).  vtb_rnn_coeff takes every update one by one: in one cooperative launch
// each CTA owns a block of rows of Mr, kept in shared memory for the whole run
// when it fits (Mr is read from HBM/L2 once, not once per step), stages the
// previous iterate in shared memory, writes its rows of the next one, and meets
// the other CTAs at a grid barrier.  The barrier's wait is bounded: a CTA that
// waits longer than the limit sets *err and returns (the host reports
// VTB_TIMEOUT).  The same kernel follows the squared form (GUARD) and takes over
// where the updates diverge.
#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "gemm_f64.cuh"

namespace vtb {

constexpr unsigned kRnnSpinLimit = 1u << 24;   // x ~64 ns sleep: about a second
constexpr int kRnnThreads = 256;

// Generation barrier over all CTAs of the launch (cooperative launch: all
// co-resident).  count/gen live in global memory, zeroed before the launch.
__device__ bool rnn_grid_barrier(unsigned* count, unsigned* gen, unsigned nblocks, int* err, unsigned limit) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        volatile unsigned* vgen = gen;
        const unsigned g = *vgen;
        __threadfence();
        if (atomicAdd(count, 1u) == nblocks - 1) {
            atomicExch(count, 0u);
            __threadfence();
            atomicAdd(gen, 1u);
        } else {
            unsigned it = 0;
            while (*vgen == g) {
                if (++it > limit || *(volatile int*)err) {
                    atomicExch(err, 1);
                    ok = 0;
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

// GUARD: x holds the iterate of the squared maps.  An update that contracts
// never lengthens the residual br - Mr x (Mr symmetric: it multiplies each
// eigenvector's part by 1 - dta lambda), so a residual longer than br shows
// updates that diverge, where the squared maps' rounding grows with the number
// of updates that each stands for instead of with its square root (402 updates,
// dta lambda = 2.4 and 3.4: 1.8 times the sum of the updates' own rounding): all
// updates are then taken here, from 0.  Else x stays.  (kRnnGrowth leaves room for
// the residual's own rounding.)  Every CTA takes the sums over all rows in the
// same order and so decides alike.  Measured at K = 1921: 16 us of 2600.
constexpr double kRnnGrowth = 1.0 + 1e-6;

template <bool GUARD>
__global__ void __launch_bounds__(kRnnThreads) rnn_coeff_kernel(const double* __restrict__ Mr, int64_t ld,
                                                                const double* __restrict__ br, double* xa,
                                                                double* xb, int K, double dta, int updates,
                                                                int rows_per_block, int cache_rows,
                                                                unsigned* bar, int* err, unsigned limit,
                                                                const double* x, double* res) {
    extern __shared__ double rnn_sm[];
    double* sx = rnn_sm;                 // K: previous iterate
    double* sM = rnn_sm + K;             // rows_per_block x K (when cache_rows)
    const int r0 = blockIdx.x * rows_per_block;
    const int r1 = min(K, r0 + rows_per_block);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (GUARD) {
        __shared__ double sums[2][kRnnThreads / 32];
        // set by the launch before, or by a CTA that gave up: no one is waited for
        // (all threads of a CTA by one vote: the word may change while they read it)
        if (__syncthreads_or(*(volatile int*)err)) return;
        for (int j = threadIdx.x; j < K; j += blockDim.x) sx[j] = __ldcg(x + j);
        __syncthreads();
        for (int r = r0 + warp; r < r1; r += nw) {
            const double* row = Mr + (int64_t)r * ld;
            double s = 0.0;
#pragma unroll 8
            for (int j = lane; j < K; j += 32) s = fma(row[j], sx[j], s);
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) __stcg(res + r, br[r] - s);
        }
        if (!rnn_grid_barrier(bar, bar + 1, gridDim.x, err, limit)) return;
        double a = 0.0, b = 0.0;
        for (int j = threadIdx.x; j < K; j += blockDim.x) {
            const double r = __ldcg(res + j), q = br[j];
            a = fma(r, r, a);
            b = fma(q, q, b);
        }
        for (int o = 16; o; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        if (lane == 0) {
            sums[0][warp] = a;
            sums[1][warp] = b;
        }
        __syncthreads();
        a = b = 0.0;
        for (int k = 0; k < nw; ++k) {
            a += sums[0][k];
            b += sums[1][k];
        }
        if (a <= kRnnGrowth * b) return;      // (not with a NaN)
    }
    if (cache_rows)
        for (int64_t e = threadIdx.x; e < (int64_t)(r1 - r0) * K; e += blockDim.x) {
            const int r = (int)(e / K), j = (int)(e % K);
            sM[e] = Mr[(int64_t)(r0 + r) * ld + j];
        }
    for (int it = 0; it < updates; ++it) {
        const double* cur = (it & 1) ? xb : xa;
        double* nxt = (it & 1) ? xa : xb;
        for (int j = threadIdx.x; j < K; j += blockDim.x) sx[j] = it ? __ldcg(cur + j) : 0.0;
        __syncthreads();
        for (int r = r0 + warp; r < r1; r += nw) {
            const double* row = cache_rows ? sM + (int64_t)(r - r0) * K : Mr + (int64_t)r * ld;
            double s = 0.0;
            for (int j = lane; j < K; j += 32) s = fma(row[j], sx[j], s);
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) __stcg(nxt + r, sx[r] + dta * (br[r] - s));
        }
        if (!rnn_grid_barrier(bar, bar + 1, gridDim.x, err, limit)) return;
    }
}

// ---------------------------------------------------------------------------
// Many updates with few exchanges (vtb_rnn_coeff_work).
//
// An update is the affine map x -> x + D x + S with D = -h Mr, S = h br, and
// 2^j of them are the map with D_j = D_{j-1}^2 + 2 D_{j-1}, S_j = D_{j-1}
// S_{j-1} + 2 S_{j-1}; all are polynomials in Mr, so they commute.  (D is the
// map less the identity: where h lambda is small, 1 - h lambda would keep only
// the absolute precision of h lambda.)  U = steps + 1 updates are therefore:
// for the s low bits of U, lowest first, the map of that bit if it is set,
// then one squaring; after them U >> s updates by D_s.  The squarings are
// float64 tensor-path products of one triangle (square_f64, 0.29 ms at
// K = 1921), the maps one pass over D (both right-hand sides at once), the
// remaining updates one launch with D_s in registers (below).  An update by
// itself costs an exchange between all SMs, 5 to 7 us whatever K is, so s is
// chosen by cost (rnn_levels).
// Measured at K = 1921, 2001 updates: 15.1 ms one update at a time,
// 2.0 ms here (five squarings and 62 updates).

__global__ void rnn_map_kernel(const double* __restrict__ Mr, int64_t ld, const double* __restrict__ br, int K, double h,
                               double* __restrict__ P, int64_t ldp, double* __restrict__ S, double* __restrict__ x) {
    const int r = blockIdx.y;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < K; j += gridDim.x * blockDim.x) {
        P[(int64_t)r * ldp + j] = -h * Mr[(int64_t)r * ld + j];
        if (r == 0) {
            S[j] = h * br[j];
            x[j] = 0.0;
        }
    }
}

// x_out = x + P x + S where `apply` (else x), S_out = P S + 2 S: one warp a row
__global__ void __launch_bounds__(256) rnn_apply_kernel(const double* __restrict__ P, int64_t ldp, int K,
                                                        const double* __restrict__ S, const double* __restrict__ x,
                                                        int apply, double* __restrict__ S_out, double* __restrict__ x_out) {
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (r >= K) return;
    const double* row = P + (int64_t)r * ldp;
    // the addends first, each row one chain of FMAs
    double s[2] = {lane == 0 ? 2.0 * S[r] : 0.0, 0.0}, t[2] = {lane == 0 ? S[r] : 0.0, 0.0};
    int j = lane;
    for (; j + 32 < K; j += 64) {
        const double a = row[j], b = row[j + 32];
        s[0] = fma(a, S[j], s[0]);
        s[1] = fma(b, S[j + 32], s[1]);
        t[0] = fma(a, x[j], t[0]);
        t[1] = fma(b, x[j + 32], t[1]);
    }
    if (j < K) {
        s[0] = fma(row[j], S[j], s[0]);
        t[0] = fma(row[j], x[j], t[0]);
    }
    double u = s[0] + s[1], v = t[0] + t[1];
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        u += __shfl_xor_sync(0xffffffffu, u, o);
        v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    if (lane == 0) {
        S_out[r] = u;
        x_out[r] = apply ? x[r] + v : x[r];
    }
}

// The updates x -> x + P x + S (from a given x) in one launch with P in registers.
//
// CTA b owns rows b*R .. b*R+R-1; thread t holds their columns t, t+512, ...
// (RR rows in registers, the other RS in shared memory), so an update reads
// no matrix from anywhere else.  The iterate travels as 16-byte packets
// (value, update number), written and read by single 128-bit accesses: a
// thread polls the packets of its own columns until they carry the update it
// needs.  Packets alternate between two buffers: a CTA writes update u + 1
// only after it has read every packet of update u, whose writers had all read
// update u - 1, the buffer's previous content.  All CTAs are co-resident
// (cooperative launch); every wait is bounded, and a wait that runs out sets
// *err and ends all CTAs.  Bound: the exchange (7.3 us an update, as with a
// grid barrier: every SM reads the whole iterate from the same few L2 lines).
constexpr int kRnnRegThreads = 512;
constexpr unsigned kRnnPollLimit = 1u << 21;

__device__ __forceinline__ void ld_packet(const ulonglong2* p, double& v, unsigned long long& u) {
    unsigned long long lo, hi;
    asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
                 : "=l"(lo), "=l"(hi)
                 : "l"(p)
                 : "memory");
    v = __longlong_as_double((long long)lo);
    u = hi;
}

__device__ __forceinline__ void st_packet(ulonglong2* p, double v, unsigned long long u) {
    asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"(u)
                 : "memory");
}

// v[0..15] summed over the warp: lane l returns the total of v[l & 15]
__device__ __forceinline__ double warp_reduce16(double (&v)[16]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < o; ++k) {
            const double send = up ? v[k] : v[k + o];
            const double keep = up ? v[k + o] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
}

template <int RR, int RS, int C>
__global__ void __launch_bounds__(kRnnRegThreads, 1) rnn_reg_kernel(const double* __restrict__ P, int64_t ld,
                                                                    const double* __restrict__ S, double* x, int K,
                                                                    int updates, ulonglong2* packets, int* err,
                                                                    unsigned limit) {
    constexpr int R = RR + RS, NW = kRnnRegThreads / 32;
    static_assert(R <= 16, "a warp reduces sixteen rows");
    extern __shared__ double rnn_rows[];           // RS x C x 512
    __shared__ double red[2][NW][16];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int r0 = blockIdx.x * R;
    double m[RR][C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const int j = tid + c * kRnnRegThreads;
#pragma unroll
        for (int r = 0; r < RR; ++r) m[r][c] = r0 + r < K && j < K ? P[(int64_t)(r0 + r) * ld + j] : 0.0;
#pragma unroll
        for (int r = 0; r < RS; ++r)
            rnn_rows[(r * C + c) * kRnnRegThreads + tid] =
                r0 + RR + r < K && j < K ? P[(int64_t)(r0 + RR + r) * ld + j] : 0.0;
    }
    const bool owner = tid < R && r0 + tid < K;
    const double b = owner ? S[r0 + tid] : 0.0;
    double xi = owner ? x[r0 + tid] : 0.0;
    for (int it = 0; it < updates; ++it) {
        const ulonglong2* cur = packets + (size_t)(it & 1) * K;   // update 0: x itself, from rnn_packets_kernel
        double v[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) v[r] = 0.0;
        double xv[C];
        unsigned long long u[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int j = tid + c * kRnnRegThreads;
            xv[c] = 0.0;
            u[c] = (unsigned long long)it;
            if (j < K) ld_packet(cur + j, xv[c], u[c]);
        }
        bool dead = false;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            unsigned polls = 0;
            while (u[c] != (unsigned long long)it) {
                if (++polls > limit || ((polls & 1023u) == 0 && *(volatile int*)err)) {
                    atomicExch(err, 1);
                    dead = true;
                    break;
                }
                ld_packet(cur + tid + c * kRnnRegThreads, xv[c], u[c]);
            }
#pragma unroll
            for (int r = 0; r < RR; ++r) v[r] = fma(m[r][c], xv[c], v[r]);
#pragma unroll
            for (int r = 0; r < RS; ++r)
                v[RR + r] = fma(rnn_rows[(r * C + c) * kRnnRegThreads + tid], xv[c], v[RR + r]);
        }
        const double s = warp_reduce16(v);
        if (lane < 16) red[it & 1][w][lane] = s;
        if (__syncthreads_or(dead)) return;
        if (owner) {
            double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int k = 0; k < NW; ++k) t[k & 3] += red[it & 1][k][tid];
            xi = xi + (((t[0] + t[1]) + (t[2] + t[3])) + b);
            st_packet(packets + (size_t)((it + 1) & 1) * K + r0 + tid, xi, (unsigned long long)(it + 1));
        }
    }
    if (owner) x[r0 + tid] = xi;
}

__global__ void rnn_packets_kernel(const double* __restrict__ x, int K, ulonglong2* __restrict__ packets) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 2 * K) packets[i] = make_ulonglong2(i < K ? (unsigned long long)__double_as_longlong(x[i]) : 0ull, 0ull);
}

template <int RR, int RS, int C>
static int launch_rnn_reg(const double* P, int64_t ld, const double* S, double* x, int K, int updates,
                          ulonglong2* packets, int* err, int nsm, cudaStream_t s) {
    auto kernel = rnn_reg_kernel<RR, RS, C>;
    const size_t sm = (size_t)RS * C * kRnnRegThreads * sizeof(double);
    VTB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    int per_sm = 0;
    VTB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kRnnRegThreads, sm));
    const int blocks = ceil_div(K, RR + RS);
    if (per_sm * nsm < blocks) return VTB_CUDA_ERR;
    unsigned limit = wait_limit(kRnnPollLimit);
    void* args[] = {(void*)&P, (void*)&ld, (void*)&S, (void*)&x, (void*)&K,
                    (void*)&updates, (void*)&packets, (void*)&err, (void*)&limit};
    rnn_packets_kernel<<<ceil_div(2 * K, 256), 256, 0, s>>>(x, K, packets);
    VTB_CUDA_TRY(cudaLaunchCooperativeKernel((void*)kernel, dim3(blocks), dim3(kRnnRegThreads), args, sm, s));
    return launch_status();
}

}  // namespace vtb

using namespace vtb;

// SM count and opt-in shared memory of the current device (attribute queries:
// reading the whole property record costs most of a millisecond a call)
static int rnn_device(int* nsm, int* smem_max) {
    int dev = 0, coop = 0;
    VTB_CUDA_TRY(cudaGetDevice(&dev));
    VTB_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    VTB_CUDA_TRY(cudaDeviceGetAttribute(nsm, cudaDevAttrMultiProcessorCount, dev));
    VTB_CUDA_TRY(cudaDeviceGetAttribute(smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    return coop ? VTB_OK : VTB_CUDA_ERR;
}

// One launch of rnn_coeff_kernel (bar: 2 unsigned, then the error word, zeroed by
// the caller); VTB_BAD_ARG where K doubles exceed a block's shared memory.
template <bool GUARD>
static int launch_rnn_updates(const double* Mr, int64_t ld, const double* br, double* xa, double* xb, int K,
                              double dt_alpha, int updates, unsigned* bar, const double* x, double* res, int nsm,
                              int smem_max, cudaStream_t s) {
    auto kernel = rnn_coeff_kernel<GUARD>;
    int rows = (K + nsm - 1) / nsm;
    int blocks = (K + rows - 1) / rows;
    size_t sm = (size_t)K * 8 + (size_t)rows * K * 8;
    int cache = 1;
    cudaFuncAttributes fa;
    VTB_CUDA_TRY(cudaFuncGetAttributes(&fa, kernel));
    smem_max -= (int)fa.sharedSizeBytes;
    if (sm > (size_t)smem_max) {
        cache = 0;
        sm = (size_t)K * 8;
        VTB_CHECK_ARG(sm <= (size_t)smem_max);
    }
    // (the limit is the kernel's, not the call's: always the same one)
    VTB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max));
    int per_sm = 0;
    VTB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kRnnThreads, sm));
    if (per_sm * nsm < blocks) return VTB_CUDA_ERR;
    int* err = reinterpret_cast<int*>(bar + 2);
    unsigned limit = wait_limit(kRnnSpinLimit);
    void* args[] = {(void*)&Mr, (void*)&ld, (void*)&br, (void*)&xa, (void*)&xb, (void*)&K, (void*)&dt_alpha,
                    (void*)&updates, (void*)&rows, (void*)&cache, (void*)&bar, (void*)&err, (void*)&limit,
                    (void*)&x, (void*)&res};
    VTB_CUDA_TRY(cudaLaunchCooperativeKernel((void*)kernel, dim3(blocks), dim3(kRnnThreads), args, sm, s));
    return launch_status();
}

// x (K doubles, device) receives the iterate after steps+1 updates from x = 0;
// x_tmp (K doubles) and bar (2 unsigned + 1 int of scratch, 16 bytes) are
// caller-owned scratch.  Replaces rnn3 + rnn3_update (vtem/neural_network.py:
// 15-128) on the real coefficient system.  Synchronises nothing; an
// exceeded barrier wait is reported in bar's third word.
VTB_API int vtb_rnn_coeff(const double* Mr, int64_t ld, const double* br, double* x, double* x_tmp, int K,
                          double dt_alpha, int steps, void* bar, void* stream) {
    VTB_CHECK_ARG(K > 0 && ld >= K && steps >= 0 && Mr && br && x && x_tmp && bar);
    int nsm = 0, smem_max = 0;
    int st = rnn_device(&nsm, &smem_max);
    if (st) return st;
    cudaStream_t s = as_stream(stream);
    VTB_CUDA_TRY(cudaMemsetAsync(bar, 0, 16, s));
    const int updates = steps + 1;
    // the last of an even number of updates writes the first buffer
    double* xa = updates & 1 ? x_tmp : x;
    double* xb = updates & 1 ? x : x_tmp;
    return launch_rnn_updates<false>(Mr, ld, br, xa, xb, K, dt_alpha, updates, reinterpret_cast<unsigned*>(bar), nullptr,
                                     nullptr, nsm, smem_max, s);
}

constexpr int kRnnGuardMax = 28000;

// Workspace of vtb_rnn_coeff_work, every part on 256 bytes: status words,
// packets, two of S and x, two of P (rows padded to 16 bytes).
struct RnnWork {
    int* status;
    ulonglong2* packets;
    double *S[2], *x[2], *P[2];
    int64_t ldp, bytes;
};

static RnnWork rnn_work(int K, char* base) {
    RnnWork w;
    int64_t off = 0;
    auto take = [&](int64_t bytes) {
        char* p = base + off;
        off += (bytes + 255) & ~(int64_t)255;
        return p;
    };
    w.ldp = (K + 1) & ~1;
    w.status = reinterpret_cast<int*>(take(16));
    w.packets = reinterpret_cast<ulonglong2*>(take(2 * (int64_t)K * 16));
    for (int i = 0; i < 2; ++i) w.S[i] = reinterpret_cast<double*>(take((int64_t)K * 8));
    for (int i = 0; i < 2; ++i) w.x[i] = reinterpret_cast<double*>(take((int64_t)K * 8));
    for (int i = 0; i < 2; ++i) w.P[i] = reinterpret_cast<double*>(take((int64_t)K * w.ldp * 8));
    w.bytes = off;
    return w;
}

// Squarings before the remaining updates run one by one, by cost in us: a
// squaring with its pass over P (15 + K^3 / 2.5e7: 300 measured at
// K = 1921) against an exchange (7.3 measured at K = 1921, 5.5 at 261).
static int rnn_levels(int K, int updates) {
    const double square = 15.0 + (double)K * K * K / 2.5e7, exchange = 7.3;
    int best = 0;
    for (int s = 1; (updates >> s) > 0; ++s)
        if (s * square + (updates >> s) * exchange < best * square + (updates >> best) * exchange) best = s;
    return best;
}

VTB_API int vtb_rnn_coeff_workspace(int K, int64_t* bytes) {
    VTB_CHECK_ARG(K > 0 && bytes);
    *bytes = rnn_work(K, nullptr).bytes;
    return VTB_OK;
}

VTB_API int vtb_rnn_coeff_work(const double* Mr, int64_t ld, const double* br, double* x, int K, double dt_alpha,
                               int steps, void* work, int64_t work_bytes, void* stream) {
    VTB_CHECK_ARG(K > 0 && ld >= K && steps >= 0 && Mr && br && x && work && ((uintptr_t)work & 255) == 0);
    const RnnWork w = rnn_work(K, reinterpret_cast<char*>(work));
    VTB_CHECK_ARG(work_bytes >= w.bytes && K <= 65535);
    int nsm = 0, smem_max = 0;
    int st = rnn_device(&nsm, &smem_max);
    if (st) return st;
    cudaStream_t s = as_stream(stream);
    // none where the guard's kernel could not hold the iterate in shared memory
    const int updates = steps + 1, levels = K <= kRnnGuardMax ? rnn_levels(K, updates) : 0;
    VTB_CUDA_TRY(cudaMemsetAsync(w.status, 0, 16, s));
    rnn_map_kernel<<<dim3(ceil_div(K, 1024), K), 256, 0, s>>>(Mr, ld, br, K, dt_alpha, w.P[0], w.ldp, w.S[0], w.x[0]);
    int cur = 0;
    const int rows_grid = ceil_div((int64_t)K * 32, 256);
    for (int j = 0; j < levels; ++j, cur ^= 1) {
        rnn_apply_kernel<<<rows_grid, 256, 0, s>>>(w.P[cur], w.ldp, K, w.S[cur], w.x[cur], (updates >> j) & 1,
                                                   w.S[cur ^ 1], w.x[cur ^ 1]);
        st = square_f64(K, w.P[cur], w.ldp, 2.0, w.P[cur ^ 1], w.ldp, s);
        if (st) return st;
    }
    const int left = updates >> levels, rows = ceil_div(K, nsm);
    double* xc = w.x[cur];
    const double *P = w.P[cur], *S = w.S[cur];
    // the squared maps' iterate into x, and the check that it is no diverging one
    double *res = w.S[cur ^ 1], *tmp = w.S[cur];
    auto finish = [&](const double* from) -> int {
        VTB_CUDA_TRY(cudaMemcpyAsync(x, from, (size_t)K * 8, cudaMemcpyDeviceToDevice, s));
        if (levels == 0) return launch_status();
        return launch_rnn_updates<true>(Mr, ld, br, updates & 1 ? tmp : x, updates & 1 ? x : tmp, K, dt_alpha, updates,
                                        reinterpret_cast<unsigned*>(w.status), x, res, nsm, smem_max, s);
    };
    // more rows than registers and shared memory hold: one pass over P an update
    if (rows > 13 || K > 4 * kRnnRegThreads || left == 1) {
        double* unused = w.S[cur ^ 1];
        for (int i = 0; i < left; ++i, cur ^= 1)
            rnn_apply_kernel<<<rows_grid, 256, 0, s>>>(P, w.ldp, K, S, w.x[cur], 1, unused, w.x[cur ^ 1]);
        return finish(w.x[cur]);
    }
    if (rows <= 2 && K <= kRnnRegThreads) st = launch_rnn_reg<2, 0, 1>(P, w.ldp, S, xc, K, left, w.packets, w.status + 2, nsm, s);
    else if (rows <= 4 && K <= 2 * kRnnRegThreads)
        st = launch_rnn_reg<4, 0, 2>(P, w.ldp, S, xc, K, left, w.packets, w.status + 2, nsm, s);
    else if (rows <= 7 && K <= 3 * kRnnRegThreads)
        st = launch_rnn_reg<7, 0, 3>(P, w.ldp, S, xc, K, left, w.packets, w.status + 2, nsm, s);
    else if (rows <= 10 && K <= 3 * kRnnRegThreads)
        st = launch_rnn_reg<10, 0, 3>(P, w.ldp, S, xc, K, left, w.packets, w.status + 2, nsm, s);
    else
        st = launch_rnn_reg<10, 3, 4>(P, w.ldp, S, xc, K, left, w.packets, w.status + 2, nsm, s);
    return st ? st : finish(xc);
}
