// Reconstruction (synthesis) of the plain float64 decoder.
//
// The reference evaluates, for every voxel, a sum over all spikes of
//   c_k norm_{n_k} phi_{n_k}(x, y) psi_k(t),
//   psi_k(t) = (t_k2 - t_k1) + (2/W) sum_{m=1..Mt} [sin(mW(t-t_k1)) - sin(mW(t-t_k2))]/m
// (reconstruct_Kernel, vtem/dirichlet.py:354-420), O(voxels * spikes * Mt)
// sine evaluations.  The same sum is regrouped here without approximation:
//   psi_k(t) = sum_{|m|<=Mt} conj(T_k(m)) e^{jmWt},
//   T_k(m) = int_{t_k1}^{t_k2} e^{jmWs} ds = (2/(mW)) sin(mW dt_k/2) e^{jmW tbar_k},
// so with beta_n(m) = sum_{k in n} c_k norm_n conj(T_k(m)) (one pass over the
// spikes) the temporal weights are H[t, n] = beta_n(0) + 2 Re sum_{m>=1}
// beta_n(m) e^{jmWt}, and the video is the FP64 GEMM u = H * phi
// (vtb_reconstruct: any sample times, any Mt).
//
// At uniform times the neurons can be summed first instead of last
// (vtb_reconstruct_uniform): the 2Mt+1 spatial weights
//   w_0(p) = sum_n beta_n(0) phi_n(p),  w_{2m-1} + j w_{2m} = 2 sum_n conj(beta_n(m)) phi_n(p)
// are one pass over phi, and the video is their product with the harmonics
// at 2Mt+1 FMAs a voxel instead of N (harmonics_kernel, synth_rank.cu), bound
// by the write of the video.
#include <cooperative_groups.h>

#include "common.cuh"
#include "gemm_f64.cuh"

namespace vtb {

// beta[n][m] (m = 0..Mt, complex interleaved), one warp per neuron.  The
// spike list must be sorted by neuron index (the reference's spike reader
// emits it neuron by neuron, spike_store.py:345-348).
template <int MAXM>
__global__ void beta_kernel(const double* __restrict__ tk1, const double* __restrict__ tk2,
                            const int32_t* __restrict__ ind, const double* __restrict__ c,
                            const double* __restrict__ norm, int nspk, int N, int Mt, double W,
                            double2* __restrict__ beta) {
    const int nr = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (nr >= N) return;
    const int lo = warp_lower_bound(ind, nspk, nr);
    const int hi = warp_lower_bound(ind, nspk, nr + 1);
    double br[MAXM + 1], bi[MAXM + 1];
#pragma unroll
    for (int m = 0; m <= MAXM; ++m) br[m] = bi[m] = 0.0;
    const double nn = norm[nr];
    for (int k = lo + lane; k < hi; k += 32) {
        const double a = tk1[k], b = tk2[k];
        const double w = c[k] * nn;
        const double d = b - a, tb = 0.5 * (a + b);
        br[0] += w * d;
#pragma unroll
        for (int m = 1; m <= MAXM; ++m) {
            if (m > Mt) break;
            const double mw = m * W;
            const double amp = w * (2.0 / mw) * sin(0.5 * mw * d);
            double s, co;
            sincos(mw * tb, &s, &co);
            br[m] += amp * co;   // conj(T) = amp e^{-j mW tbar}
            bi[m] -= amp * s;
        }
    }
#pragma unroll
    for (int m = 0; m <= MAXM; ++m) {
        if (m > Mt) break;
        double r = br[m], i = bi[m];
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            r += __shfl_xor_sync(0xffffffffu, r, o);
            i += __shfl_xor_sync(0xffffffffu, i, o);
        }
        if (lane == 0) beta[(int64_t)nr * (Mt + 1) + m] = make_double2(r, i);
    }
}

// H[t][n] = beta_n(0) + 2 sum_m Re(beta_n(m) e^{jmW t}); one block per time sample
__global__ void h_kernel(const double2* __restrict__ beta, int N, int Mt, double W, const double* __restrict__ t,
                         double* __restrict__ H) {
    extern __shared__ double2 e[];
    const int it = blockIdx.x;
    const double tt = t[it];
    for (int m = threadIdx.x; m <= Mt; m += blockDim.x) {
        double s, c;
        sincos(m * W * tt, &s, &c);
        e[m] = make_double2(c, s);
    }
    __syncthreads();
    for (int nr = threadIdx.x; nr < N; nr += blockDim.x) {
        const double2* b = beta + (int64_t)nr * (Mt + 1);
        double acc = 0.0;
        for (int m = 1; m <= Mt; ++m) acc += b[m].x * e[m].x - b[m].y * e[m].y;
        H[(int64_t)it * N + nr] = b[0].x + 2.0 * acc;
    }
}

// Spatial weights H[p * KT + k] of vtb_reconstruct_uniform.  A cluster of
// kWSplit CTAs covers kWPix pixels, each CTA a contiguous part of the neurons
// in four interleaved groups (one thread per pixel and group, KT sums in
// registers; phi read once, 512 consecutive bytes a row of pixels, the
// coefficients broadcast from shared memory); partial sums are added across
// groups and then across the cluster in a fixed order.  Bound: the HBM read
// of phi.  Measured at N = 1024, 64 x 64 pixels, Mt = 8: 27 us;
// the whole reconstruction of 10,000 frames takes 0.11 ms of device time where
// the N-term product took 7.8 ms (7.7 ms of it the GEMM).
constexpr int kWPix = 64, kWSplit = 8, kWChunk = 32;

template <int KT>
__global__ void __cluster_dims__(kWSplit, 1, 1) __launch_bounds__(4 * kWPix)
    spatial_weights_kernel(const double* __restrict__ dirich, int N, int64_t P, const double2* __restrict__ beta,
                           double* __restrict__ H) {
    namespace cg = cooperative_groups;
    constexpr int MT = (KT - 1) / 2;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    __shared__ __align__(16) double coef[kWChunk][KT + 1];
    __shared__ double part[4][KT][kWPix];
    const int tid = threadIdx.x, px = tid % kWPix, grp = tid / kWPix;
    const int64_t p = (int64_t)(blockIdx.x / kWSplit) * kWPix + px;
    const int per = (N + kWSplit - 1) / kWSplit;
    const int n0 = rank * per, n1 = min(N, n0 + per);
    double acc[KT];
#pragma unroll
    for (int k = 0; k < KT; ++k) acc[k] = 0.0;
    for (int c = n0; c < n1; c += kWChunk) {
        const int nc = min(kWChunk, n1 - c);
        double f[kWChunk / 4];
#pragma unroll
        for (int i = 0; i < kWChunk / 4; ++i)
            f[i] = (p < P && 4 * i + grp < nc) ? __ldg(dirich + (int64_t)(c + 4 * i + grp) * P + p) : 0.0;
        __syncthreads();
        for (int e = tid; e < kWChunk * (MT + 1); e += 4 * kWPix) {
            const int n = e / (MT + 1), m = e % (MT + 1);
            const double2 b = n < nc ? beta[(int64_t)(c + n) * (MT + 1) + m] : make_double2(0.0, 0.0);
            if (m == 0) {
                coef[n][0] = b.x;
            } else {
                coef[n][2 * m - 1] = 2.0 * b.x;
                coef[n][2 * m] = -2.0 * b.y;
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kWChunk / 4; ++i)
            if (4 * i + grp < nc) {
                const double* q = coef[4 * i + grp];
#pragma unroll
                for (int k = 0; k < MT; ++k) {
                    const double2 v = reinterpret_cast<const double2*>(q)[k];
                    acc[2 * k] = fma(f[i], v.x, acc[2 * k]);
                    acc[2 * k + 1] = fma(f[i], v.y, acc[2 * k + 1]);
                }
                acc[KT - 1] = fma(f[i], q[KT - 1], acc[KT - 1]);
            }
    }
#pragma unroll
    for (int k = 0; k < KT; ++k) part[grp][k][px] = acc[k];
    __syncthreads();
    for (int e = tid; e < KT * kWPix; e += 4 * kWPix) {
        double* q = &part[0][0][0] + e;
        q[0] = (q[0] + q[KT * kWPix]) + (q[2 * KT * kWPix] + q[3 * KT * kWPix]);
    }
    cluster.sync();
    for (int e = rank * 4 * kWPix + tid; e < KT * kWPix; e += kWSplit * 4 * kWPix) {
        double v = 0.0;
#pragma unroll
        for (int r = 0; r < kWSplit; ++r) v += cluster.map_shared_rank(&part[0][0][0], r)[e];
        const int64_t q = (int64_t)(blockIdx.x / kWSplit) * kWPix + e % kWPix;
        if (q < P) H[q * KT + e / kWPix] = v;
    }
    cluster.sync();   // the partial sums stay valid until every rank has read them
}

static int launch_beta(const double* tk1, const double* tk2, const int32_t* ind, const double* c, const double* norm,
                       int nspk, int N, int Mt, double WM, double2* beta, cudaStream_t s) {
    const int blocks = ceil_div((int64_t)N * 32, 256);
    if (nspk == 0) {
        VTB_CUDA_TRY(cudaMemsetAsync(beta, 0, (size_t)N * (Mt + 1) * 16, s));
    } else if (Mt <= 8) {
        beta_kernel<8><<<blocks, 256, 0, s>>>(tk1, tk2, ind, c, norm, nspk, N, Mt, WM, beta);
    } else if (Mt <= 16) {
        beta_kernel<16><<<blocks, 256, 0, s>>>(tk1, tk2, ind, c, norm, nspk, N, Mt, WM, beta);
    } else {
        beta_kernel<64><<<blocks, 256, 0, s>>>(tk1, tk2, ind, c, norm, nspk, N, Mt, WM, beta);
    }
    return launch_status();
}

}  // namespace vtb

using namespace vtb;

VTB_API int vtb_reconstruct_workspace(int N, int Nt, int Mt, int64_t* bytes) {
    VTB_CHECK_ARG(N >= 0 && Nt >= 0 && Mt >= 0 && bytes);
    *bytes = (int64_t)N * (Mt + 1) * 16 + (int64_t)Nt * N * 8 + 256;
    return VTB_OK;
}

VTB_API int vtb_reconstruct(const double* dirich, int N, int P, const double* tk1, const double* tk2,
                            const double* c, const int32_t* ind, const double* norm, int nspk, const double* t,
                            int Nt, int Mt, double WM, double* u, void* work, int64_t work_bytes, void* stream) {
    VTB_CHECK_ARG(N > 0 && P > 0 && nspk >= 0 && Nt >= 0 && Mt >= 1 && Mt <= 64);
    if (Nt == 0) return VTB_OK;
    VTB_CHECK_ARG(dirich && norm && t && u && work);
    VTB_CHECK_ARG(nspk == 0 || (tk1 && tk2 && c && ind));
    int64_t need = 0;
    vtb_reconstruct_workspace(N, Nt, Mt, &need);
    VTB_CHECK_ARG(work_bytes >= need);
    cudaStream_t s = as_stream(stream);
    double2* beta = reinterpret_cast<double2*>(work);
    double* H = reinterpret_cast<double*>(reinterpret_cast<char*>(work) + (((int64_t)N * (Mt + 1) * 16 + 255) & ~255));
    int st = launch_beta(tk1, tk2, ind, c, norm, nspk, N, Mt, WM, beta, s);
    if (st) return st;
    h_kernel<<<Nt, 256, (Mt + 1) * sizeof(double2), s>>>(beta, N, Mt, WM, t, H);
    st = launch_status();
    if (st) return st;
    GemmF64Args g{Nt, P, N, H, N, 1, dirich, 1, P, u, P, 1, 1.0, 0.0};
    return gemm_f64(g, s);
}

VTB_API int vtb_reconstruct_uniform_workspace(int N, int P, int Mt, int64_t* bytes) {
    VTB_CHECK_ARG(N >= 0 && P >= 0 && Mt >= 0 && bytes);
    *bytes = (((int64_t)N * (Mt + 1) * 16 + 255) & ~(int64_t)255) + (int64_t)P * (2 * Mt + 1) * 8;
    return VTB_OK;
}

VTB_API int vtb_reconstruct_uniform(const double* dirich, int N, int P, const double* tk1, const double* tk2,
                                    const double* c, const int32_t* ind, const double* norm, int nspk, double t0,
                                    double dt, int Nt, int Mt, double WM, double* u, void* work, int64_t work_bytes,
                                    void* stream) {
    VTB_CHECK_ARG(N > 0 && P > 0 && nspk >= 0 && Nt >= 0 && Mt >= 1 && Mt <= 10);
    if (Nt == 0) return VTB_OK;
    VTB_CHECK_ARG(dirich && norm && u && work && ((uintptr_t)work & 15) == 0);
    VTB_CHECK_ARG(nspk == 0 || (tk1 && tk2 && c && ind));
    int64_t need = 0;
    vtb_reconstruct_uniform_workspace(N, P, Mt, &need);
    VTB_CHECK_ARG(work_bytes >= need);
    cudaStream_t s = as_stream(stream);
    double2* beta = reinterpret_cast<double2*>(work);
    double* H = reinterpret_cast<double*>(reinterpret_cast<char*>(work) + (((int64_t)N * (Mt + 1) * 16 + 255) & ~255));
    int st = launch_beta(tk1, tk2, ind, c, norm, nspk, N, Mt, WM, beta, s);
    if (st) return st;
    const int grid = ceil_div(P, kWPix) * kWSplit;
    switch (Mt) {
        case 1: spatial_weights_kernel<3><<<grid, 4 * kWPix, 0, s>>>(dirich, N, P, beta, H); break;
        case 2: spatial_weights_kernel<5><<<grid, 4 * kWPix, 0, s>>>(dirich, N, P, beta, H); break;
        case 3: spatial_weights_kernel<7><<<grid, 4 * kWPix, 0, s>>>(dirich, N, P, beta, H); break;
        case 4: spatial_weights_kernel<9><<<grid, 4 * kWPix, 0, s>>>(dirich, N, P, beta, H); break;
        case 5: spatial_weights_kernel<11><<<grid, 4 * kWPix, 0, s>>>(dirich, N, P, beta, H); break;
        case 6: spatial_weights_kernel<13><<<grid, 4 * kWPix, 0, s>>>(dirich, N, P, beta, H); break;
        case 7: spatial_weights_kernel<15><<<grid, 4 * kWPix, 0, s>>>(dirich, N, P, beta, H); break;
        case 8: spatial_weights_kernel<17><<<grid, 4 * kWPix, 0, s>>>(dirich, N, P, beta, H); break;
        case 9: spatial_weights_kernel<19><<<grid, 4 * kWPix, 0, s>>>(dirich, N, P, beta, H); break;
        default: spatial_weights_kernel<21><<<grid, 4 * kWPix, 0, s>>>(dirich, N, P, beta, H); break;
    }
    st = launch_status();
    if (st) return st;
    return vtb_synth_harmonics(H, 2 * Mt + 1, P, Mt, WM, t0, dt, Nt, u, 0, stream);
}
