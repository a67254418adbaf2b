// Dirichlet-space kernels of the plain float64 decoder.
//
//  vtb_dirichlet_coeffs : Ds[n, My-my, mx+Mx] = dxdy (-1)^(mx+my) DFT2(RF_n)
//      restricted to the spatial ellipse (compute_Ds + fft2Ds_kernel,
//      vtem/vrf.py:333-377, :1293-1350).  Only (2Mx+1)(2My+1) of the
//      LPy*LPx frequencies are ever used, so instead of a full 2-D FFT the
//      kernels evaluate a separable DFT for just those bins against exact
//      twiddle tables (sincospi of integer ratios).
//  vtb_dirich_space : phi_n on the decode grid, equal to the reference's
//      unnormalised inverse FFT on the (Py1, Px1) period grid followed by the
//      centred crop (compute_dirich_space_fft, vrf.py:437-499, :585-677),
//      evaluated as a separable direct sum over the nonzero bins.
//  vtb_dsw : Dsw = Re(Ds Ds^H) scaled by norm_a norm_b (compute_Dsw + put_norm,
//      vrf.py:502-559), as one real GEMM over the interleaved (re, im) planes.
//  vtb_compute_q : compute_q_Kernel (vtem/dirichlet.py:204-222).
//  vtb_compute_G : compute_G_Kernel + diag_add_Kernel (dirichlet.py:272-350),
//      the same entries as products of the intervals' harmonics.
#include <algorithm>

#include "common.cuh"
#include "gemm_f64.cuh"

namespace vtb {

// ---------------------------------------------------------------- Ds (DFT)

// The same coefficients on the float64 tensor path, for up to 16 bins each way
// (2Mx+1, 2My+1 <= 16).  An RF is real, so the bins of +-m are the sums with
// cos and sin of |m|: 2M+1 real columns each way, at most 16.  A block takes
// one RF at a time (persistent over the RFs, the cos/sin tables formed once):
//   R = RF (rows x px) * X (px x 16): a warp per 16 rows, the RF's fragments
//       straight from global memory (whole sectors, read once), X from shared
//       memory;
//   S = Y^T (16 x rows) * R: the rows split over the warps, the partial sums
//       added in warp order;
// then the four real sums of each |my|, |mx| give its (up to) four bins.
// Bound: the HBM read of the RFs (537 MB at 1024 RFs of 256 x 256, 82 us).
// A lane's fragment holds the pixels 2q and 2q + 1 of a step's eight (16-byte
// loads where rows allow), so both products take k in that order.  Measured at
// that size: 2306 us with a dot product per bin and row, 125 here.
constexpr int kDfWarps = 8;
constexpr int kDfS = 18;        // row stride of tables and R: fragment reads free of bank conflicts

__device__ __forceinline__ void df_mma(double (&c)[4], double a0, double a1, double b) {
    asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a0), "d"(a1), "d"(b));
}

// t[p * kDfS + col]: col 0 = 1, 2b - 1 = cos(2 pi b p / L), 2b = sin(2 pi b p / L), b <= M; zero elsewhere
__device__ void df_table(int L, int Lpad, int M, double* __restrict__ t) {
    for (int e = threadIdx.x; e < Lpad * 9; e += blockDim.x) {
        const int p = e / 9, b = e % 9;
        double s = 0.0, c = 0.0;
        if (p < L && b <= M) sincospi(2.0 * (double)(((int64_t)b * p) % L) / L, &s, &c);
        if (b == 0) {
            t[p * kDfS] = c;
        } else if (b < 8) {
            t[p * kDfS + 2 * b - 1] = c;
            t[p * kDfS + 2 * b] = s;
        } else {
            t[p * kDfS + 15] = 0.0;
        }
    }
}

template <bool VEC>
__global__ void __launch_bounds__(kDfWarps * 32) ds_mma_kernel(const double* __restrict__ rf, int64_t rf_ld, int N,
                                                               int LPy, int LPx, int Mx, int My, double dxdy,
                                                               double2* __restrict__ Ds) {
    extern __shared__ double dsm[];
    const int Xp = (LPx + 7) & ~7, Yp = (LPy + 15) & ~15;
    double* R = dsm;                               // Yp x kDfS
    double* ty = R + (size_t)Yp * kDfS;            // Yp x kDfS
    double* tx = LPx == LPy && Mx == My ? ty : ty + (size_t)Yp * kDfS;   // Xp x kDfS
    __shared__ double part[kDfWarps][16 * 16];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int fr = lane >> 2, fq = lane & 3;
    df_table(LPy, Yp, My, ty);
    if (tx != ty) df_table(LPx, Xp, Mx, tx);
    const int Kx = 2 * Mx + 1, Ky = 2 * My + 1;
    for (int n = blockIdx.x; n < N; n += gridDim.x) {
        __syncthreads();                           // tables formed; the last RF's sums have been read
        const double* src = rf + (int64_t)n * rf_ld;
        for (int r0 = 16 * w; r0 < Yp; r0 += 16 * kDfWarps) {
            double acc[2][4];
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int h = 0; h < 4; ++h) acc[j][h] = 0.0;
            const bool in0 = r0 + fr < LPy, in1 = r0 + fr + 8 < LPy;
            const double* p0 = src + (int64_t)(in0 ? r0 + fr : 0) * LPx + 2 * fq;
            const double* p1 = src + (int64_t)(in1 ? r0 + fr + 8 : 0) * LPx + 2 * fq;
            constexpr int kU = 4;                  // steps of eight pixels whose loads are issued together
            for (int x0 = 0; x0 < Xp; x0 += 8 * kU) {
                double2 v0[kU], v1[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const int x = x0 + 8 * u, c = x + 2 * fq;
                    v0[u] = v1[u] = make_double2(0.0, 0.0);
                    if (VEC) {                     // LPx even: a pair is whole or outside
                        if (c < LPx) {
                            if (in0) v0[u] = __ldcs(reinterpret_cast<const double2*>(p0 + x));
                            if (in1) v1[u] = __ldcs(reinterpret_cast<const double2*>(p1 + x));
                        }
                    } else {
                        if (c < LPx) {
                            if (in0) v0[u].x = __ldcs(p0 + x);
                            if (in1) v1[u].x = __ldcs(p1 + x);
                        }
                        if (c + 1 < LPx) {
                            if (in0) v0[u].y = __ldcs(p0 + x + 1);
                            if (in1) v1[u].y = __ldcs(p1 + x + 1);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const int x = x0 + 8 * u;
                    if (x >= Xp) break;
                    const double* t = tx + (size_t)(x + 2 * fq) * kDfS + fr;
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        df_mma(acc[j], v0[u].x, v1[u].x, t[8 * j]);
                        df_mma(acc[j], v0[u].y, v1[u].y, t[kDfS + 8 * j]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int h = 0; h < 4; ++h)
                    R[(size_t)(r0 + fr + 8 * (h >> 1)) * kDfS + 8 * j + 2 * fq + (h & 1)] = acc[j][h];
        }
        __syncthreads();
        {
            double acc[2][4];
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int h = 0; h < 4; ++h) acc[j][h] = 0.0;
            for (int y = 8 * w; y < Yp; y += 8 * kDfWarps) {
                const double* t = ty + (size_t)(y + 2 * fq) * kDfS + fr;
                const double* r = R + (size_t)(y + 2 * fq) * kDfS + fr;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    df_mma(acc[j], t[0], t[8], r[8 * j]);
                    df_mma(acc[j], t[kDfS], t[kDfS + 8], r[kDfS + 8 * j]);
                }
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int h = 0; h < 4; ++h)
                    part[w][(fr + 8 * (h >> 1)) * 16 + 8 * j + 2 * fq + (h & 1)] = acc[j][h];
        }
        __syncthreads();
        {
            double v = part[0][tid];
#pragma unroll
            for (int k = 1; k < kDfWarps; ++k) v += part[k][tid];
            part[0][tid] = v;
        }
        __syncthreads();
        if (tid < Kx * Ky) {
            const int mx = tid % Kx - Mx, my = My - tid / Kx;      // storage row holds my = My - row
            double2 out = make_double2(0.0, 0.0);
            if ((int64_t)mx * mx * My * My + (int64_t)my * my * Mx * Mx <= (int64_t)Mx * Mx * My * My) {
                const int b = abs(mx), a = abs(my);
                const int rc = a ? 2 * a - 1 : 0, cc = b ? 2 * b - 1 : 0;
                const double* S = part[0];
                const double Cc = S[rc * 16 + cc];
                const double Sc = a ? S[(rc + 1) * 16 + cc] : 0.0, Cs = b ? S[rc * 16 + cc + 1] : 0.0;
                const double Ss = a && b ? S[(rc + 1) * 16 + cc + 1] : 0.0;
                const double ya = my < 0 ? -1.0 : 1.0, xb = mx < 0 ? -1.0 : 1.0;
                const double sgn = ((mx + my) % 2 == 0) ? dxdy : -dxdy;
                out = make_double2(sgn * (Cc - ya * xb * Ss), -sgn * (ya * Sc + xb * Cs));
            }
            Ds[(int64_t)n * Kx * Ky + tid] = out;
        }
    }
}

constexpr int kDsRows = 16;

// Any bin count (2Mx+1)(2My+1) <= 256: a dot product per bin and row.
__global__ void __launch_bounds__(256) ds_kernel(const double* __restrict__ rf, int64_t rf_ld, int LPy, int LPx,
                                                  int Mx, int My, double dxdy, double2* __restrict__ Ds) {
    extern __shared__ double smem[];
    const int Kx = 2 * Mx + 1, Ky = 2 * My + 1;
    double2* twx = reinterpret_cast<double2*>(smem);               // LPx entries: e^{-2 pi i r / LPx}
    double2* twy = twx + LPx;                                        // LPy entries
    double* rows = reinterpret_cast<double*>(twy + LPy);             // kDsRows x LPx
    double2* R = reinterpret_cast<double2*>(rows + kDsRows * LPx);   // kDsRows x Kx
    const int n = blockIdx.x;
    const int tid = threadIdx.x;
    for (int r = tid; r < LPx; r += blockDim.x) {
        double s, c;
        sincospi(2.0 * r / LPx, &s, &c);
        twx[r] = make_double2(c, -s);
    }
    for (int r = tid; r < LPy; r += blockDim.x) {
        double s, c;
        sincospi(2.0 * r / LPy, &s, &c);
        twy[r] = make_double2(c, -s);
    }
    // accumulator of F(my, mx) owned by thread tid < Kx*Ky
    double accr = 0.0, acci = 0.0;
    const int my_t = tid / Kx - My, mx_t = tid % Kx - Mx;
    const double* src = rf + (int64_t)n * rf_ld;
    for (int py0 = 0; py0 < LPy; py0 += kDsRows) {
        const int nr = min(kDsRows, LPy - py0);
        __syncthreads();
        for (int e = tid; e < nr * LPx; e += blockDim.x) rows[e] = src[(int64_t)py0 * LPx + e];
        __syncthreads();
        // row DFT at the Kx bins: R[row][mx] = sum_px rows[row][px] e^{-2 pi i mx px / LPx}
        for (int o = tid; o < nr * Kx; o += blockDim.x) {
            const int row = o / Kx, mx = o % Kx - Mx;
            const int mxm = ((mx % LPx) + LPx) % LPx;
            double sr = 0.0, si = 0.0;
            int r = 0;
            const double* rr = rows + row * LPx;
            for (int px = 0; px < LPx; ++px) {
                const double2 w = twx[r];
                sr = fma(rr[px], w.x, sr);
                si = fma(rr[px], w.y, si);
                r += mxm;
                if (r >= LPx) r -= LPx;
            }
            R[row * Kx + mx + Mx] = make_double2(sr, si);
        }
        __syncthreads();
        if (tid < Kx * Ky) {
            const int mym = ((my_t % LPy) + LPy) % LPy;
            for (int row = 0; row < nr; ++row) {
                const int py = py0 + row;
                const int r = (int)(((int64_t)mym * py) % LPy);
                const double2 w = twy[r];
                const double2 v = R[row * Kx + mx_t + Mx];
                accr = fma(v.x, w.x, fma(-v.y, w.y, accr));
                acci = fma(v.x, w.y, fma(v.y, w.x, acci));
            }
        }
    }
    if (tid < Kx * Ky) {
        const int mx = mx_t, my = my_t;
        double2 out = make_double2(0.0, 0.0);
        if ((int64_t)mx * mx * My * My + (int64_t)my * my * Mx * Mx <= (int64_t)Mx * Mx * My * My) {
            const double sgn = ((mx + my) % 2 == 0) ? dxdy : -dxdy;
            out = make_double2(sgn * accr, sgn * acci);
        }
        Ds[(int64_t)n * Kx * Ky + (My - my) * Kx + (mx + Mx)] = out;
    }
}

// ---------------------------------------------------------------- phi

// Thread = a pixel column and four rows of it at a time: a spectral column
// sum Q read from shared memory serves four pixels.  The twiddles of the
// period (exact integer reductions) are formed once per block, not per term.
// Measured at 1024 RFs, 64 x 64, Mx = My = 6: 150 us with a sincospi per term,
// 52 here.
constexpr int kPhiRows = 4;

__global__ void __launch_bounds__(256) dirich_space_kernel(const double2* __restrict__ Ds, int Mx, int My, int Px,
                                                            int Py, int Px1, int Py1, int table,
                                                            double* __restrict__ out) {
    extern __shared__ double smem[];
    const int Kx = 2 * Mx + 1, Ky = 2 * My + 1;
    double2* Q = reinterpret_cast<double2*>(smem);  // Ky x Px : sum over mx
    double2* ey = Q + Ky * Px;                       // Ky x Py
    double2* tw = ey + Ky * Py;                      // e^{2 pi i r / Px1}, r < Px1 (when table)
    const int n = blockIdx.x;
    const int tid = threadIdx.x;
    const int xd = (Px1 - Px) / 2, yd = (Py1 - Py) / 2;
    const double2* D = Ds + (int64_t)n * Kx * Ky;
    auto twiddle = [](int r, int L) {
        double s, c;
        sincospi(2.0 * r / L, &s, &c);
        return make_double2(c, s);
    };
    if (table) {
        for (int r = tid; r < Px1; r += blockDim.x) tw[r] = twiddle(r, Px1);
        __syncthreads();
    }
    for (int o = tid; o < Ky * Px; o += blockDim.x) {
        const int myi = o / Px, px = o % Px;
        const int my = myi - My;
        double sr = 0.0, si = 0.0;
        int r = (int)((((int64_t)-Mx * (px + xd)) % Px1 + Px1) % Px1);   // mx (px + xd) mod Px1
        const int step = (px + xd) % Px1;
        for (int mx = -Mx; mx <= Mx; ++mx) {
            const double2 d = D[(My - my) * Kx + (mx + Mx)];
            const double sg = (((mx + my) % 2) == 0) ? 1.0 : -1.0;
            const double2 e = table ? tw[r] : twiddle(r, Px1);
            sr += sg * (d.x * e.x - d.y * e.y);
            si += sg * (d.x * e.y + d.y * e.x);
            r += step;
            if (r >= Px1) r -= Px1;
        }
        Q[o] = make_double2(sr, si);
    }
    for (int o = tid; o < Ky * Py; o += blockDim.x) {
        const int myi = o / Py, py = o % Py;
        const int my = myi - My;
        ey[o] = twiddle((int)(((((int64_t)my * (py + yd)) % Py1) + Py1) % Py1), Py1);
    }
    __syncthreads();
    const int groups = (Py + kPhiRows - 1) / kPhiRows;
    for (int p = tid; p < Px * groups; p += blockDim.x) {
        const int py = (p / Px) * kPhiRows, px = p % Px;
        double acc[kPhiRows];
        int row[kPhiRows];
#pragma unroll
        for (int i = 0; i < kPhiRows; ++i) {
            acc[i] = 0.0;
            row[i] = min(py + i, Py - 1);
        }
        for (int myi = 0; myi < Ky; ++myi) {
            const double2 q = Q[myi * Px + px];
#pragma unroll
            for (int i = 0; i < kPhiRows; ++i) {
                const double2 e = ey[myi * Py + row[i]];
                acc[i] = fma(q.x, e.x, fma(-q.y, e.y, acc[i]));
            }
        }
#pragma unroll
        for (int i = 0; i < kPhiRows; ++i)
            if (py + i < Py) out[(int64_t)n * Px * Py + (int64_t)(py + i) * Px + px] = acc[i];
    }
}

// ---------------------------------------------------------------- Dsw

__global__ void put_norm_kernel(double* __restrict__ W, int64_t ld, int N, const double* __restrict__ norm) {
    const int a = blockIdx.y;
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= N) return;
    W[(int64_t)a * ld + b] *= norm[a] * norm[b];
}

// ---------------------------------------------------------------- q, G

__global__ void compute_q_kernel(const double* __restrict__ tk1, const double* __restrict__ tk2,
                                 const int32_t* __restrict__ ind, int n, const double* __restrict__ kappa,
                                 const double* __restrict__ delta, const double* __restrict__ bias,
                                 const double* __restrict__ norm, double* __restrict__ q) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int nr = ind[i];
        q[i] = (kappa[nr] * delta[nr] - bias[nr] * (tk2[i] - tk1[i])) * norm[nr];
    }
}

// G[r][c] = Dsw[ind_r][ind_c] int_r int_c D(s - t) ds dt with the Dirichlet
// kernel D.  compute_G_Kernel's bracket (dirichlet.py:300-320)
//   sum_m [cos mW(r2-c2) - cos mW(r2-c1) - cos mW(r1-c2) + cos mW(r1-c1)] 2/(mW)^2 + |r||c|
// is the product of two (2Mt+1)-vectors, one per interval:
//   |r||c| + 2 sum_m Re T_r(m) conj T_c(m),
//   T_k(m) = int_{tk1}^{tk2} e^{jmWs} ds = (2/(mW)) sin(mW d/2) e^{jmW tbar},
// so an entry costs 2Mt+1 float64 FMAs instead of 4 Mt cosines, and no
// difference of cosines cancels.  Only differences of times count: they are
// taken from the first interval's start.  Bound: the HBM write of G (n^2 * 8 bytes).
//
// A block forms 64 x 64 tiles of the lower triangle of tiles on the float64
// tensor-core path (mma m8n8k4, exact float64 FMAs: few shared-memory reads
// and instructions per entry, which a register tile with bounds checks and
// gathers per entry was bound by), stages the products in shared memory and
// writes them by whole rows (256 bytes a warp), times Dsw, and, unless only
// the lower triangle is wanted, again transposed as the mirror tile: half the
// products.  A block walks `strip` tiles of one tile row and keeps that row's
// harmonics.
//
// The harmonics (two sincos, a division and two complex products per
// harmonic, a fresh sincos every kGHarm so that powers lose a few ulp at any
// Mt) are formed once per interval in the caller's workspace
// (harmonics_table_kernel), or, without one, by every tile that meets the
// interval.  Measured at n = 24001, Mt = 8 (4.6 GB): 41.6 ms with the cosines,
// 1.51 ms with a register tile on the FMA pipe, 1.31 ms here (3.5 TB/s; with
// rows of whole sectors, n = 24000, 1.06 ms, where a fill takes 0.62): the odd
// row length's split sectors and the latency of a tile's phases, four blocks
// per SM.  Three blocks with deeper gathers: 1.36 ms; strips of 16: 1.36 ms.
constexpr int kGT = 64;        // tile side
constexpr int kGHarm = 8;      // harmonics per pass over the tile
constexpr int kGF = 2 * kGHarm + 1;
constexpr int kGK = 20;        // kGF up to whole k-steps of 4
constexpr int kGS = kGT + 4;   // row stride of the staged harmonics: fragment reads free of bank conflicts

// place of entry (r, c) of the staged products: rows, columns and the
// products' 4 x 4 fragment corners all free of bank conflicts
__device__ __forceinline__ int g_at(int r, int c) { return r * kGT + (c ^ (((r & 3) << 2) | ((r >> 2) & 3))); }

// place of tile column c among the staged harmonics: a product's 8 columns
// 2q, 2q + 1 hold the tile's q, q + 4, so that a fragment's stores are contiguous
__device__ __forceinline__ int g_col(int c) { return (c & ~7) | ((c & 3) << 1) | ((c >> 2) & 1); }

// a number as a double and its rounding error (error-free sums and products:
// Knuth's two-sum, one FMA)
struct GPair {
    double hi, lo;
};

__device__ __forceinline__ GPair g_sum(double a, double b) {
    const double s = a + b, t = s - a;
    return GPair{s, (a - (s - t)) + (b - t)};
}

// k x to twice the precision, and its sine and cosine
__device__ __forceinline__ GPair g_times(double k, const GPair& x) {
    const double p = __dmul_rn(k, x.hi);
    return GPair{p, fma(k, x.hi, -p) + k * x.lo};
}

__device__ __forceinline__ void g_sincos(const GPair& x, double* s, double* c) {
    double s0, c0;
    sincos(x.hi, &s0, &c0);
    *s = fma(c0, x.lo, s0);
    *c = fma(-s0, x.lo, c0);
}

// Harmonics m0 .. m0+kGHarm-1 (m >= 1; zero beyond Mt) of the interval (t1, t2)
// from the origin t0, scaled: f[S * (2i + 1)] = Re, f[S * (2i + 2)] = Im, and
// f[0] = t2 - t1 in the first pass.  The phases are formed to twice the
// precision: all harmonics of an interval share them, so that a rounded phase
// moves the whole interval.  Relative error of G over a window of 1 s, Mt = 8:
// 1.2e-15 by a cosine per difference of times, 2.1e-15 by rounded phases, 3e-16
// here.
template <int S>
__device__ __forceinline__ void g_features(double t1, double t2, double t0, int m0, int Mt, double W, double scale,
                                           double* __restrict__ f) {
    const GPair a = g_sum(t1, -t0), b = g_sum(t2, -t0), d = g_sum(t2, -t1);
    GPair tb = g_sum(a.hi, b.hi);
    tb.lo += a.lo + b.lo;
    const GPair ph = g_times(0.5 * W, tb), pd = g_times(0.5 * W, d);
    f[0] = m0 == 1 ? d.hi : 0.0;
    double s1, c1, sh, ch, sp, cp, sq, cq;
    g_sincos(ph, &s1, &c1);
    g_sincos(pd, &sh, &ch);
    if (m0 == 1) {
        sp = s1;
        cp = c1;
        sq = sh;
        cq = ch;
    } else {
        g_sincos(g_times(m0, ph), &sp, &cp);
        g_sincos(g_times(m0, pd), &sq, &cq);
    }
#pragma unroll
    for (int i = 0; i < kGHarm; ++i) {
        const int m = m0 + i;
        const double amp = m <= Mt ? scale * (2.0 / (m * W)) * sq : 0.0;
        f[S * (2 * i + 1)] = amp * cp;
        f[S * (2 * i + 2)] = amp * sp;
        const double c2 = cp * c1 - sp * s1, s2 = cp * s1 + sp * c1;
        const double c3 = cq * ch - sq * sh, s3 = cq * sh + sq * ch;
        cp = c2;
        sp = s2;
        cq = c3;
        sq = s3;
    }
}

// table[(k) * n + i]: feature k = 0..2Mt of interval i, unscaled
__global__ void __launch_bounds__(128) harmonics_table_kernel(const double* __restrict__ tk1,
                                                              const double* __restrict__ tk2, int n, double W, int Mt,
                                                              double* __restrict__ table) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int m0 = 1 + blockIdx.y * kGHarm;
    if (i >= n) return;
    double f[kGF];
    g_features<1>(tk1[i], tk2[i], tk1[0], m0, Mt, W, 1.0, f);
    if (m0 == 1) table[i] = f[0];
#pragma unroll
    for (int h = 0; h < kGHarm; ++h) {
        const int m = m0 + h;
        if (m <= Mt) {
            table[(int64_t)(2 * m - 1) * n + i] = f[2 * h + 1];
            table[(int64_t)(2 * m) * n + i] = f[2 * h + 2];
        }
    }
}

// features of the tile's intervals i0 .. i0+kGT-1 for the pass from harmonic m0, from the table (zero-padded to kGK)
template <bool COLS>
__device__ __forceinline__ void g_load(const double* __restrict__ table, int n, int i0, int m0, int nf, double scale,
                                       double* __restrict__ f) {
    for (int e = threadIdx.x; e < kGK * kGT; e += 256) {
        const int k = e / kGT, i = e % kGT;
        double v = 0.0;
        if (i0 + i < n && k < nf && (k > 0 || m0 == 1)) {
            v = __ldg(table + (int64_t)(k + (k > 0 ? 2 * (m0 - 1) : 0)) * n + i0 + i);
            if (k > 0) v *= scale;
        }
        f[k * kGS + (COLS ? g_col(i) : i)] = v;
    }
}

__device__ __forceinline__ void dmma_8x8x4(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// Rows w, w + 8, ... of a staged tile times Dsw into G, one row of 64 entries
// at a time by a warp.  TRANS: the mirror tile (tile columns become G's rows).
// EDGE: the tile crosses G's edge or its diagonal.
template <bool TRANS, bool EDGE>
__device__ __forceinline__ void g_store(const double* __restrict__ tile, const int* __restrict__ ri,
                                        const int* __restrict__ ci, int r0, int c0, int n,
                                        const double* __restrict__ Dsw, int64_t dsw_ld, double lamb, int lower_only,
                                        double* __restrict__ G, int64_t G_ld) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k0 = ci[lane], k1 = ci[lane + 32];
#pragma unroll 4
    for (int r = w; r < kGT; r += 8) {
        const double v0 = tile[TRANS ? g_at(lane, r) : g_at(r, lane)];
        const double v1 = tile[TRANS ? g_at(lane + 32, r) : g_at(r, lane + 32)];
        const double* dr = Dsw + (int64_t)ri[r] * dsw_ld;
        double* g = G + (int64_t)(r0 + r) * G_ld + c0 + lane;
        if (!EDGE) {
            __stcs(g, v0 * __ldg(dr + k0));
            __stcs(g + 32, v1 * __ldg(dr + k1));
        } else if (r0 + r < n) {
            const int row = r0 + r, a = c0 + lane, b = a + 32;
            if (a < n && !(lower_only && a > row)) __stcs(g, v0 * __ldg(dr + k0) + (a == row ? lamb : 0.0));
            if (b < n && !(lower_only && b > row)) __stcs(g + 32, v1 * __ldg(dr + k1) + (b == row ? lamb : 0.0));
        }
    }
}

template <bool TABLE>
__global__ void __launch_bounds__(256, 4) compute_G_kernel(const double* __restrict__ tk1, const double* __restrict__ tk2,
                                                           const int32_t* __restrict__ ind, int n, double W, int Mt,
                                                           const double* __restrict__ Dsw, int64_t dsw_ld, double lamb,
                                                           int lower_only, int strip,
                                                           const double* __restrict__ table, double* __restrict__ G,
                                                           int64_t G_ld) {
    extern __shared__ double gsm[];
    double* fr = gsm;                       // kGK x kGS: the tile row's harmonics
    double* fc = fr + kGK * kGS;            // kGK x kGS: the tile column's, doubled
    double* tile = fc + kGK * kGS;          // kGT x kGT: the products
    __shared__ int ri[kGT], ci[kGT];
    // block -> (tile row, strip of tile columns): tile rows in groups of `strip`
    // rows, group g having g + 1 strips a row
    int g = (int)((sqrt(1.0 + 8.0 * (double)blockIdx.x / strip) - 1.0) * 0.5);
    while ((int64_t)strip * g * (g + 1) / 2 > blockIdx.x) --g;
    while ((int64_t)strip * (g + 1) * (g + 2) / 2 <= blockIdx.x) ++g;
    const int rem = (int)(blockIdx.x - (int64_t)strip * g * (g + 1) / 2);
    const int ti = g * strip + rem / (g + 1);
    const int tj0 = (rem % (g + 1)) * strip;
    const int row0 = ti * kGT;
    if (row0 >= n) return;
    const int tid = threadIdx.x;
    const double t0 = TABLE ? 0.0 : tk1[0];
    // warp (wr, wc) of 2 x 4: 32 rows x 16 columns as 4 x 2 products of 8 x 8
    const int lane = tid & 31, wr = (tid >> 5) & 1, wc = tid >> 6;
    const int fl = (lane & 3) * kGS + (lane >> 2);
    if (tid < kGT) ri[tid] = row0 + tid < n ? ind[row0 + tid] : 0;
    if (!TABLE)
        for (int e = tid; e < (kGK - kGF) * kGS; e += 256) fr[kGF * kGS + e] = fc[kGF * kGS + e] = 0.0;
    for (int tj = tj0; tj < min(tj0 + strip, ti + 1); ++tj) {
        const int col0 = tj * kGT;
        double acc[4][2][2];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
        for (int m0 = 1; m0 <= Mt; m0 += kGHarm) {
            __syncthreads();                // the previous pass's harmonics and the previous tile have been read
            const int nf = 1 + 2 * min(kGHarm, Mt + 1 - m0);
            const bool rows = tj == tj0 || Mt > kGHarm;
            if (TABLE) {
                g_load<true>(table, n, col0, m0, nf, 2.0, fc);
                if (rows) g_load<false>(table, n, row0, m0, nf, 1.0, fr);
            } else if (tid < kGT) {
                const int c = col0 + tid;
                g_features<kGS>(c < n ? tk1[c] : t0, c < n ? tk2[c] : t0, t0, m0, Mt, W, 2.0, fc + g_col(tid));
            } else if (tid < 2 * kGT && rows) {
                const int r = row0 + tid - kGT;
                g_features<kGS>(r < n ? tk1[r] : t0, r < n ? tk2[r] : t0, t0, m0, Mt, W, 1.0, fr + tid - kGT);
            }
            if (m0 == 1 && tid >= 192) ci[tid - 192] = col0 + tid - 192 < n ? ind[col0 + tid - 192] : 0;
            __syncthreads();
            const double* fa = fr + fl + 32 * wr;
            const double* fb = fc + fl + 16 * wc;
            for (int k = 0; k < nf; k += 4, fa += 4 * kGS, fb += 4 * kGS) {
                const double b0 = fb[0], b1 = fb[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const double a = fa[8 * i];
                    dmma_8x8x4(acc[i][0], a, b0);
                    dmma_8x8x4(acc[i][1], a, b1);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int r = 32 * wr + 8 * i + (lane >> 2), c = 16 * wc + 8 * j + (lane & 3);
                tile[g_at(r, c)] = acc[i][j][0];
                tile[g_at(r, c + 4)] = acc[i][j][1];
            }
        __syncthreads();
        if (ti == tj || row0 + kGT > n || col0 + kGT > n) {
            g_store<false, true>(tile, ri, ci, row0, col0, n, Dsw, dsw_ld, lamb, lower_only, G, G_ld);
            if (!lower_only && ti != tj)
                g_store<true, true>(tile, ci, ri, col0, row0, n, Dsw, dsw_ld, lamb, 0, G, G_ld);
        } else {
            g_store<false, false>(tile, ri, ci, row0, col0, n, Dsw, dsw_ld, lamb, 0, G, G_ld);
            if (!lower_only) g_store<true, false>(tile, ci, ri, col0, row0, n, Dsw, dsw_ld, lamb, 0, G, G_ld);
        }
    }
}

}  // namespace vtb

using namespace vtb;

VTB_API int vtb_dirichlet_coeffs(const double* rf, int N, int LPy, int LPx, int64_t rf_ld, int Mx, int My,
                                 double dxdy, double* Ds, void* stream) {
    VTB_CHECK_ARG(N >= 0 && LPy > 0 && LPx > 0 && Mx >= 0 && My >= 0 && rf_ld >= (int64_t)LPx * LPy);
    if (N == 0) return VTB_OK;
    VTB_CHECK_ARG(rf && Ds);
    const int Kx = 2 * Mx + 1, Ky = 2 * My + 1;
    VTB_CHECK_ARG(Kx * Ky <= 256);
    // the tensor path needs its tables and one RF's row sums in shared memory
    // (256 x 256: 74 KB beside 16 KB of partial sums, two blocks per SM); longer
    // sides and more bins take the general kernel.  Where fewer blocks fit on an
    // SM than the grid counts on (sides of 144 to 200), the others follow.
    const int Xp = (LPx + 7) & ~7, Yp = (LPy + 15) & ~15;
    const size_t smm = (size_t)(2 * Yp + (LPx == LPy && Mx == My ? 0 : Xp)) * kDfS * sizeof(double);
    if (Kx <= 16 && Ky <= 16 && smm <= kCallSmem) {
        const bool vec = LPx % 2 == 0 && rf_ld % 2 == 0 && ((uintptr_t)rf & 15) == 0;
        auto kernel = vec ? ds_mma_kernel<true> : ds_mma_kernel<false>;
        VTB_CUDA_TRY(allow_call_smem(kernel));
        const int per_sm = smm > 100 * 1024 ? 1 : smm > 56 * 1024 ? 2 : 4;
        kernel<<<std::min(N, per_sm * kNumSMs), kDfWarps * 32, smm, as_stream(stream)>>>(
            rf, rf_ld, N, LPy, LPx, Mx, My, dxdy, reinterpret_cast<double2*>(Ds));
        return launch_status();
    }
    const size_t sm = (size_t)(LPx + LPy) * sizeof(double2) + (size_t)kDsRows * LPx * sizeof(double) +
                      (size_t)kDsRows * Kx * sizeof(double2);
    VTB_CHECK_ARG(sm <= kCallSmem);
    if (sm > 48 * 1024) VTB_CUDA_TRY(allow_call_smem(ds_kernel));
    ds_kernel<<<N, 256, sm, as_stream(stream)>>>(rf, rf_ld, LPy, LPx, Mx, My, dxdy,
                                                 reinterpret_cast<double2*>(Ds));
    return launch_status();
}

VTB_API int vtb_dirich_space(const double* Ds, int N, int Mx, int My, int Px, int Py, int Px1, int Py1,
                             double* out, void* stream) {
    VTB_CHECK_ARG(N >= 0 && Mx >= 0 && My >= 0 && Px > 0 && Py > 0 && Px1 >= Px && Py1 >= Py);
    // the reference's FFT placement folds bins that alias on the period grid
    VTB_CHECK_ARG(2 * Mx + 1 <= Px1 && 2 * My + 1 <= Py1);
    if (N == 0) return VTB_OK;
    VTB_CHECK_ARG(Ds && out);
    const int Ky = 2 * My + 1;
    const size_t base = (size_t)Ky * (Px + Py) * sizeof(double2);
    VTB_CHECK_ARG(base <= kCallSmem);
    const int table = base + (size_t)Px1 * sizeof(double2) <= kCallSmem;
    const size_t sm = base + (table ? (size_t)Px1 * sizeof(double2) : 0);
    if (sm > 48 * 1024) VTB_CUDA_TRY(allow_call_smem(dirich_space_kernel));
    dirich_space_kernel<<<N, 256, sm, as_stream(stream)>>>(reinterpret_cast<const double2*>(Ds), Mx, My, Px, Py,
                                                          Px1, Py1, table, out);
    return launch_status();
}

VTB_API int vtb_dsw(const double* Ds, int N, int Ks, const double* norm, double* Dsw, int64_t ld, void* stream) {
    VTB_CHECK_ARG(N >= 0 && Ks >= 0 && ld >= N);
    if (N == 0) return VTB_OK;
    VTB_CHECK_ARG(Ds && norm && Dsw);
    // Re(conj(a) b) = a.re b.re + a.im b.im: a real GEMM over the interleaved planes
    GemmF64Args g{N, N, 2 * Ks, Ds, 2 * (int64_t)Ks, 1, Ds, 2 * (int64_t)Ks, 1, Dsw, ld, 1, 1.0, 0.0};
    int st = gemm_f64(g, as_stream(stream));
    if (st) return st;
    dim3 grid(ceil_div(N, 256), N);
    put_norm_kernel<<<grid, 256, 0, as_stream(stream)>>>(Dsw, ld, N, norm);
    return launch_status();
}

VTB_API int vtb_compute_q(const double* tk1, const double* tk2, const int32_t* ind, int n, const double* kappa,
                          const double* delta, const double* bias, const double* norm, double* q, void* stream) {
    VTB_CHECK_ARG(n >= 0);
    if (n == 0) return VTB_OK;
    VTB_CHECK_ARG(tk1 && tk2 && ind && kappa && delta && bias && norm && q);
    const int blocks = min(ceil_div(n, 256), 6 * kNumSMs);
    compute_q_kernel<<<blocks, 256, 0, as_stream(stream)>>>(tk1, tk2, ind, n, kappa, delta, bias, norm, q);
    return launch_status();
}

static int launch_G(const double* tk1, const double* tk2, const int32_t* ind, int n, double Wt, int Mt,
                    const double* Dsw, int64_t dsw_ld, double lamb, int lower_only, double* table, double* G,
                    int64_t G_ld, cudaStream_t s) {
    const int T = ceil_div(n, kGT);
    VTB_CHECK_ARG(ceil_div(n, 32) <= 65535);
    // one tile a block while that is at most two waves of four blocks per SM,
    // else four (the row's harmonics formed or read once for four tiles)
    const int strip = (int64_t)T * (T + 1) / 2 <= 8 * kNumSMs ? 1 : 4;
    const int64_t groups = ceil_div(T, strip);
    const unsigned blocks = (unsigned)(strip * groups * (groups + 1) / 2);
    const size_t sm = (size_t)(2 * kGK * kGS + kGT * kGT) * sizeof(double);
    const double W = Wt / Mt;
    if (table) {
        harmonics_table_kernel<<<dim3(ceil_div(n, 128), ceil_div(Mt, kGHarm)), 128, 0, s>>>(tk1, tk2, n, W, Mt, table);
        VTB_CUDA_TRY(cudaFuncSetAttribute(compute_G_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        compute_G_kernel<true><<<blocks, 256, sm, s>>>(tk1, tk2, ind, n, W, Mt, Dsw, dsw_ld, lamb, lower_only, strip,
                                                       table, G, G_ld);
    } else {
        VTB_CUDA_TRY(cudaFuncSetAttribute(compute_G_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        compute_G_kernel<false><<<blocks, 256, sm, s>>>(tk1, tk2, ind, n, W, Mt, Dsw, dsw_ld, lamb, lower_only, strip,
                                                        nullptr, G, G_ld);
    }
    return launch_status();
}

VTB_API int vtb_compute_G(const double* tk1, const double* tk2, const int32_t* ind, int n, double Wt, int Mt,
                          const double* Dsw, int64_t dsw_ld, double lamb, int lower_only, double* G, int64_t G_ld,
                          void* stream) {
    VTB_CHECK_ARG(n >= 0 && Mt >= 0 && G_ld >= n);
    if (n == 0) return VTB_OK;
    VTB_CHECK_ARG(tk1 && tk2 && ind && Dsw && G && Mt > 0);
    return launch_G(tk1, tk2, ind, n, Wt, Mt, Dsw, dsw_ld, lamb, lower_only, nullptr, G, G_ld, as_stream(stream));
}

VTB_API int vtb_compute_G_workspace(int n, int Mt, int64_t* bytes) {
    VTB_CHECK_ARG(n >= 0 && Mt > 0 && bytes);
    *bytes = (int64_t)n * (2 * (int64_t)Mt + 1) * 8;
    return VTB_OK;
}

VTB_API int vtb_compute_G_work(const double* tk1, const double* tk2, const int32_t* ind, int n, double Wt, int Mt,
                               const double* Dsw, int64_t dsw_ld, double lamb, int lower_only, double* G, int64_t G_ld,
                               void* work, int64_t work_bytes, void* stream) {
    VTB_CHECK_ARG(n >= 0 && Mt >= 0 && G_ld >= n);
    if (n == 0) return VTB_OK;
    VTB_CHECK_ARG(tk1 && tk2 && ind && Dsw && G && Mt > 0 && work && ((uintptr_t)work & 7) == 0);
    VTB_CHECK_ARG(work_bytes >= (int64_t)n * (2 * (int64_t)Mt + 1) * 8 && ceil_div(Mt, kGHarm) <= 65535);
    return launch_G(tk1, tk2, ind, n, Wt, Mt, Dsw, dsw_ld, lamb, lower_only, reinterpret_cast<double*>(work), G, G_ld,
                    as_stream(stream));
}
