// Receptive-field banks and the float64 RF projection.
//
//  vtb_rf_gabor / vtb_rf_cs : the RF formulas of gabor_Kernel / cs_Kernel
//      (vtem/vrf.py:1197-1291, :1120-1193) on a pixel grid, a thread per
//      column of a tile.
//  vtb_rf_filter : L[f, n] = scale * sum_p V[f, p] RF[n, p] (the DGEMM of
//      vrf.py:291 / :871), written straight into the layout the IAF scan
//      reads (no separate transpose pass, unlike vrf.py:292).
#include "common.cuh"
#include "gemm_f64.cuh"

namespace vtb {

// A block generates a tile of kRfCols columns x kRfRows rows of one filter:
// thread = column, walking the rows.  What depends on the column or the row
// alone is formed once per block (rows in shared memory): with X = xc + ys,
// Y = yc - xs (xc, xs of the column, ys, yc of the row) and the modulation by
// the angle sum, cos(kX) = cos(k xc) cos(k ys) - sin(k xc) sin(k ys), a pixel
// costs one exp and about ten float64 operations instead of an exp, two
// sincos and three divisions.  Bound: the float64 rate (exp).  Measured, 768
// Gabor filters on 256 x 256: 559 us before, 138 here; 256 centre-surround: 189 us
// before, 61 here.
constexpr int kRfCols = 128, kRfRows = 32;

struct RfGrid {
    int Px, Py;
    double dx, dy, x_start, y_start;
};

__device__ __forceinline__ double grid_x(const RfGrid& g, int px) { return (double)px * g.dx + g.x_start; }
__device__ __forceinline__ double grid_y(const RfGrid& g, int py) { return -((double)py * g.dy + g.y_start); }

__global__ void __launch_bounds__(kRfCols) rf_gabor_kernel(const double* __restrict__ h_alpha,
                                                           const double* __restrict__ h_l,
                                                           const double* __restrict__ h_x0,
                                                           const double* __restrict__ h_y0,
                                                           const int32_t* __restrict__ h_ab,
                                                           const double* __restrict__ gain, RfGrid g, double kappa,
                                                           double* __restrict__ out, int64_t out_ld) {
    __shared__ double2 s_y[kRfRows], s_e[kRfRows];     // (y st, y ct), (cos, sin)(kappa y st)
    const int n = blockIdx.y, tid = threadIdx.x;
    const int tx = (g.Px + kRfCols - 1) / kRfCols;
    const int px = (blockIdx.x % tx) * kRfCols + tid, py0 = (blockIdx.x / tx) * kRfRows;
    const int rows = min(kRfRows, g.Py - py0);
    const double alpha = 1.0 / h_alpha[n];
    double st, ct;
    sincos(h_l[n], &st, &ct);
    if (tid < rows) {
        const double y = alpha * (grid_y(g, py0 + tid) - h_y0[n]);
        double s, c;
        sincos(kappa * (y * st), &s, &c);
        s_y[tid] = make_double2(y * st, y * ct);
        s_e[tid] = make_double2(c, s);
    }
    __syncthreads();
    if (px >= g.Px) return;
    const double x = alpha * (grid_x(g, px) - h_x0[n]);
    const double xc = x * ct, xs = x * st;
    double sx, cx;
    sincos(kappa * xc, &sx, &cx);
    const bool even = h_ab[n] == 0;
    const double scale = alpha * (1.0 / sqrt(2.0 * 3.141592653589793)), gn = gain ? gain[n] : 1.0;
    double* o = out + (int64_t)n * out_ld + (int64_t)py0 * g.Px + px;
#pragma unroll 4
    for (int r = 0; r < rows; ++r) {
        const double2 y = s_y[r], e = s_e[r];
        const double X = xc + y.x, Y = y.y - xs;
        const double w = even ? fma(cx, e.x, -(sx * e.y)) : fma(sx, e.x, cx * e.y);
        o[(int64_t)r * g.Px] = scale * exp(-((4 * X * X) + (Y * Y)) / 8) * w * gn;
    }
}

__global__ void __launch_bounds__(kRfCols) rf_cs_kernel(const double* __restrict__ h_alpha,
                                                        const double* __restrict__ h_x0,
                                                        const double* __restrict__ h_y0,
                                                        const double* __restrict__ gain, RfGrid g, double sc2,
                                                        double ss2, double* __restrict__ out, int64_t out_ld) {
    const int n = blockIdx.y, tid = threadIdx.x;
    const int tx = (g.Px + kRfCols - 1) / kRfCols;
    const int px = (blockIdx.x % tx) * kRfCols + tid, py0 = (blockIdx.x / tx) * kRfRows;
    if (px >= g.Px) return;
    const int rows = min(kRfRows, g.Py - py0);
    const double alpha = 1.0 / h_alpha[n], y0 = h_y0[n];
    const double x = alpha * (grid_x(g, px) - h_x0[n]), x2 = x * x;
    const double ec = 1.0 / (2 * sc2), es = 1.0 / (2 * ss2);
    const double wc = alpha / sc2 / 6.283185307179586, ws = 0.9 * alpha / ss2 / 6.283185307179586;
    const double gn = gain ? gain[n] : 1.0;
    double* o = out + (int64_t)n * out_ld + (int64_t)py0 * g.Px + px;
#pragma unroll 4
    for (int r = 0; r < rows; ++r) {
        const double y = alpha * (grid_y(g, py0 + r) - y0);
        const double XY = -(x2 + y * y);
        o[(int64_t)r * g.Px] = (wc * exp(XY * ec) - ws * exp(XY * es)) * gn;
    }
}

static dim3 rf_tiles(int Px, int Py, int n) {
    return dim3(ceil_div(Px, kRfCols) * ceil_div(Py, kRfRows), n);
}

}  // namespace vtb

using namespace vtb;

VTB_API int vtb_rf_gabor(const double* h_alpha, const double* h_l, const double* h_x0, const double* h_y0,
                         const int32_t* h_ab, const double* gain, int n_filters, int Px, int Py, double Sx,
                         double Sy, double x_start, double y_start, double KAPPA, double* out, int64_t out_ld,
                         void* stream) {
    VTB_CHECK_ARG(n_filters >= 0 && Px > 0 && Py > 0 && out_ld >= (int64_t)Px * Py);
    if (n_filters == 0) return VTB_OK;
    VTB_CHECK_ARG(h_alpha && h_l && h_x0 && h_y0 && h_ab && out && n_filters <= 65535);
    const RfGrid g{Px, Py, Sx / Px, Sy / Py, x_start, y_start};
    rf_gabor_kernel<<<rf_tiles(Px, Py, n_filters), kRfCols, 0, as_stream(stream)>>>(h_alpha, h_l, h_x0, h_y0, h_ab, gain,
                                                                                  g, KAPPA, out, out_ld);
    return launch_status();
}

VTB_API int vtb_rf_cs(const double* h_alpha, const double* h_x0, const double* h_y0, const double* gain,
                      int n_filters, int Px, int Py, double Sx, double Sy, double x_start, double y_start,
                      double sigma_center, double sigma_surround, double* out, int64_t out_ld, void* stream) {
    VTB_CHECK_ARG(n_filters >= 0 && Px > 0 && Py > 0 && out_ld >= (int64_t)Px * Py);
    if (n_filters == 0) return VTB_OK;
    VTB_CHECK_ARG(h_alpha && h_x0 && h_y0 && out && n_filters <= 65535);
    const RfGrid g{Px, Py, Sx / Px, Sy / Py, x_start, y_start};
    rf_cs_kernel<<<rf_tiles(Px, Py, n_filters), kRfCols, 0, as_stream(stream)>>>(
        h_alpha, h_x0, h_y0, gain, g, sigma_center * sigma_center, sigma_surround * sigma_surround, out, out_ld);
    return launch_status();
}

VTB_API int vtb_rf_filter(const double* video, int F, int P, int64_t video_ld, const double* rf, int N,
                          int64_t rf_ld, double scale, double* out, int64_t out_t_stride, int64_t out_n_stride,
                          void* stream) {
    VTB_CHECK_ARG(F >= 0 && P >= 0 && N >= 0 && video_ld >= P && rf_ld >= P);
    if (F == 0 || N == 0) return VTB_OK;
    VTB_CHECK_ARG(video && rf && out);
    GemmF64Args a{F, N, P, video, video_ld, 1, rf, rf_ld, 1, out, out_t_stride, out_n_stride, scale, 0.0};
    return gemm_f64(a, as_stream(stream));
}

VTB_API int vtb_gemm_f64(int M, int N, int K, const double* A, int64_t a_m, int64_t a_k, const double* B,
                         int64_t b_n, int64_t b_k, double* C, int64_t c_m, int64_t c_n, double alpha, double beta,
                         void* stream) {
    VTB_CHECK_ARG(M >= 0 && N >= 0 && K >= 0);
    if (M == 0 || N == 0) return VTB_OK;
    VTB_CHECK_ARG(A && B && C);
    GemmF64Args a{M, N, K, A, a_m, a_k, B, b_n, b_k, C, c_m, c_n, alpha, beta};
    return gemm_f64(a, as_stream(stream));
}
