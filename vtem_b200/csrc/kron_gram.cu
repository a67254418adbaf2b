// Float64 Kronecker Gram on the float64 tensor path (kron_gram.cuh).
//
// M is Hermitian and so is every W_n, so the pairs s <= s' and the entries
// m <= m' hold all of it: with a_n = d_n[s] conj(d_n[s']), the four real sums
// over n of {Re a, Im a} x {Re W, Im W}[m][m'] give
//   M((s,m),(s',m')) = (rr - ii, ri + ir),  M((s,m'),(s',m)) = (rr + ii, ir - ri),
// and their conjugates the mirror.  That is one real product of 2 pairs x
// Kt(Kt+1) columns over n: a quarter of the products of the complex form over
// all entries (1.9 ms at N = 1024, Ks = 113, Kt = 17 out of the FMA pipe;
// 8.1 GFLOP and 0.37 ms here), bound by the float64 rate.
//
// A CTA forms TP pairs x TE entries.  The pair products are formed on
// the way into shared memory (4 operations against 2 TE products each), the
// temporal entries arrive by cp.async; slabs of 16 neurons, the pair operand
// double-buffered through registers.  A product's 16 rows are the real parts
// of 8 pairs and their imaginary parts, so that a lane ends up with the four
// sums of its pair and entry.
#include "kron_gram.cuh"

namespace vtb {

constexpr int kKgThreads = 128, kKgK = 16, kKgStages = 3;

__device__ __forceinline__ void kg_mma(double (&c)[4], double a0, double a1, double b) {
    asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a0), "d"(a1), "d"(b));
}

// first entry (i, j), i <= j < n, of the row-major upper triangle at index p
__device__ __forceinline__ void upper_entry(int64_t p, int n, int& i, int& j) {
    const double b = 2.0 * n + 1.0;
    i = (int)((b - sqrt(b * b - 8.0 * (double)p)) * 0.5);
    if (i < 0) i = 0;
    auto start = [&](int64_t r) { return r * n - r * (r - 1) / 2; };
    while (i > 0 && start(i) > p) --i;
    while (start(i + 1) <= p) ++i;
    j = i + (int)(p - start(i));
}

// TP pairs and TE entries a CTA; 2 x 2 warps of (TP / 16) x (TE / 8) products of 16 x 8
template <int TP, int TE>
__global__ void __launch_bounds__(kKgThreads) kron_gram_kernel(const double2* __restrict__ d, int N, int Ks,
                                                               const double2* __restrict__ Wn, int Kt,
                                                               double2* __restrict__ M, int64_t ldm) {
    constexpr int SA = 2 * TP + 4, SB = 2 * TE + 4;    // row strides 4 mod 16: fragment reads free of bank conflicts
    constexpr int MT = TP / 16, NT = TE / 8;
    constexpr int PA = kKgK * TP / kKgThreads;         // pair products a thread
    constexpr int PB = kKgK * TE / kKgThreads;
    __shared__ __align__(16) double sa[2][kKgK * SA];
    __shared__ __align__(16) double sb[kKgStages][kKgK * SB];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int fr = lane >> 2, fk = lane & 3;
    const int64_t pairs = (int64_t)Ks * (Ks + 1) / 2;
    const int entries = Kt * (Kt + 1) / 2, KK = Kt * Kt;
    // the tiles of one row of pairs follow each other (the pairs alone can exceed
    // the 65,535 of the grid's other dimensions: Ks > 2047)
    const int et = (entries + TE - 1) / TE;
    const int64_t p0 = (int64_t)(blockIdx.x / et) * TP;
    const int e0 = blockIdx.x % et * TE;
    const int nk = (N + kKgK - 1) / kKgK;
    // this thread's pair (the same in every slab) and its neurons' stride
    const int q = tid % TP;
    int s = 0, s2 = 0;
    const bool pin = p0 + q < pairs;
    if (pin) upper_entry(p0 + q, Ks, s, s2);
    const int arow = 16 * (q >> 3) + (q & 7);
    // this thread's temporal entry
    const int c = tid % TE;
    int m = 0, m2 = 0;
    const bool ein = e0 + c < entries;
    if (ein) upper_entry(e0 + c, Kt, m, m2);
    const double2* wsrc = Wn + m * Kt + m2;
    double2 ra[PA], rb[PA];
    auto fetch = [&](int kb) {
#pragma unroll
        for (int i = 0; i < PA; ++i) {
            const int n = kb * kKgK + tid / TP + i * (kKgThreads / TP);
            ra[i] = rb[i] = make_double2(0.0, 0.0);
            if (pin && n < N) {
                ra[i] = __ldg(d + (int64_t)n * Ks + s);
                rb[i] = __ldg(d + (int64_t)n * Ks + s2);
            }
        }
    };
    auto put = [&](double* a) {
#pragma unroll
        for (int i = 0; i < PA; ++i) {
            double* x = a + (tid / TP + i * (kKgThreads / TP)) * SA + arow;
            x[0] = ra[i].x * rb[i].x + ra[i].y * rb[i].y;
            x[8] = s == s2 ? 0.0 : ra[i].y * rb[i].x - ra[i].x * rb[i].y;
        }
    };
    auto copy_w = [&](int kb) {
        if (kb < nk) {
            double* b = sb[kb % kKgStages];
#pragma unroll
            for (int i = 0; i < PB; ++i) {
                const int k = tid / TE + i * (kKgThreads / TE), n = kb * kKgK + k;
                const unsigned dst = (unsigned)__cvta_generic_to_shared(b + k * SB + 2 * c);
                const int bytes = ein && n < N ? 16 : 0;
                const double2* src = bytes ? wsrc + (int64_t)n * KK : Wn;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    double acc[MT][NT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 4; ++h) acc[i][j][h] = 0.0;
    const int wm = (w & 1) * (16 * MT), wn = (w >> 1) * (8 * NT);
    copy_w(0);
    copy_w(1);
    fetch(0);
    put(sa[0]);
    fetch(1);
    for (int kb = 0; kb < nk; ++kb) {
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();   // slab kb is complete; slab kb - 1 has been read by every warp
        if (kb + 1 < nk) {
            put(sa[(kb + 1) & 1]);
            fetch(kb + 2);
        }
        copy_w(kb + 2);
        const double* a = sa[kb & 1] + wm + fr;
        const double* b = sb[kb % kKgStages] + wn + fr;
#pragma unroll
        for (int k = 0; k < kKgK; k += 4) {
            double fb[NT];
#pragma unroll
            for (int j = 0; j < NT; ++j) fb[j] = b[(k + fk) * SB + 8 * j];
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                const double a0 = a[(k + fk) * SA + 16 * i], a1 = a[(k + fk) * SA + 16 * i + 8];
#pragma unroll
                for (int j = 0; j < NT; ++j) kg_mma(acc[i][j], a0, a1, fb[j]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < MT; ++i) {
        const int64_t p = p0 + (wm + 16 * i) / 2 + fr;
        if (p >= pairs) continue;
        int si, sj;
        upper_entry(p, Ks, si, sj);
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const int e = e0 + (wn + 8 * j) / 2 + fk;
            if (e >= entries) continue;
            int a, b;
            upper_entry(e, Kt, a, b);
            const double rr = acc[i][j][0], ri = acc[i][j][1], ir = acc[i][j][2], ii = acc[i][j][3];
            const double2 v = make_double2(rr - ii, si == sj && a == b ? 0.0 : ri + ir);
            const int64_t r1 = (int64_t)si * Kt, r2 = (int64_t)sj * Kt;
            M[(r2 + b) * ldm + r1 + a] = v;
            if (si != sj) M[(r1 + a) * ldm + r2 + b] = make_double2(v.x, -v.y);
            if (a != b) {
                const double2 u = make_double2(rr + ii, ir - ri);
                M[(r2 + a) * ldm + r1 + b] = u;
                if (si != sj) M[(r1 + b) * ldm + r2 + a] = make_double2(u.x, -u.y);
            }
        }
    }
}

int kron_gram_f64(const double2* d, int N, int Ks, const double2* Wn, int Kt, double2* M, int64_t ldm, cudaStream_t s) {
    const int64_t pairs = (int64_t)Ks * (Ks + 1) / 2;
    const int entries = Kt * (Kt + 1) / 2;
    // 32 pairs x 32 entries (each operand read for 64 rows or columns), or 16 x 16
    // while the larger tiles leave SMs without one
    const int64_t large = (pairs + 31) / 32 * ceil_div(entries, 32);
    if (large >= kNumSMs) {
        if (large > 0x7fffffff) return VTB_BAD_ARG;
        kron_gram_kernel<32, 32><<<(unsigned)large, kKgThreads, 0, s>>>(d, N, Ks, Wn, Kt, M, ldm);
    } else {
        kron_gram_kernel<16, 16><<<ceil_div(entries, 16) * ceil_div(pairs, 16), kKgThreads, 0, s>>>(d, N, Ks, Wn, Kt, M,
                                                                                                    ldm);
    }
    return launch_status();
}

}  // namespace vtb
