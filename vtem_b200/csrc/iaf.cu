// Ideal IAF time encoder: warp-per-neuron FP64 scan.
//
// Semantics follow the reference kernels exactly (vtem/ensemble_encode.py:
// 438-552 deterministic thresholds, :555-674 random thresholds, including the
// draw of the next threshold before `area -= (delta - v0)` at :623-627) and
// VTEM_IAF's block loop (vtem/vtem.py:165-200): frames are grouped in blocks of
// `block_frames` sharing one boundary frame, time_count restarts at 0 at every
// block boundary and v0 carries over.  Spike times are block-relative, as the
// reference stores them.
//
// This file is compiled with --fmad=false: every product and sum rounds
// separately, in the reference's source order, so spike times and sample
// indices are bit-identical to a non-contracting host execution of the
// reference kernel.
//
// Work split: one warp per neuron.  For each chunk of 32 steps the lanes take
// 32 samples (coalesced when the input is neuron-major; asynchronous copies
// run kIafAhead chunks ahead of their use), form y = (x+b)/kappa
// and the trapezoid area of their own step in parallel, and stage them in
// shared memory; the warp then walks the 32 steps in order (the membrane
// recursion is a strict sequential FP64 chain that no reordering may touch).
// The common step is one add and one compare; steps with a threshold crossing
// or a negative slope take the reference's full loop.  Spikes are appended by
// lane 0 to the neuron's slice of the output.  Each neuron stops once its
// spike count reaches `cap`, which bounds every loop by the buffer size.
#include "common.cuh"

namespace vtb {

struct IafArgs {
    const double* in;
    int64_t ts, ns;          // strides of in(t, n)
    int N, F, block_frames;
    double dt;
    const double* kappa;
    const double* bias;
    const double* delta;     // threshold (mean threshold for random thresholds)
    double* v0;
    double* time_count;
    // random thresholds (randn == nullptr: deterministic)
    const double* randn;
    int64_t rb, rs, rn;      // strides of randn(block, slot, n)
    int block_cap;           // slots per block in randn
    const double* sigma;
    double* delta_value;
    // outputs, neuron-major [n * cap + j]
    double* spike_time;
    int32_t* spike_step;
    int32_t* spike_count;
    int cap;
    unsigned long long* near_count;
    double near_eps;
    int32_t* status;
    double block_rate;       // > 0: per-block spike limit ceil(block length / block_rate)
};

constexpr int kIafWarps = 4;
constexpr int kIafAhead = 16;  // chunks of 32 samples in flight to shared memory

// What a warp carries from step to step (the same in every lane).
struct IafState {
    double v0, tc, delta;
    unsigned long long near;
    int count, cnt_block, block, next_reset, lim_block;
    bool stop, limit_hit;
};

// A warp's shared memory.
struct IafWarp {
    double area[2][32], v[32], t[32];      // areas of this chunk and the next
    double y1[32], y2[32];
    double in[kIafAhead * 32];
};

// spike limit of a frame block of `len` frames (the reference's per-call buffer)
__device__ __noinline__ int iaf_limit(double block_rate, int len) {
    if (!(block_rate > 0.0)) return 0x7fffffff;
    const double lim = ceil((double)len / block_rate);
    return lim < 2147483647.0 ? (int)lim : 0x7fffffff;
}

__device__ __noinline__ double iaf_quotient(double a, double b) { return a / b; }

// A chunk that may hold a crossing, a negative slope or the clip's end, walked
// as register chains between slow steps.  A chain covers the steps j0.. of the
// positive-slope form: the warp runs the membrane recursion v += area_j in the
// reference's order (uniform across lanes: the 32 areas are loaded from shared
// memory into registers first, so the chain is nothing but dependent adds;
// steps outside j0..nst-1 have area 0, which leaves v as it is) and the time
// recursion tc += dt beside it, and stores both after each step; lane j tests
// step j's value and ballots find the first step that is a crossing or not of
// the positive-slope form.  Steps before it are final as computed (the same
// float64 operations in the same order as the reference's step loop; after a
// block start inside the chain the time is one of the sums of ts).  The
// found step runs the reference's full loop (slow_step) from the exact state,
// and the next chain starts after it.  With frame blocks shorter than 32 steps
// every step takes the full loop.  (Not inlined: the loop over the common
// chunks stays small enough for the instruction cache.)
template <bool RT>
__device__ __noinline__ IafState iaf_walk(const IafArgs& p, IafState st, IafWarp& sm, double* area, const double* ts,
                                          int n, int t0, int nst, unsigned posmask, int lim_full, int lim_last) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int bstep = p.block_frames - 1;
    const double dt = p.dt;
    const double dmean = p.delta[n];
    const double sg = RT ? p.sigma[n] : 0.0;
    double v0 = st.v0, tc = st.tc, delta = st.delta;
    int count = st.count, cnt_block = st.cnt_block, block = st.block, next_reset = st.next_reset;
    int lim_block = st.lim_block;
    unsigned long long near = st.near;
    bool stop = st.stop, limit_hit = st.limit_hit;
    auto start_block = [&]() {
        cnt_block = 0;
        ++block;
        next_reset += bstep;
        lim_block = p.F - block * bstep >= p.block_frames ? lim_full : lim_last;
    };
    auto slow_step = [&](int j) {
        const int g = t0 + j;
        if (g == next_reset) {  // start of the next frame block
            tc = 0.0;
            start_block();
        }
        const double area0 = area[j];
        const bool pos = (posmask >> j) & 1u;
        if (pos) {
            const double s = v0 + area0;
            near += (fabs(s - delta) < p.near_eps) ? 1ull : 0ull;
            if (!(s >= delta)) {  // the common step: no crossing
                v0 = s;
                tc += dt;
                return;
            }
            // crossing(s) inside this step: the reference's loop
            double y1 = sm.y1[j];
            const double y2 = sm.y2[j];
            double area = area0;
            double ddt = dt;
            for (;;) {
                const double a = ((y2 - y1) / ddt);
                const double remain = (fabs(a) <= 1e-12) ? ((delta - v0) / y1)
                                                         : (sqrt(y1 * y1 + 2 * (delta - v0) * a) - y1) / (a);
                tc += remain;
                if (RT) {
                    const int slot = cnt_block < p.block_cap - 1 ? cnt_block : p.block_cap - 1;
                    delta = p.randn[(int64_t)block * p.rb + (int64_t)slot * p.rs + (int64_t)n * p.rn] * sg + dmean;
                }
                if (lane == 0) {
                    p.spike_time[(int64_t)n * p.cap + count] = tc;
                    p.spike_step[(int64_t)n * p.cap + count] = g;
                }
                ++count;
                ++cnt_block;
                limit_hit |= cnt_block >= lim_block;
                area -= (delta - v0);
                v0 = 0;
                ddt -= remain;
                y1 = y1 + remain * a;
                if (count >= p.cap) { stop = true; break; }
                const double s2 = v0 + area;
                near += (fabs(s2 - delta) < p.near_eps) ? 1ull : 0ull;
                if (!(s2 >= delta)) break;
            }
            if (stop) return;
            v0 += area;
            tc += ddt;
        } else {
            // negative slope through zero (ensemble_encode.py:515-535)
            double y1 = sm.y1[j];
            const double y2 = sm.y2[j];
            double ddt = dt;
            double a = ((y2 - y1) / ddt);
            double remain;
            for (;;) {
                remain = y1 * y1 + 2 * (delta - v0) * a;
                near += (fabs(remain) < p.near_eps) ? 1ull : 0ull;
                if (!(remain >= 0)) break;
                remain = (sqrt(remain) - y1) / a;
                tc += remain;
                if (RT) {
                    const int slot = cnt_block < p.block_cap - 1 ? cnt_block : p.block_cap - 1;
                    delta = p.randn[(int64_t)block * p.rb + (int64_t)slot * p.rs + (int64_t)n * p.rn] * sg + dmean;
                }
                if (lane == 0) {
                    p.spike_time[(int64_t)n * p.cap + count] = tc;
                    p.spike_step[(int64_t)n * p.cap + count] = g;
                }
                ++count;
                ++cnt_block;
                limit_hit |= cnt_block >= lim_block;
                v0 = 0;
                ddt -= remain;
                y1 = y1 + remain * a;
                a = ((y2 - y1) / ddt);
                if (count >= p.cap) { stop = true; break; }
            }
            if (stop) return;
            v0 += (y1 + y2) / 2 * ddt;
            tc += ddt;
        }
    };
    const bool fastok = bstep >= 32 || bstep <= 0;
    int j0 = 0;
    while (j0 < nst && !stop) {
        int f = j0;
        if (fastok) {
            const int rpos = (next_reset >= t0 + j0 && next_reset < t0 + nst) ? next_reset - t0 : -1;
            if (j0 > 0 || nst < 32) {
                if (lane < j0 || lane >= nst) area[lane] = 0.0;
                __syncwarp();
            }
            double v = v0, tt = tc;
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                const double2 q = *reinterpret_cast<const double2*>(&area[j]);
                const double va = v + q.x;
                v = va + q.y;
                *reinterpret_cast<double2*>(&sm.v[j]) = make_double2(va, v);
                const double ta = j >= j0 && j < nst ? tt + dt : tt;
                tt = j + 1 >= j0 && j + 1 < nst ? ta + dt : ta;
                *reinterpret_cast<double2*>(&sm.t[j]) = make_double2(ta, tt);
            }
            // tc after the steps j0..j-1 (j > j0)
            auto time_after = [&](int j) -> double { return rpos >= j0 && rpos < j ? ts[j - rpos] : sm.t[j - 1]; };
            __syncwarp();
            const double s_l = sm.v[lane];
            const bool inseg = lane >= j0 && lane < nst;
            const unsigned npos = __ballot_sync(full, inseg && !((posmask >> lane) & 1u));
            const unsigned cross = __ballot_sync(full, inseg && s_l >= delta);
            const unsigned nearm = __ballot_sync(full, inseg && fabs(s_l - delta) < p.near_eps);
            const unsigned stopm = npos | cross;
            f = stopm ? __ffs(stopm) - 1 : nst;
            near += (unsigned long long)__popc(f < 32 ? (nearm & ((1u << f) - 1u)) : nearm);
            if (f == nst) {
                v0 = v;
                tc = time_after(nst);
            } else if (f > j0) {
                v0 = sm.v[f - 1];
                tc = time_after(f);
            }
            if (rpos >= j0 && rpos < f) start_block();
            __syncwarp();
            if (f >= nst) break;
        }
        slow_step(f);
        j0 = f + 1;
    }
    return IafState{v0, tc, delta, near, count, cnt_block, block, next_reset, lim_block, stop, limit_hit};
}

// Bound: latency.  A chunk's membrane chain is 32 dependent float64 adds of
// 8.6 cycles, and about twice that goes into the shared-memory reads, votes
// and branches around it; seven warps per SM leave both exposed.  Measured at
// 1024 neurons x 10,000 samples (spikes in 8 % of the chunks, a block start in a
// third): 312 us with every chunk tested step by step, samples prefetched into
// registers (each shift waited for the newest load) and chains with a block
// start predicated step by step; 214 us here.  Chunks of 64 steps, and chunks
// restarted after each crossing from a ring of samples: 240 us.
template <bool RT>
__global__ void __launch_bounds__(kIafWarps * 32, 1) iaf_scan_kernel(const __grid_constant__ IafArgs p) {
    __shared__ __align__(16) IafWarp warps[kIafWarps];
    __shared__ double s_ts[33];            // k-fold sums of dt from 0, in the order the time recursion adds them
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < 33; ++k) {
            s_ts[k] = t;
            t = t + p.dt;
        }
    }
    __syncthreads();
    const int n = blockIdx.x * kIafWarps + w;
    if (n >= p.N) return;  // uniform per warp
    IafWarp& sm = warps[w];

    const double kap = p.kappa[n];
    const double bia = p.bias[n];
    const double dt = p.dt;
    const int steps = p.F - 1;
    const int bstep = p.block_frames - 1;
    const int lim_full = iaf_limit(p.block_rate, p.block_frames);
    // the one block with fewer frames is the last
    const int last = p.F >= p.block_frames && bstep > 0 ? (p.F - p.block_frames) / bstep + 1 : 0;
    const int lim_last = iaf_limit(p.block_rate, p.F - last * bstep);
    IafState st{p.v0[n], p.time_count[n], RT ? p.delta_value[n] : p.delta[n], 0ull, 0, 0, 0,
                bstep > 0 ? bstep : 0x7fffffff, p.F >= p.block_frames ? lim_full : lim_last, false, false};
    const double* base = p.in + (int64_t)n * p.ns;
    auto ld = [&](int t) -> double { return t < p.F ? __ldg(base + (int64_t)t * p.ts) : 0.0; };

    // (x + b) / kappa; a quotient by 1 is its dividend
    const bool unit = kap == 1.0;
    auto drive = [&](double x) -> double {
        const double y = x + bia;
        return unit ? y : iaf_quotient(y, kap);
    };
    // the chunk in hand (y1, y2 of each lane's step, its area in sm.area[cur])
    // and the two after it
    double y1 = drive(ld(lane)), y2, ynext = drive(ld(32 + lane)), ynn = drive(ld(64 + lane));
    int cur = 0;
    auto prepare = [&](double ya, double yb, int b) -> double {   // areas of the chunk ya, whose successor is yb
        double z = __shfl_down_sync(full, ya, 1);
        const double z0 = __shfl_sync(full, yb, 0);
        if (lane == 31) z = z0;
        sm.area[b][lane] = (ya + z) / 2 * dt;
        return z;
    };
    y2 = prepare(y1, ynext, 0);
    // Input samples beyond ynext: a ring of kIafAhead chunks in shared memory,
    // filled by asynchronous copies (each lane copies and reads its own
    // sample), so that no register waits for a load that is still in flight.
    auto copy = [&](int t, int slot) {
        const unsigned dst = (unsigned)__cvta_generic_to_shared(sm.in + slot * 32 + lane);
        const int bytes = t < p.F ? 8 : 0;
        const double* src = bytes ? base + (int64_t)t * p.ts : base;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (int i = 0; i < kIafAhead; ++i) copy(96 + 32 * i + lane, i);

    int slot = 0;
    const bool fastok = bstep >= 32 || bstep <= 0;
    auto below_of = [&](double delta) -> double {
        const double b = delta - 2 * p.near_eps;
        return b - fabs(b) * 1e-15;
    };
    double below = below_of(st.delta);
    // every step of the positive-slope form with an area >= 0
    auto rises = [&]() -> bool {
        return __all_sync(full, (y2 >= 0 || (y2 < 0 && y1 <= 0)) && (y1 + y2) / 2 * dt >= 0);
    };
    bool rising = rises();
    __syncwarp();
    for (int t0 = 0; t0 < steps && !st.stop; t0 += 32) {
        const int nst = min(32, steps - t0);
        double ar[32];
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
            const double2 q = *reinterpret_cast<const double2*>(&sm.area[cur][j]);
            ar[j] = q.x;
            ar[j + 1] = q.y;
        }
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kIafAhead - 1) : "memory");
        const double x3 = sm.in[slot * 32 + lane];
        // the next chunk, prepared while this one's chain runs
        const double z = prepare(ynext, ynn, cur ^ 1);
        // A whole chunk of positive-slope steps with areas >= 0: the membrane
        // does not fall, so the chunk has no crossing, and no value near the
        // threshold, where its last value stays below both (the common case;
        // `below` is under delta and under every value counted as near it).
        bool done = false;
        double v = st.v0, tt = st.tc;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            v = v + ar[j];
            tt = tt + dt;
        }
        asm volatile("" : "+d"(tt));               // the two chains run side by side, not tt's after the test
        if (fastok && nst == 32 && rising) {
            if (v < below) {
                done = true;
                st.v0 = v;
                st.tc = tt;
                if (st.next_reset < t0 + 32) {     // a frame block starts inside: its time runs from there
                    st.tc = s_ts[32 - (st.next_reset - t0)];
                    st.cnt_block = 0;
                    ++st.block;
                    st.next_reset += bstep;
                    st.lim_block = p.F - st.block * bstep >= p.block_frames ? lim_full : lim_last;
                }
            }
        }
        if (!done) {
            const unsigned posmask = __ballot_sync(full, y2 >= 0 || (y2 < 0 && y1 <= 0));
            sm.y1[lane] = y1;
            sm.y2[lane] = y2;
            __syncwarp();
            st = iaf_walk<RT>(p, st, sm, sm.area[cur], s_ts, n, t0, nst, posmask, lim_full, lim_last);
            below = below_of(st.delta);
        }
        y1 = ynext;
        y2 = z;
        ynext = ynn;
        ynn = drive(x3);
        cur ^= 1;
        rising = rises();
        __syncwarp();                              // areas written by every lane before any lane's chain reads them
        copy(t0 + 96 + 32 * kIafAhead + lane, slot);   // refill the slot just read
        slot = slot + 1 == kIafAhead ? 0 : slot + 1;
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    if (lane == 0) {
        p.v0[n] = st.v0;
        p.time_count[n] = st.tc;
        p.spike_count[n] = st.count;
        if (RT) p.delta_value[n] = st.delta;
        if (p.near_count && st.near) atomicAdd(p.near_count, st.near);
        if (p.status) {
            if (st.limit_hit) atomicExch(p.status, VTB_BLOCK_LIMIT);
            else if (st.stop) atomicCAS(p.status, 0, VTB_OVERFLOW);
        }
    }
}

// offs[n] = pairs of the neurons before n (max(count - 1, 0) each), meta[0] =
// all of them (one block, any N).  Bound: launches and host reads; with
// spike_window_kernel it takes the place of five torch launches, and of one of
// the two reads that the pairs' count and the window test took (encoding and
// pairing 1024 neurons x 10,000 samples: 418 -> 378 us).
__global__ void __launch_bounds__(1024) spike_offsets_kernel(const int32_t* __restrict__ count, int N,
                                                             int64_t* __restrict__ offs, int64_t* __restrict__ meta) {
    __shared__ int64_t s_w[32];
    __shared__ int64_t s_base;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_base = 0;
    __syncthreads();
    for (int n0 = 0; n0 < N; n0 += 1024) {
        const int n = n0 + threadIdx.x;
        const int64_t c = n < N ? max(count[n] - 1, 0) : 0;
        int64_t x = c;
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_w[w] = x;
        __syncthreads();
        int64_t before = s_base;
        for (int k = 0; k < w; ++k) before += s_w[k];
        if (n < N) offs[n] = before + x - c;
        __syncthreads();
        if (threadIdx.x == 1023) s_base = before + x;
        __syncthreads();
    }
    if (threadIdx.x == 0) meta[0] = s_base;
}

// meta[1] = 1 if a spike lies outside (0, T); one warp per neuron
__global__ void __launch_bounds__(256) spike_window_kernel(const double* __restrict__ time,
                                                           const int32_t* __restrict__ step,
                                                           const int32_t* __restrict__ count, int N, int cap, int bstep,
                                                           double R, double t0, double T, int64_t* __restrict__ meta) {
    const int n = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (n >= N) return;
    const int c = min(count[n], cap);
    bool bad = false;
    for (int j = lane; j < c; j += 32) {
        const int64_t k = (int64_t)n * cap + j;
        const double t = time[k] + (double)(step[k] / bstep) * R - t0;
        bad |= !(t > 0.0 && t < T);
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicExch(reinterpret_cast<unsigned long long*>(meta + 1), 1ull);
}

// Consecutive pairs of each neuron's spikes, one warp per neuron (this file
// is compiled without FMA contraction, so t rounds as the reference's
// expression time + block * refresh - t0 does).
__global__ void __launch_bounds__(256) spike_pairs_kernel(const double* __restrict__ time,
                                                          const int32_t* __restrict__ step,
                                                          const int32_t* __restrict__ count, int N, int cap,
                                                          int bstep, double R, double t0, double T,
                                                          const int64_t* __restrict__ offs, double* __restrict__ tk1,
                                                          double* __restrict__ tk2, int32_t* __restrict__ ind,
                                                          int32_t* __restrict__ outside) {
    const int n = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (n >= N) return;
    const int c = min(count[n], cap);
    const int64_t o = offs[n];
    bool bad = false;
    for (int j = lane; j < c; j += 32) {
        const int64_t k = (int64_t)n * cap + j;
        const double blk = (double)(step[k] / bstep);
        const double t = time[k] + blk * R - t0;
        bad |= !(t > 0.0 && t < T);
        if (j + 1 < c) {
            tk1[o + j] = t;
            ind[o + j] = n;
        }
        if (j > 0) tk2[o + j - 1] = t;
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicExch(outside, 1);
}

}  // namespace vtb

using namespace vtb;

VTB_API int vtb_iaf_encode(const double* input, int64_t in_t_stride, int64_t in_n_stride, int N, int F,
                           int block_frames, double dt, const double* kappa, const double* bias,
                           const double* delta, double* v0, double* time_count, const double* randn,
                           int64_t randn_block_stride, int64_t randn_slot_stride, int64_t randn_n_stride,
                           int randn_block_cap, const double* sigma, double* delta_value, double* spike_time,
                           int32_t* spike_step, int32_t* spike_count, int cap,
                           unsigned long long* near_count, double near_eps, int32_t* status, double block_rate,
                           void* stream) {
    VTB_CHECK_ARG(N >= 0 && F >= 0 && block_frames >= 1 && cap >= 1);
    if (N == 0) return VTB_OK;
    VTB_CHECK_ARG(input && kappa && bias && delta && v0 && time_count && spike_time && spike_step &&
                  spike_count);
    if (randn) VTB_CHECK_ARG(sigma && delta_value && randn_block_cap >= 1);
    IafArgs a{input, in_t_stride, in_n_stride, N, F, block_frames, dt, kappa, bias, delta, v0, time_count,
              randn, randn_block_stride, randn_slot_stride, randn_n_stride, randn_block_cap, sigma,
              delta_value, spike_time, spike_step, spike_count, cap, near_count, near_eps, status, block_rate};
    const int blocks = ceil_div(N, kIafWarps);
    if (randn)
        iaf_scan_kernel<true><<<blocks, kIafWarps * 32, 0, as_stream(stream)>>>(a);
    else
        iaf_scan_kernel<false><<<blocks, kIafWarps * 32, 0, as_stream(stream)>>>(a);
    return launch_status();
}

VTB_API int vtb_spike_pairs(const double* spike_time, const int32_t* spike_step, const int32_t* spike_count, int N,
                            int cap, int block_frames, double refresh_interval, double t0, double T,
                            const int64_t* offsets, double* tk1, double* tk2, int32_t* ind, int32_t* outside,
                            void* stream) {
    VTB_CHECK_ARG(N >= 0 && cap >= 1 && block_frames >= 2);
    if (N == 0) return VTB_OK;
    VTB_CHECK_ARG(spike_time && spike_step && spike_count && offsets && outside);
    spike_pairs_kernel<<<ceil_div((int64_t)N * 32, 256), 256, 0, as_stream(stream)>>>(
        spike_time, spike_step, spike_count, N, cap, block_frames - 1, refresh_interval, t0, T, offsets, tk1, tk2,
        ind, outside);
    return launch_status();
}

VTB_API int vtb_spike_offsets(const double* spike_time, const int32_t* spike_step, const int32_t* spike_count, int N,
                              int cap, int block_frames, double refresh_interval, double t0, double T, int64_t* offsets,
                              int64_t* meta, void* stream) {
    VTB_CHECK_ARG(N >= 0 && cap >= 1 && block_frames >= 2 && meta);
    cudaStream_t s = as_stream(stream);
    VTB_CUDA_TRY(cudaMemsetAsync(meta, 0, 16, s));
    if (N == 0) return VTB_OK;
    VTB_CHECK_ARG(spike_time && spike_step && spike_count && offsets);
    spike_offsets_kernel<<<1, 1024, 0, s>>>(spike_count, N, offsets, meta);
    spike_window_kernel<<<ceil_div((int64_t)N * 32, 256), 256, 0, s>>>(spike_time, spike_step, spike_count, N, cap,
                                                                      block_frames - 1, refresh_interval, t0, T, meta);
    return launch_status();
}
