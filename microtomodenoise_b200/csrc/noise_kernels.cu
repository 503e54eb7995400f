// Noise-level estimators on the device (Noise/noiselevel.cpp).
//
//  * patch std: one thread per sample, the 15x15 sums accumulated in the
//    reference's order in float (noiselevel.cpp:235-283), so every per-sample
//    std equals the reference's bit for bit.
//  * two-cluster hard EM (noiselevel.cpp:366-528): one thread-block cluster
//    per z window (z-adaptive) or over all samples (global), the samples and
//    their assignments in registers. The per-sample decisions equal the
//    reference's formulas; the cluster sums, counts and variances are accumulated
//    in FP64 (warp shuffles, shared memory, then the cluster's CTAs). Windows
//    larger than a cluster holds run one CTA over a global int8 scratch array.
//  * neighbour fill of empty windows (noiselevel.cpp:571-603) and
//    sigma = mean + shift*std, sequential in one thread (nz is small).
#include <cooperative_groups.h>

#include <mutex>

#include "common.cuh"
#include "noise_kernels.cuh"

namespace inlm {

__global__ void __launch_bounds__(256) noise_patchstd_kernel(const float* __restrict__ stack,
                                                             long long pitch_y, long long pitch_z,
                                                             int nx, long long nslice,
                                                             const long long* __restrict__ samples,
                                                             long long n, int patchsize,
                                                             float* __restrict__ out, int z_base) {
    long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s >= n) return;
    long long idx = samples[s];
    // stack holds slices z_base.. (a z-slab of the volume, or all of it)
    int z0 = (int)(idx / nslice);
    idx -= (long long)z_base * nslice;
    z0 -= z_base;
    int y0 = (int)((idx - z0 * nslice) / nx);
    int x0 = (int)(idx - z0 * nslice - (long long)y0 * nx);
    const int patchlength = patchsize * patchsize;
    float sum = 0.0f;
    for (int y = y0; y < y0 + patchsize; y++) {
        const float* row = stack + z0 * pitch_z + (long long)y * pitch_y + x0;
        for (int x = 0; x < patchsize; x++) sum = __fadd_rn(sum, row[x]);
    }
    float mean = __fdiv_rn(sum, (float)patchlength);
    float sq = 0.0f;
    for (int y = y0; y < y0 + patchsize; y++) {
        const float* row = stack + z0 * pitch_z + (long long)y * pitch_y + x0;
        for (int x = 0; x < patchsize; x++) {
            float d = __fsub_rn(row[x], mean);
            sq = __fadd_rn(sq, __fmul_rn(d, d));
        }
    }
    out[s] = __fsqrt_rn(__fdiv_rn(sq, (float)patchlength));
}

// Gaussian membership as written at noiselevel.cpp:456-457: 1./sqrtf(...) is a
// double division and the product is rounded to float.
__device__ __forceinline__ float cluster_prob(float v, float mean, float var) {
    const float PI = 3.141592654f;
    float d = __fsub_rn(v, mean);
    float q = __fdiv_rn(__fmul_rn(d, d), __fmul_rn(2.f, var));
    float e = expf(-q);
    double inv = __ddiv_rn(1.0, (double)__fsqrt_rn(__fmul_rn(__fmul_rn(var, 2.f), PI)));
    return __double2float_rn(__dmul_rn(inv, (double)e));
}

constexpr int kEmThreads = 256;

struct EmRed {
    double s1, s2;
    long long n1, n2;
};

// Block-wide sum of (s1, s2, n1, n2) and OR of flag; result broadcast to all
// NT threads.
template <int NT>
__device__ __forceinline__ void block_reduce(EmRed& r, int& flag, EmRed* sh, int* shflag) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        r.s1 += __shfl_down_sync(0xffffffffu, r.s1, o);
        r.s2 += __shfl_down_sync(0xffffffffu, r.s2, o);
        r.n1 += __shfl_down_sync(0xffffffffu, r.n1, o);
        r.n2 += __shfl_down_sync(0xffffffffu, r.n2, o);
    }
    int any = __any_sync(0xffffffffu, flag);
    __syncthreads();
    if (lane == 0) {
        sh[warp] = r;
        shflag[warp] = any;
    }
    __syncthreads();
    if (warp == 0) {
        constexpr int NW = NT / 32;
        EmRed t = (lane < NW) ? sh[lane] : EmRed{0.0, 0.0, 0, 0};
        int f = (lane < NW) ? shflag[lane] : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            t.s1 += __shfl_down_sync(0xffffffffu, t.s1, o);
            t.s2 += __shfl_down_sync(0xffffffffu, t.s2, o);
            t.n1 += __shfl_down_sync(0xffffffffu, t.n1, o);
            t.n2 += __shfl_down_sync(0xffffffffu, t.n2, o);
        }
        f = __any_sync(0xffffffffu, f);
        if (lane == 0) {
            sh[0] = t;
            shflag[0] = f;
        }
    }
    __syncthreads();
    r = sh[0];
    flag = shflag[0];
    __syncthreads();
}

// Two-cluster EM over values[fs..ls] by one CTA of NT threads; asg[i] holds
// sample i's cluster (-1 excluded, 0, 1). Writes out_mean[w], out_sd[w].
template <int NT>
__device__ __forceinline__ void em_window(const float* __restrict__ values, int fs, int ls,
                                          signed char* __restrict__ asg, int w,
                                          float* __restrict__ out_mean,
                                          float* __restrict__ out_sd) {
    __shared__ EmRed sh[NT / 32];
    __shared__ int shflag[NT / 32];
    __shared__ float shmin[NT / 32], shmax[NT / 32];
    // assignments indexed by sample id
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    // min / max (noiselevel.cpp:384-390)
    float mn = 1e20f, mx = -1e20f;
    for (int i = fs + tid; i <= ls; i += NT) {
        float v = values[i];
        mn = fminf(mn, v);
        mx = fmaxf(mx, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_down_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, o));
    }
    if (lane == 0) {
        shmin[warp] = mn;
        shmax[warp] = mx;
    }
    __syncthreads();
    mn = 1e20f;
    mx = -1e20f;
    for (int q = 0; q < NT / 32; q++) {
        mn = fminf(mn, shmin[q]);
        mx = fmaxf(mx, shmax[q]);
    }
    float range = __fsub_rn(mx, mn);
    float mean1 = __double2float_rn(__dadd_rn((double)mn, __dmul_rn(0.25, (double)range)));
    float mean2 = __double2float_rn(__dsub_rn((double)mx, __dmul_rn(0.25, (double)range)));

    // initial assignment, zero values excluded (noiselevel.cpp:398-423)
    EmRed r{0.0, 0.0, 0, 0};
    int flag = 0;
    for (int i = fs + tid; i <= ls; i += NT) {
        float v = values[i];
        signed char a;
        if (v == 0.0f) {
            a = -1;
        } else if (fabsf(__fsub_rn(v, mean1)) < fabsf(__fsub_rn(v, mean2))) {
            a = 0;
            r.s1 += (double)v;
            r.n1++;
        } else {
            a = 1;
            r.s2 += (double)v;
            r.n2++;
        }
        asg[i] = a;
    }
    block_reduce<NT>(r, flag, sh, shflag);
    if (r.n1 > 0) mean1 = __double2float_rn(r.s1 / (double)r.n1);
    if (r.n2 > 0) mean2 = __double2float_rn(r.s2 / (double)r.n2);
    if (r.n1 == 0 && r.n2 == 0) {
        if (tid == 0) {
            out_mean[w] = 0.0f;
            out_sd[w] = 0.0f;
        }
        return;
    }
    long long n1 = r.n1, n2 = r.n2;

    // cluster variances (noiselevel.cpp:428-443)
    auto variances = [&](float m1, float m2, float& v1, float& v2) {
        EmRed q{0.0, 0.0, 0, 0};
        int f = 0;
        for (int i = fs + tid; i <= ls; i += NT) {
            float v = values[i];
            signed char a = asg[i];
            if (a == 0) {
                float d = __fsub_rn(v, m1);
                q.s1 += (double)__fmul_rn(d, d);
            } else if (a == 1) {
                float d = __fsub_rn(v, m2);
                q.s2 += (double)__fmul_rn(d, d);
            }
        }
        block_reduce<NT>(q, f, sh, shflag);
        v1 = __double2float_rn(q.s1 / (double)(n1 > 1 ? n1 : 1));
        v2 = __double2float_rn(q.s2 / (double)(n2 > 1 ? n2 : 1));
    };
    __syncthreads();  // assignments visible to all threads
    float var1, var2;
    variances(mean1, mean2, var1, var2);

    // hard EM, at most 1000 passes (noiselevel.cpp:445-521)
    int change = 1;
    int iters = 0;
    while (change && var1 > 0.0f && var2 > 0.0f) {
        change = 0;
        iters++;
        EmRed q{0.0, 0.0, 0, 0};
        int f = 0;
        for (int i = fs + tid; i <= ls; i += NT) {
            float v = values[i];
            if (v == 0.0f) continue;
            float p1 = cluster_prob(v, mean1, var1);
            float p2 = cluster_prob(v, mean2, var2);
            signed char a = asg[i];
            if (p2 > p1) {
                if (a != 1) {
                    f = 1;
                    asg[i] = 1;
                }
                q.s2 += (double)v;
                q.n2++;
            } else {
                if (a != 0) {
                    f = 1;
                    asg[i] = 0;
                }
                q.s1 += (double)v;
                q.n1++;
            }
        }
        block_reduce<NT>(q, f, sh, shflag);
        change = f;
        n1 = q.n1;
        n2 = q.n2;
        if (n1 > 0) mean1 = __double2float_rn(q.s1 / (double)n1);
        if (n2 > 0) mean2 = __double2float_rn(q.s2 / (double)n2);
        variances(mean1, mean2, var1, var2);
        if (iters == 1000) break;
    }
    if (tid == 0) {
        if (mean1 <= mean2 || var2 <= 0.0f) {
            out_mean[w] = mean1;
            out_sd[w] = __fsqrt_rn(var1);
        } else {
            out_mean[w] = mean2;
            out_sd[w] = __fsqrt_rn(var2);
        }
    }
}

// ---- EM with the window in the registers of a cluster ----
//
// What bounds it: dependent passes (25 to 120, at most 1000) of two reductions
// each, and issue slots (60 % busy with 256 windows). So a window's samples stay
// in registers (VPT per thread) over up to 8 CTAs instead of being read from L2
// in every pass, a decision takes a dozen FP32 operations, and a reduction is
// one warp-shuffle tree, one barrier in the CTA and one in the cluster. A global
// estimate of 100000 samples takes 0.21 ms (one 1024-thread CTA: 2.49 ms), 256
// windows of up to 39000 samples 0.73 ms (1.67 ms), 4000 samples 0.060 ms (0.18 ms).
//
// Decision: p2 > p1 with p = float(1/sqrt(2 pi var) * expf(-q)) as cluster_prob
// rounds it. In logarithms that is t = q1 - q2 + ln(var1/var2)/2 > 0, and every
// rounding of either side moves t by less than 1e-6 (8 + q1 + q2 + |ln var1| +
// |ln var2|). Where |t| exceeds twice that and one of the exponentials is a normal
// number, its sign decides; any other sample (near a tie, an underflow, a NaN)
// takes cluster_prob itself.
constexpr int kEmClusterThreads = 512;
constexpr int kEmManyThreads = 256, kEmManyValues = 40;  // the shape for many windows
constexpr int kEmMaxCluster = 8;
constexpr int kEmSms = 148;
constexpr int kEmMaxValues = 28;  // per thread (64 registers at two CTAs per SM)

struct __align__(16) EmPartial {
    double s1, s2;
    int n1, n2, flag, pad;
};

// Sums (s1, s2 and, with COUNTS, n1, n2) and the OR of flag over the cluster, in
// an order that depends on nothing but the launch; all threads of all its CTAs
// call it and get the result. The two sums share one shuffle tree: lanes 0-15
// carry s1, lanes 16-31 s2.
template <int NT, bool COUNTS>
__device__ __forceinline__ void cluster_sum(EmPartial& r, EmPartial* warp_part, EmPartial (*slots)[kEmMaxCluster],
                                            int& parity, int ctas, unsigned rank) {
    namespace cg = cooperative_groups;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NW = NT / 32;
    static_assert(NW <= 16, "one partial per lane of a half warp");
    const bool low = lane < 16;
    double x = (low ? r.s1 : r.s2) + __shfl_xor_sync(0xffffffffu, low ? r.s2 : r.s1, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    EmPartial* part = warp_part + parity * NW;
    if (COUNTS) {
        r.n1 = __reduce_add_sync(0xffffffffu, r.n1);
        r.n2 = __reduce_add_sync(0xffffffffu, r.n2);
        r.flag = __any_sync(0xffffffffu, r.flag);
        if (lane == 0) *reinterpret_cast<int4*>(&part[warp].n1) = make_int4(r.n1, r.n2, r.flag, 0);
    }
    if (lane == 0) part[warp].s1 = x;
    if (lane == 16) part[warp].s2 = x;
    __syncthreads();
    x = (lane & 15) >= NW ? 0.0 : low ? part[lane].s1 : part[lane - 16].s2;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    r.s1 = __shfl_sync(0xffffffffu, x, 0);
    r.s2 = __shfl_sync(0xffffffffu, x, 16);
    if (COUNTS) {
        const int4 c = lane < NW ? *reinterpret_cast<const int4*>(&part[lane].n1) : make_int4(0, 0, 0, 0);
        r.n1 = __reduce_add_sync(0xffffffffu, c.x);
        r.n2 = __reduce_add_sync(0xffffffffu, c.y);
        r.flag = __any_sync(0xffffffffu, c.z);
    }
    if (ctas > 1) {
        cg::cluster_group cl = cg::this_cluster();
        if (warp == 0 && lane < ctas) *cl.map_shared_rank(&slots[parity][rank], lane) = r;
        cl.sync();
        r = slots[parity][0];
        for (int c = 1; c < ctas; c++) {
            const EmPartial& u = slots[parity][c];
            r.s1 += u.s1;
            r.s2 += u.s2;
            if (COUNTS) {
                r.n1 += u.n1;
                r.n2 += u.n2;
                r.flag |= u.flag;
            }
        }
    }
    parity ^= 1;  // the other buffers, so that one barrier per sum suffices
}

// float(s1 / n1) and float(s2 / n2): one division, half a warp each.
__device__ __forceinline__ float2 quotients(double s1, double s2, int n1, int n2) {
    const bool low = (threadIdx.x & 31) < 16;
    const float f = __double2float_rn((low ? s1 : s2) / (double)(low ? n1 : n2));
    return make_float2(__shfl_sync(0xffffffffu, f, 0), __shfl_sync(0xffffffffu, f, 16));
}

// One bit per sample of a thread.
template <int N>
struct Bits {
    unsigned w[(N + 31) / 32];
    __device__ __forceinline__ bool operator[](int k) const { return w[k / 32] >> (k % 32) & 1u; }
    __device__ __forceinline__ void set(int k) { w[k / 32] |= 1u << (k % 32); }
    __device__ __forceinline__ void put(int k, bool b) { w[k / 32] = (w[k / 32] & ~(1u << (k % 32))) | (unsigned)b << (k % 32); }
    template <class F>
    __device__ __forceinline__ static Bits map(F f) {
        Bits r;
#pragma unroll
        for (int i = 0; i < (N + 31) / 32; i++) r.w[i] = f(i);
        return r;
    }
    __device__ __forceinline__ int count() const {
        int n = 0;
#pragma unroll
        for (int i = 0; i < (N + 31) / 32; i++) n += __popc(w[i]);
        return n;
    }
};

template <int NT, int VPT>
__global__ void __launch_bounds__(NT, NT == kEmManyThreads ? 3 : 2)
    noise_em_cluster_kernel(const float* __restrict__ values, const int2* __restrict__ windows, int ctas,
                            float* __restrict__ out_mean, float* __restrict__ out_sd) {
    using B = Bits<VPT>;
    __shared__ EmPartial warp_part[2 * NT / 32];
    __shared__ EmPartial slots[2][kEmMaxCluster];
    __shared__ float range_part[2][2 * NT / 32];
    __shared__ float range_slots[kEmMaxCluster][2];
    namespace cg = cooperative_groups;
    // A CTA's shared memory may be written from outside once that CTA has
    // started: every one arrives here, and the first remote store waits for all.
    cg::cluster_group cl = cg::this_cluster();
    cl.barrier_arrive();
    const int w = blockIdx.x / ctas;
    const unsigned rank = blockIdx.x % ctas;
    const int fs = windows[w].x, ls = windows[w].y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int stride = NT * ctas;
    float v[VPT];
    B in = B::map([](int) { return 0u; });  // samples of the window that are not zero
    bool odd = false;   // one of them is not a number
    float mn = 1e20f, mx = -1e20f;
#pragma unroll
    for (int k = 0; k < VPT; k++) {
        const int i = fs + (int)rank * NT + tid + k * stride;
        v[k] = 0.0f;
        if (i <= ls) {
            v[k] = values[i];
            mn = fminf(mn, v[k]);
            mx = fmaxf(mx, v[k]);
            if (v[k] != 0.0f) in.set(k);
            odd |= v[k] != v[k];
        }
    }
    // min / max (noiselevel.cpp:384-390)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if (lane == 0) {
        range_part[0][warp] = mn;
        range_part[1][warp] = mx;
    }
    __syncthreads();
    for (int q = 0; q < NT / 32; q++) {
        mn = fminf(mn, range_part[0][q]);
        mx = fmaxf(mx, range_part[1][q]);
    }
    cl.barrier_wait();
    if (ctas > 1) {
        if (tid < ctas) {
            float* dst = cl.map_shared_rank(&range_slots[rank][0], tid);
            dst[0] = mn;
            dst[1] = mx;
        }
        cl.sync();
        for (int c = 0; c < ctas; c++) {
            mn = fminf(mn, range_slots[c][0]);
            mx = fmaxf(mx, range_slots[c][1]);
        }
    }
    const float range = __fsub_rn(mx, mn);
    float mean1 = __double2float_rn(__dadd_rn((double)mn, __dmul_rn(0.25, (double)range)));
    float mean2 = __double2float_rn(__dsub_rn((double)mx, __dmul_rn(0.25, (double)range)));

    // initial assignment, zero values excluded (noiselevel.cpp:398-423)
    int parity = 0;
    B two = B::map([](int) { return 0u; });  // samples of the second cluster
    EmPartial r;
    // the thread's cluster sums and counts under the assignment `two`
    auto sums = [&]() {
        double s1 = 0.0, s2 = 0.0;
        const B first = B::map([&](int i) { return in.w[i] & ~two.w[i]; });
#pragma unroll
        for (int k = 0; k < VPT; k++) {
            const double d = (double)v[k];
            if (two[k]) s2 += d;
            if (first[k]) s1 += d;
        }
        r.s1 = s1;
        r.s2 = s2;
        r.n1 = first.count();
        r.n2 = two.count();
    };
#pragma unroll
    for (int k = 0; k < VPT; k++)
        if (!(fabsf(__fsub_rn(v[k], mean1)) < fabsf(__fsub_rn(v[k], mean2)))) two.set(k);
    two = B::map([&](int i) { return two.w[i] & in.w[i]; });
    r.flag = 0;
    sums();
    double own1 = r.s1, own2 = r.s2;
    cluster_sum<NT, true>(r, warp_part, slots, parity, ctas, rank);
    float2 mean = quotients(r.s1, r.s2, r.n1, r.n2);
    if (r.n1 > 0) mean1 = mean.x;
    if (r.n2 > 0) mean2 = mean.y;
    if (r.n1 == 0 && r.n2 == 0) {
        if (rank == 0 && tid == 0) {
            out_mean[w] = 0.0f;
            out_sd[w] = 0.0f;
        }
        return;
    }
    int n1 = r.n1, n2 = r.n2;
    // cluster variances (noiselevel.cpp:428-443)
    float var1, var2;
    auto variances = [&]() {
        double s1 = 0.0, s2 = 0.0;
        const B first = B::map([&](int i) { return in.w[i] & ~two.w[i]; });
#pragma unroll
        for (int k = 0; k < VPT; k++) {
            const bool b = two[k];
            const float d = __fsub_rn(v[k], b ? mean2 : mean1);
            const double q = (double)__fmul_rn(d, d);
            if (b) s2 += q;
            if (first[k]) s1 += q;
        }
        EmPartial q;
        q.s1 = s1;
        q.s2 = s2;
        cluster_sum<NT, false>(q, warp_part, slots, parity, ctas, rank);
        const float2 var = quotients(q.s1, q.s2, max(n1, 1), max(n2, 1));
        var1 = var.x;
        var2 = var.y;
    };
    variances();

    // hard EM, at most 1000 passes (noiselevel.cpp:445-521)
    int change = 1;
    for (int iters = 0; change && var1 > 0.0f && var2 > 0.0f && iters < 1000; iters++) {
        const float l1 = logf(var1), l2 = logf(var2);
        const float shift = 0.5f * (l1 - l2);
        const float r1 = 0.5f / var1, r2 = 0.5f / var2;
        const float slack = 2e-6f * (8.f + fabsf(l1) + fabsf(l2));
        // the larger exponential of any sample is smallest at the ends of the
        // range or between the means
        auto q = [](float x, float m, float rv) { return (x - m) * (x - m) * rv; };
        const bool safe = fmaxf(fmaxf(fminf(q(mn, mean1, r1), q(mn, mean2, r2)),
                                      fminf(q(mx, mean1, r1), q(mx, mean2, r2))),
                                fminf(q(mean2, mean1, r1), q(mean1, mean2, r2))) < 80.f;
        B one = B::map([](int) { return 0u; });
        float nearest = 1e30f;
#pragma unroll
        for (int k = VPT - 1; k >= 0; k--) {
            const float d1 = v[k] - mean1, d2 = v[k] - mean2;
            const float q1 = d1 * d1 * r1, q2 = d2 * d2 * r2;
            const float t = q1 - q2 + shift;
            nearest = fminf(nearest, fmaf(-2e-6f, q1 + q2, fabsf(t)));
            one.w[k / 32] = __funnelshift_l(__float_as_uint(t), one.w[k / 32], 1);  // bit k: t < 0
        }
        B next = B::map([&](int i) { return ~one.w[i]; });
        if (!(nearest > slack) || !safe || odd) {
            for (int k = 0; k < VPT; k++) {
                const float x = values[min(fs + (int)rank * NT + tid + k * stride, ls)];
                const float q1 = q(x, mean1, r1), q2 = q(x, mean2, r2);
                if (safe && fmaf(-2e-6f, q1 + q2, fabsf(q1 - q2 + shift)) > 2.f * slack) continue;
                const bool b = cluster_prob(x, mean2, var2) > cluster_prob(x, mean1, var1);
                next.put(k, b);
            }
        }
        r.flag = 0;
#pragma unroll
        for (int i = 0; i < (VPT + 31) / 32; i++) {
            next.w[i] &= in.w[i];
            r.flag |= next.w[i] != two.w[i];
        }
        if (r.flag) {
            two = next;
            sums();
            own1 = r.s1;
            own2 = r.s2;
        }
        r.s1 = own1;
        r.s2 = own2;
        r.n1 = in.count() - two.count();  // two lies in in
        r.n2 = two.count();
        cluster_sum<NT, true>(r, warp_part, slots, parity, ctas, rank);
        change = r.flag;
        n1 = r.n1;
        n2 = r.n2;
        mean = quotients(r.s1, r.s2, n1, n2);
        if (n1 > 0) mean1 = mean.x;
        if (n2 > 0) mean2 = mean.y;
        variances();
    }
    if (rank == 0 && tid == 0) {
        if (mean1 <= mean2 || var2 <= 0.0f) {
            out_mean[w] = mean1;
            out_sd[w] = __fsqrt_rn(var1);
        } else {
            out_mean[w] = mean2;
            out_sd[w] = __fsqrt_rn(var2);
        }
    }
}

template <int NT, int VPT>
static cudaError_t launch_em_cluster(const float* values, const int2* windows, int n_windows, int ctas,
                                     float* out_mean, float* out_sd, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(n_windows * ctas);
    cfg.blockDim = dim3(NT);
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, noise_em_cluster_kernel<NT, VPT>, values, windows, ctas, out_mean, out_sd);
}

template <int NT>
__global__ void __launch_bounds__(NT) noise_em_kernel(const float* __restrict__ values,
                                                      const int2* __restrict__ windows,
                                                      const long long* __restrict__ scratch_off,
                                                      signed char* __restrict__ assign_scratch,
                                                      float* __restrict__ out_mean,
                                                      float* __restrict__ out_sd) {
    const int w = blockIdx.x;
    const int fs = windows[w].x, ls = windows[w].y;
    em_window<NT>(values, fs, ls, assign_scratch + scratch_off[w] - fs, w, out_mean, out_sd);
}

// ---- allocation-free EM: scratch in file-scope device arrays ----
//
// For callers that cannot allocate device memory. The cluster-assignment
// scratch (one byte per sample per window) and the window table live in
// static device arrays that every GPU loading this library holds until the
// process exits: 16 MiB + 256 KiB. Every call on a device shares them and
// leaves the last call's contents behind; calls whose work overlaps on the
// GPU (different streams, or different host threads) race on them.
// Nothing needs clearing between calls: the EM writes every assignment of a
// window (its initial pass) before it reads any, and every call rewrites the
// window-table entries it uses.
// The window table reaches the device inside kernel launch parameters (a
// small copy kernel per 1024 windows), so a call enqueues kernels only: no
// host-to-device copy from pageable memory and no wait on the host.
struct NoAllocWindow {
    int first, last;     // inclusive sample range (last < first: empty)
    long long offset;    // byte offset of the window's assignments in the scratch
};

static __device__ __align__(256) signed char g_noalloc_assign[kNoAllocAssignBytes];
static __device__ __align__(256) NoAllocWindow g_noalloc_windows[kNoAllocMaxWindows];

constexpr int kNoAllocChunk = 1024;  // windows per launch-parameter block (16 KiB)
struct NoAllocTableChunk {
    int base, count;
    NoAllocWindow win[kNoAllocChunk];
};

__global__ void __launch_bounds__(256) noalloc_table_kernel(const __grid_constant__ NoAllocTableChunk c,
                                                            NoAllocWindow* __restrict__ table) {
    for (int i = threadIdx.x; i < c.count; i += blockDim.x) table[c.base + i] = c.win[i];
}

__global__ void __launch_bounds__(kEmThreads) noise_em_noalloc_kernel(
    const float* __restrict__ values, const NoAllocWindow* __restrict__ windows,
    signed char* __restrict__ assign_scratch, float* __restrict__ out_mean,
    float* __restrict__ out_sd) {
    const int w = blockIdx.x;
    const NoAllocWindow win = windows[w];
    em_window<kEmThreads>(values, win.first, win.last, assign_scratch + win.offset - win.first, w,
                          out_mean, out_sd);
}

// Device addresses of the two arrays, looked up once per device with that
// device current (host code must not use the symbols themselves: they are
// host-side stand-ins, not device addresses).
struct NoAllocPtrs {
    bool ready = false;
    signed char* assign = nullptr;
    NoAllocWindow* windows = nullptr;
};
static NoAllocPtrs g_noalloc_ptrs[kNoAllocMaxDevices];
static std::mutex g_noalloc_mutex;

static cudaError_t noalloc_setup(int device, NoAllocPtrs* out) {
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    NoAllocPtrs& p = g_noalloc_ptrs[device];
    if (!p.ready) {
        int cur = -1;
        cudaError_t e = cudaGetDevice(&cur);
        if (e != cudaSuccess) return e;
        if (cur != device) return cudaErrorInvalidDevice;
        e = cudaGetSymbolAddress((void**)&p.assign, g_noalloc_assign);
        if (e != cudaSuccess) return e;
        e = cudaGetSymbolAddress((void**)&p.windows, g_noalloc_windows);
        if (e != cudaSuccess) return e;
        p.ready = true;
    }
    *out = p;
    return cudaSuccess;
}

cudaError_t launch_noise_em_noalloc(int device, const float* values, const long long* windows_host,
                                    int n_windows, float* out_mean, float* out_sd,
                                    cudaStream_t st) {
    if (n_windows <= 0) return cudaSuccess;
    if (device < 0 || device >= kNoAllocMaxDevices || n_windows > kNoAllocMaxWindows)
        return cudaErrorInvalidValue;
    NoAllocPtrs ptrs;
    cudaError_t e = noalloc_setup(device, &ptrs);
    if (e != cudaSuccess) return e;
    // the chunk is copied into the launch parameters when the kernel is enqueued
    static thread_local NoAllocTableChunk chunk;
    long long offset = 0;
    for (int base = 0; base < n_windows; base += kNoAllocChunk) {
        const int cnt = n_windows - base < kNoAllocChunk ? n_windows - base : kNoAllocChunk;
        chunk.base = base;
        chunk.count = cnt;
        for (int i = 0; i < cnt; i++) {
            const long long f = windows_host[2 * (base + i)], l = windows_host[2 * (base + i) + 1];
            NoAllocWindow& w = chunk.win[i];
            if (l < f) {  // empty: stored as 0..-1 whatever the caller's values
                w.first = 0;
                w.last = -1;
            } else {
                w.first = (int)f;
                w.last = (int)l;
            }
            w.offset = offset;
            offset += (long long)w.last - w.first + 1;
        }
        noalloc_table_kernel<<<1, 256, 0, st>>>(chunk, ptrs.windows);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    noise_em_noalloc_kernel<<<n_windows, kEmThreads, 0, st>>>(values, ptrs.windows, ptrs.assign,
                                                              out_mean, out_sd);
    return cudaGetLastError();
}

// Neighbour fill (z-adaptive) and sigma = mean + shift*sd. Slices without a
// filled mean are rare: only they send the fill through one thread.
constexpr int kFinalizeThreads = 256;
__global__ void __launch_bounds__(kFinalizeThreads) noise_finalize_kernel(float* __restrict__ mean, float* __restrict__ sd,
                                                                          int nz, int zadaptive, float shift,
                                                                          float* __restrict__ sigma) {
    if (!zadaptive) {
        const float s = __fadd_rn(mean[0], __fmul_rn(shift, sd[0]));
        for (int z = threadIdx.x; z < nz; z += kFinalizeThreads) sigma[z] = s;
        return;
    }
    int empty = 0;
    for (int z = threadIdx.x; z < nz; z += kFinalizeThreads) empty |= mean[z] == 0.0f;
    if (!__syncthreads_or(empty)) {
        for (int z = threadIdx.x; z < nz; z += kFinalizeThreads) sigma[z] = __fadd_rn(mean[z], __fmul_rn(shift, sd[z]));
        return;
    }
    if (threadIdx.x != 0) return;
    float max_std = -1.f;
    int zero = 0;
    for (int i = 0; i < nz; i++) {
        if (mean[i] > max_std) max_std = mean[i];
        if (mean[i] == 0.0f) zero = 1;
    }
    if (zero && max_std > 0.0f) {
        // every sweep fills at least one more slice next to a filled one
        for (int sweep = 0; zero && sweep <= nz; sweep++) {
            zero = 0;
            for (int i = 0; i < nz; i++) {
                float this_var = mean[i];
                if (this_var == 0.0f) {
                    float nv = 0.0f, nvs = 0.0f;
                    int count = 0;
                    if (i > 0 && mean[i - 1] > 0.0f) {
                        nv = __fadd_rn(nv, mean[i - 1]);
                        nvs = __fadd_rn(nvs, sd[i - 1]);
                        count++;
                    }
                    if (i < nz - 1 && mean[i + 1] > 0.0f) {
                        nv = __fadd_rn(nv, mean[i + 1]);
                        nvs = __fadd_rn(nvs, sd[i + 1]);
                        count++;
                    }
                    if (count > 0) {
                        this_var = __fdiv_rn(nv, (float)count);
                        mean[i] = this_var;
                        sd[i] = __fdiv_rn(nvs, (float)count);
                    }
                }
                if (this_var == 0.0f) zero = 1;
            }
        }
    }
    for (int z = 0; z < nz; z++) sigma[z] = __fadd_rn(mean[z], __fmul_rn(shift, sd[z]));
}

cudaError_t launch_noise_patchstd(const float* stack, long long pitch_y, long long pitch_z, int nx,
                                  long long nslice, const long long* samples, long long n,
                                  int patchsize, float* out, cudaStream_t st, int z_base) {
    if (n <= 0) return cudaSuccess;
    noise_patchstd_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
        stack, pitch_y, pitch_z, nx, nslice, samples, n, patchsize, out, z_base);
    return cudaGetLastError();
}

cudaError_t launch_noise_em(const float* values, const int2* windows, int n_windows,
                            const long long* scratch_off, signed char* scratch, float* out_mean,
                            float* out_sd, cudaStream_t st, long long mean_window, long long max_window) {
    if (n_windows <= 0) return cudaSuccess;
    // the fewest CTAs that hold the largest window, and more while the GPU has
    // idle SMs: a pass is then shorter
    if (max_window > 0 && max_window <= (long long)kEmMaxCluster * kEmClusterThreads * kEmMaxValues) {
        int ctas = 1;
        // Many windows: half the threads with more samples each, so that the
        // reductions take fewer of the issue slots. It pays where the CTAs are at
        // least 0.7 full and make two waves (three per SM); against 512 threads,
        // us, by windows x samples: 256 x 39000 650 / 651, 256 x 31000 694 / 743,
        // 600 x 32000 1241 / 1388, 600 x 80000 3516 / 3844, 1000 x 18000 1042 /
        // 1133; below that 256 x 27000 631 / 491, 600 x 43000 2884 / 1959, and with
        // fewer CTAs 300 x 18000 464 / 439, 600 x 9000 366 / 338.
        while ((long long)ctas * kEmManyThreads * kEmManyValues < max_window) ctas *= 2;
        if (ctas <= kEmMaxCluster && (long long)n_windows * ctas >= 6 * kEmSms &&
            10 * max_window >= 7ll * ctas * kEmManyThreads * kEmManyValues)
            return launch_em_cluster<kEmManyThreads, kEmManyValues>(values, windows, n_windows, ctas, out_mean, out_sd, st);
        ctas = 1;
        while ((long long)ctas * kEmClusterThreads * kEmMaxValues < max_window) ctas *= 2;
        // (a barrier of the cluster costs as much as a dozen samples per thread)
        while (ctas < kEmMaxCluster && (long long)n_windows * ctas * 2 <= kEmSms &&
               (long long)ctas * kEmClusterThreads * 12 < max_window)
            ctas *= 2;
        const long long per = (max_window + (long long)ctas * kEmClusterThreads - 1) / ((long long)ctas * kEmClusterThreads);
        if (per <= 4) return launch_em_cluster<kEmClusterThreads, 4>(values, windows, n_windows, ctas, out_mean, out_sd, st);
        if (per <= 12) return launch_em_cluster<kEmClusterThreads, 12>(values, windows, n_windows, ctas, out_mean, out_sd, st);
        if (per <= 20) return launch_em_cluster<kEmClusterThreads, 20>(values, windows, n_windows, ctas, out_mean, out_sd, st);
        return launch_em_cluster<kEmClusterThreads, kEmMaxValues>(values, windows, n_windows, ctas, out_mean, out_sd, st);
    }
    // long windows (few of them, e.g. a global estimate or a short stack) get
    // 1024 threads each so one CTA per window still keeps an SM busy
    if (mean_window >= kEmWideWindow)
        noise_em_kernel<1024><<<n_windows, 1024, 0, st>>>(values, windows, scratch_off, scratch,
                                                          out_mean, out_sd);
    else
        noise_em_kernel<kEmThreads><<<n_windows, kEmThreads, 0, st>>>(values, windows, scratch_off,
                                                                      scratch, out_mean, out_sd);
    return cudaGetLastError();
}

cudaError_t launch_noise_finalize(float* mean, float* sd, int nz, int zadaptive, float shift,
                                  float* sigma, cudaStream_t st) {
    noise_finalize_kernel<<<1, kFinalizeThreads, 0, st>>>(mean, sd, nz, zadaptive, shift, sigma);
    return cudaGetLastError();
}

}  // namespace inlm
