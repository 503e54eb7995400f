// Second kernel of the paired-offset FP32 form (filter_pair.cu): weights, sums
// and results of every voxel from the stored patch distances, all S offsets in
// reference order (Denoiser/iternlm_cpu.cpp:758-843).
#include <algorithm>

#include "common.cuh"
#include "filter_pair.cuh"
#include "pair_math.cuh"

namespace inlm {

namespace {

constexpr int kWeightWarps = 4;                      // consumer warps
constexpr int kWeightThreads = 32 * (kWeightWarps + 1);
constexpr int kWeightRows = 8;                       // y voxels per thread
constexpr int kWeightRowsSmall = 2;                  // ... of small volumes
constexpr int kWeightStages = 3;                     // stages of the ring
constexpr int kStageOffsets = 2;                     // offsets per stage (their number is even)
constexpr int kDistPitch = kPairDistBox;             // floats per staged distance row

// An offset's byte positions: of its distances in the stage (the copy starts on
// a multiple of 4 columns, up to 3 before the tile) and in the staged raw tile.
struct StageMeta {
    int dist, raw;
};

template <int ROWS, int RAWP>
struct WeightSmem {
    static constexpr int TY = kWeightWarps * ROWS;
    static constexpr int kTile = (TY * kDistPitch * 4 + 127) / 128 * 128;
    static constexpr int kStage = kStageOffsets * kTile;
    static constexpr int kHead = 256;  // barriers and metadata
    static int raw_bytes(int syr) { return ((TY + 2 * syr) * RAWP * 4 + 127) / 128 * 128; }
    static size_t bytes(int syr) { return kHead + kWeightStages * (size_t)kStage + 2 * (size_t)raw_bytes(syr); }
};

// Waits for a phase; the clock is read only when the first try fails.
__device__ __forceinline__ bool wait_phase(uint64_t* bar, uint32_t parity) {
    return mbar_try_wait(bar, parity) || mbar_wait_bounded(bar, parity);
}

// A CTA filters 32 columns x (4 warps x ROWS) rows of one plane, a consumer
// thread ROWS voxels along y. One producer thread streams the offsets'
// distance tiles, two offsets per stage, through a ring in shared memory by 4D
// TMA loads (the rows of x for the first half of the offsets, of x + s for the
// second; a copy starts on a multiple of 4 columns and is 4 columns wider than
// the tile), and the raw tile of each z plane that holds offsets (the reference
// order is z-major) through two buffers, so the consumers only wait on full
// barriers. Raw tiles are counted as they come, u = 0, 1, ...: u & 1 is the
// buffer and u >> 1 its use. A stage is armed before the raw tiles of its offsets
// are waited for: the consumers give tile u - 2 back when they enter tile u - 1,
// which may be in the same stage (one offset per plane at the ends of a thin
// search shape).
//
// What bounds it: DRAM and FP32 lanes alike. Every distance is read twice, 8
// bytes per voxel and pair of offsets: at 256 x 256 x 96, patch radius 2, search
// radius 5 the 13.9 GB take 2.76 ms, 5.0 TB/s, 0.77 of the measured copy
// bandwidth, with the FP32 pipe 66 % busy (20 operations per voxel and offset
// for the Pade quotient and the sums). Distances loaded into registers up to
// four offsets ahead took 3.48 ms, one offset per stage 2.87 ms; 16 rows per
// thread, 5 CTAs per SM or 8 warps per CTA changed it by less than 2 %.
template <int ROWS, int RAWP, bool FUSED>
__global__ void __launch_bounds__(kWeightThreads, 4)
    nlm_pair_weight_kernel(const __grid_constant__ CUtensorMap tm_dist, const __grid_constant__ CUtensorMap tm_raw,
                           const __grid_constant__ PairArgs a, int z_first) {
    using M = WeightSmem<ROWS, RAWP>;
    constexpr int NP = ROWS / 2;
    constexpr int NS = kWeightStages;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);
    uint64_t* empty = full + NS;
    uint64_t* raw_full = empty + NS;
    uint64_t* raw_empty = raw_full + 2;
    volatile StageMeta* meta = reinterpret_cast<volatile StageMeta*>(raw_empty + 2);
    unsigned char* ring = smem + M::kHead;
    unsigned char* rawb = ring + NS * M::kStage;
    const int raw_rows = M::TY + 2 * a.syr;
    const int raw_bytes = (raw_rows * RAWP * 4 + 127) / 128 * 128;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int xb = a.x0 + blockIdx.x * 32, yb = a.y0 + blockIdx.y * M::TY;
    const int z = z_first + blockIdx.z;
    if (tid == 0) {
        for (int i = 0; i < NS; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], kWeightWarps);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&raw_full[i], 1);
            mbar_init(&raw_empty[i], kWeightWarps);
        }
        fence_mbar_init();
    }
    __syncthreads();

    if (warp == kWeightWarps) {
        if (lane != 0) return;
        prefetch_tmap(&tm_dist);
        prefetch_tmap(&tm_raw);
        const int zr = z % a.ring, cx = xb - a.xs, cy = yb - a.ys;
        int g = -1, next = 0, stage = 0, u = 0, armed = 0;
        uint32_t phase = 1;  // of the empty barriers: the first round passes
        bool ok = true;
        for (int s = 0; s < a.S && ok; s += kStageOffsets) {
            ok = wait_phase(&empty[stage], phase);
            if (!ok) break;
            int x[kStageOffsets], y[kStageOffsets], zz[kStageOffsets];
#pragma unroll
            for (int i = 0; i < kStageOffsets; i++) {
                const PairOffset o = a.offsets[s + i];
                const bool first = s + i < a.H;
                x[i] = cx + (first ? 0 : o.x);
                y[i] = cy + (first ? 0 : o.y);
                zz[i] = zr + (first ? 0 : o.z);
                if (zz[i] >= a.ring) zz[i] -= a.ring;
                meta[stage * kStageOffsets + i].dist = i * M::kTile + (x[i] & 3) * 4;
                meta[stage * kStageOffsets + i].raw = (o.y * RAWP + o.x) * 4;
            }
            mbar_arrive_expect_tx(&full[stage], (uint32_t)(kStageOffsets * M::TY * kDistPitch * 4));
            armed++;
#pragma unroll
            for (int i = 0; i < kStageOffsets; i++)
                tma_load_4d(ring + stage * M::kStage + i * M::kTile, &tm_dist, x[i] & ~3, y[i], zz[i],
                            s + i < a.H ? s + i : a.S - 1 - s - i, &full[stage]);
#pragma unroll
            for (int i = 0; i < kStageOffsets; i++) {
                if (s + i != next || !ok) continue;
                while (s + i == next) next = a.z_start[++g + 1];
                const int b = u & 1;
                ok = wait_phase(&raw_empty[b], ((u >> 1) & 1) ^ 1);
                if (!ok) continue;
                mbar_arrive_expect_tx(&raw_full[b], (uint32_t)(raw_rows * RAWP * 4));
                // voxel xb - sxr is column px - sxr = RX of the box
                tma_load_3d(rawb + b * raw_bytes, &tm_raw, xb, yb - a.syr + a.py, z + g - a.szc + a.pz, &raw_full[b]);
                u++;
            }
            if (++stage == NS) {
                stage = 0;
                phase ^= 1u;
            }
        }
        if (!ok) {
            set_error(a.err, DEV_TMA_TIMEOUT);
            // let the copies in flight land before the CTA's memory goes away
            for (int q = max(0, armed - NS); q < armed; q++) mbar_wait_bounded(&full[q % NS], (q / NS) & 1);
            for (int q = max(0, u - 2); q < u; q++) mbar_wait_bounded(&raw_full[q & 1], (q >> 1) & 1);
        }
        return;
    }

    const int y = yb + warp * ROWS, x = xb + lane;
    const f32x2 m2 = splat2(a.mult[z]), neg0 = splat2(a.neg0);
    f32x2 acc[NP], wsum[NP];
    float wmax[ROWS];
#pragma unroll
    for (int p = 0; p < NP; p++) acc[p] = wsum[p] = 0ull;
#pragma unroll
    for (int r = 0; r < ROWS; r++) wmax[r] = 0.0f;
    const unsigned char* dlane = ring + (warp * ROWS * kDistPitch + lane) * 4;
    const unsigned char* rlane = rawb + ((warp * ROWS + a.syr) * RAWP + a.px + lane) * 4;
    const unsigned char* rcur = rlane;
    int g = -1, next = 0, stage = 0, u = 0;
    uint32_t phase = 0;
    for (int s = 0; s < a.S; s += kStageOffsets) {
        if (!wait_phase(&full[stage], phase)) {
            set_error(a.err, DEV_TMA_TIMEOUT);
            return;
        }
#pragma unroll
        for (int i = 0; i < kStageOffsets; i++) {
            if (s + i == next) {
                // this warp is done with the previous raw tile
                __syncwarp();
                if (u > 0 && lane == 0) mbar_arrive(&raw_empty[(u - 1) & 1]);
                while (s + i == next) next = a.z_start[++g + 1];
                if (!wait_phase(&raw_full[u & 1], (u >> 1) & 1)) {
                    set_error(a.err, DEV_TMA_TIMEOUT);
                    return;
                }
                rcur = rlane + (u & 1) * raw_bytes;
                u++;
            }
            const float* dq =
                reinterpret_cast<const float*>(dlane + stage * M::kStage + meta[stage * kStageOffsets + i].dist);
            const float* rq = reinterpret_cast<const float*>(rcur + meta[stage * kStageOffsets + i].raw);
            float d[ROWS], r[ROWS];
#pragma unroll
            for (int k = 0; k < ROWS; k++) d[k] = dq[k * kDistPitch];
#pragma unroll
            for (int k = 0; k < ROWS; k++) r[k] = rq[k * RAWP];
            if (i == kStageOffsets - 1) {
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[stage]);
            }
#pragma unroll
            for (int p = 0; p < NP; p++) {
                const f32x2 dd = pack2(d[2 * p], d[2 * p + 1]);
                if (FUSED)
                    fused_weight_pair(dd, m2, make_float2(r[2 * p], r[2 * p + 1]), acc[p], wsum[p], wmax[2 * p],
                                      wmax[2 * p + 1]);
                else
                    exact_weight_pair_fast(dd, m2, pack2(r[2 * p], r[2 * p + 1]), neg0, acc[p], wsum[p], wmax[2 * p],
                                           wmax[2 * p + 1]);
            }
        }
        if (++stage == NS) {
            stage = 0;
            phase ^= 1u;
        }
    }
    if (x >= a.x1) return;
    const float* rc = a.raw_pad + (long long)(z + a.pz) * a.gpitch_z + (long long)(y + a.py) * a.gpitch_y + (x + a.px);
#pragma unroll
    for (int i = 0; i < ROWS; i++) {
        if (y + i >= a.y1) break;
        const float raw0 = __ldg(rc + i * a.gpitch_y);
        const float2 acp = unpack2(acc[i / 2]), wsp = unpack2(wsum[i / 2]);
        float ac = (i & 1) ? acp.y : acp.x;
        float ws = (i & 1) ? wsp.y : wsp.x;
        float res = raw0;
        if (wmax[i] > 0.0f) {
            ac = __fadd_rn(ac, __fmul_rn(wmax[i], raw0));
            ws = __fadd_rn(ws, wmax[i]);
            res = __fdiv_rn(ac, ws);
        }
        a.out[((long long)z * a.ny + y + i) * a.nx + x] = res;
    }
}

template <int ROWS, int RAWP>
cudaError_t launch_rows(bool fused, const PairMaps& m, const PairArgs& a, int z0, int z1, cudaStream_t st) {
    using M = WeightSmem<ROWS, RAWP>;
    const size_t smem = M::bytes(a.syr);
    auto kern = fused ? nlm_pair_weight_kernel<ROWS, RAWP, true> : nlm_pair_weight_kernel<ROWS, RAWP, false>;
    cudaError_t e = allow_shared_memory(kern, smem);
    if (e != cudaSuccess) return e;
    // a plane per grid z, of which a launch takes 65535
    for (int z = z0; z < z1; z += kPairGridZ) {
        const dim3 grid((a.x1 - a.x0 + 31) / 32, (a.y1 - a.y0 + M::TY - 1) / M::TY, std::min(kPairGridZ, z1 - z));
        kern<<<grid, kWeightThreads, smem, st>>>(m.dist[ROWS != kWeightRows], m.raw[ROWS != kWeightRows], a, z);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

__global__ void __launch_bounds__(256) weight_mismatch_kernel(unsigned long long* n, float nz) {
    const unsigned last = __float_as_uint(-3.6f);
    const f32x2 one = splat2(1.f);
    for (unsigned b = 0x80000000u + blockIdx.x * 256u + threadIdx.x; b <= last; b += gridDim.x * 256u) {
        const f32x2 x = splat2(__uint_as_float(b));
        f32x2 acc0 = 0ull, sum0 = 0ull, acc1 = 0ull, sum1 = 0ull;
        float max0[2] = {0.f, 0.f}, max1[2] = {0.f, 0.f};
        exact_weight_pair(x, one, make_float2(0.7f, 0.7f), acc0, sum0, max0[0], max0[1]);
        exact_weight_pair_fast(x, one, splat2(0.7f), splat2(nz), acc1, sum1, max1[0], max1[1]);
        if (acc0 != acc1 || sum0 != sum1 || max0[0] != max1[0] || max0[1] != max1[1]) atomicAdd(n, 1ull);
    }
}

// Largest relative error of fused_weight_pair's weight over the x in
// [-3.56648, -0], against the quotient in 64 bits (bits of a positive double); x
// past the cutoff, -inf and NaN must weigh 0.
__global__ void __launch_bounds__(256) fused_weight_error_kernel(unsigned long long* worst) {
    const unsigned last = __float_as_uint(-3.56648f);
    const f32x2 one = splat2(1.f);
    auto weight = [&](float x) {
        f32x2 acc = 0ull, sum = 0ull;
        float max0 = 0.f, max1 = 0.f;
        fused_weight_pair(splat2(x), one, make_float2(1.f, 1.f), acc, sum, max0, max1);
        const float2 a = unpack2(acc), s = unpack2(sum);
        return a.x == s.x && a.y == s.x && s.y == s.x && max0 == s.x && max1 == s.x ? s.x : __int_as_float(0x7fffffff);
    };
    double e = 0.0;
    for (unsigned b = 0x80000000u + blockIdx.x * 256u + threadIdx.x; b < last; b += gridDim.x * 256u) {
        const double x = (double)__uint_as_float(b);
        const double q = (120.0 + x * (60.0 + x * (12.0 + x))) / (120.0 - x * (60.0 - x * (12.0 - x)));
        const double d = fabs((double)weight(__uint_as_float(b)) - q) / q;
        if (!(d <= e)) e = d == d ? d : 1e300;
    }
    if (threadIdx.x < 4) {
        const float out[4] = {-3.56648f, -1e30f, -INFINITY, NAN};
        if (!(weight(out[threadIdx.x]) == 0.f)) e = 1e300;
    }
    if (e > 0.0) atomicMax(worst, (unsigned long long)__double_as_longlong(e));
}

}  // namespace

cudaError_t launch_fused_weight_error(double* worst, cudaStream_t st) {
    fused_weight_error_kernel<<<148 * 8, 256, 0, st>>>(reinterpret_cast<unsigned long long*>(worst));
    return cudaGetLastError();
}

cudaError_t launch_weight_mismatches(unsigned long long* n, float neg0, cudaStream_t st) {
    weight_mismatch_kernel<<<148 * 8, 256, 0, st>>>(n, neg0);
    return cudaGetLastError();
}

int pair_weight_rows(int i) { return kWeightWarps * (i ? kWeightRowsSmall : kWeightRows); }

// 8 rows per thread where that still gives every SM its warps, else 2
int pair_weight_small(long long warps, int sms) { return warps < 16ll * sms; }

cudaError_t launch_pair_weights(bool fused, const PairMaps& m, const PairArgs& a, int z0, int z1, int sms,
                                cudaStream_t st) {
    if (z1 <= z0) return cudaSuccess;
    const bool big = !pair_weight_small((long long)((a.x1 - a.x0 + 31) / 32) * ((a.y1 - a.y0 + 7) / 8) * (z1 - z0), sms);
#define X(PITCH)                                                                       \
    if (a.pbx == PITCH)                                                                 \
        return big ? launch_rows<kWeightRows, PITCH>(fused, m, a, z0, z1, st)         \
                   : launch_rows<kWeightRowsSmall, PITCH>(fused, m, a, z0, z1, st);
    X(44) X(52) X(60)
#undef X
    return cudaErrorInvalidConfiguration;
}

}  // namespace inlm
