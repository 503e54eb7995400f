// Paired-offset form of the plain FP32 iterNLM filter (sm_100a), bit-identical
// to the reference CPU filter like the tile kernel (filter_kernels.cu), and of
// the fused FP32 form, bit-identical to the fused tile kernel.
//
// The patch distance is symmetric: with D_s(x) = (prev[x+s] - prev[x])^2,
//   dist(-s, x) = sum_p w_p D_-s(x+p) = sum_p w_p D_s(x-s+p) = dist(s, x-s),
// tap for tap in the same order, and (a-b)^2 rounds as (b-a)^2, so both sides
// are the same float. The offsets come in z-major order, so offset S-1-j is
// the negative of offset j: the distances of the first half serve all S.
//
//  * nlm_pair_dist_kernel writes dist(s, x) of the first half into a
//    workspace of a ring of z planes, for every x whose value some voxel
//    needs (the block and a search halo around it);
//  * nlm_pair_weight_kernel walks all S offsets in reference order per voxel:
//    distance from the workspace (of x for the first half, of x + s for the
//    second), Pade weight, weighted sums, and the normalisation.
//
// Splitting the two also lets a small volume spread its offsets over the whole
// GPU: distances have no order among offsets, only the sums do.
#include <type_traits>

#include "common.cuh"
#include "filter_pair.cuh"
#include "geometry.hpp"
#include "pair_math.cuh"

namespace inlm {

namespace {

constexpr int kPairRows = 8;  // y voxels per thread

// Patch as columns of constant (|zp|, |xp|): extent[b][c] = largest |yp|, -1
// where the column is empty; tap[zp][yp][xp] = index in reference tap order.
struct PairPatch {
    int extent[4][4];
    int tap[7][7][7];
};

constexpr PairPatch make_pair_patch(int rx, int ry, int rz) {
    PairPatch g{};
    for (int b = 0; b < 4; b++)
        for (int c = 0; c < 4; c++) g.extent[b][c] = -1;
    for (int z = 0; z < 7; z++)
        for (int y = 0; y < 7; y++)
            for (int x = 0; x < 7; x++) g.tap[z][y][x] = -1;
    const PatchRows rows = make_patch_rows(rx, ry, rz);
    int t = 1;
    g.tap[3][3][3] = 0;
    for (int r = 0; r < rows.n; r++)
        for (int xp = -rows.e[r]; xp <= rows.e[r]; xp++) {
            const int zp = rows.zp[r], yp = rows.yp[r];
            const int b = zp < 0 ? -zp : zp, a = yp < 0 ? -yp : yp, c = xp < 0 ? -xp : xp;
            if (g.extent[b][c] < a) g.extent[b][c] = a;
            if (zp == 0 && yp == 0 && xp == 0) continue;
            g.tap[zp + 3][yp + 3][xp + 3] = t++;
        }
    return g;
}

// Every tap lies in its column's extent and every extent is full.
constexpr bool pair_patch_full(const PairPatch& g) {
    for (int z = -3; z <= 3; z++)
        for (int y = -3; y <= 3; y++)
            for (int x = -3; x <= 3; x++) {
                const int b = z < 0 ? -z : z, a = y < 0 ? -y : y, c = x < 0 ? -x : x;
                if ((g.tap[z + 3][y + 3][x + 3] >= 0) != (g.extent[b][c] >= a)) return false;
            }
    return true;
}

// Patch radius 2 stages its D planes (below); radius 1 and 3 form their columns
// directly.
constexpr bool pair_staged(int rx) { return rx == 2; }
constexpr int kStageRows = 12;  // staged y rows: -2 ... 9

template <int RX, int RY, int RZ>
struct PairGeom {
    static constexpr PairPatch g = make_pair_patch(RX, RY, RZ);
    static_assert(pair_patch_full(make_pair_patch(RX, RY, RZ)), "patch columns");
    // D column of shift xp as pairs of y values: rows [-lead, ...), the extent
    // of its taps, or all staged rows
    static constexpr int e0(int c) { return g.extent[0][c]; }
    static constexpr int lead(int c) { return pair_staged(RX) ? 2 : e0(c); }
    static constexpr int pairs(int c) { return pair_staged(RX) ? kStageRows / 2 : kPairRows / 2 + e0(c); }
    static constexpr int first(int xp) {  // first pair of column xp in the D array
        int n = 0;
        for (int x = -RX; x < xp; x++) n += pairs(x < 0 ? -x : x);
        return n;
    }
    static constexpr int NV2 = first(RX + 1);  // pairs per plane
    // largest |zp| of the taps in column xp
    static constexpr int bmax(int c) {
        int b = 0;
        while (b < RZ && g.extent[b + 1][c] >= 0) b++;
        return b;
    }
    static constexpr bool member(int b, int a, int c) { return g.extent[b][c] >= a; }
    static constexpr int weight(int b, int a, int c) { return g.tap[3 + b][3 + a][3 + c]; }
    static constexpr int ymax(int b) {  // largest |yp| among the taps of |zp| = b
        int m = -1;
        for (int c = 0; c <= RX; c++) m = g.extent[b][c] > m ? g.extent[b][c] : m;
        return m;
    }
};

// Shared memory of the distance kernel: barrier and work counter, per warp the
// finished plane on its way out and the staged D planes, then the prev box.
template <int RX, int RZ>
struct PairSmem {
    static constexpr int kWarps = RX <= 2 ? 16 : 12;
    static constexpr int kOut = kPairRows * 32 * 4;
    static constexpr int kPlane = (32 + 2 * RX) * kStageRows;  // floats per staged D plane
    static constexpr int kWarp = kOut + (pair_staged(RX) ? ((RZ + 1) * kPlane * 4 + 127) / 128 * 128 : 0);
    static constexpr size_t kBox = 128 + (size_t)kWarps * kWarp;
};

template <int I0, int I1, class F>
__device__ __forceinline__ void static_for(F&& f) {
    if constexpr (I0 < I1) {
        f(std::integral_constant<int, I0>{});
        static_for<I0 + 1, I1>(f);
    }
}

template <int N>
__device__ __forceinline__ float element(const f32x2 (&v)[N], int i) {
    const float2 p = unpack2(v[i >> 1]);
    return (i & 1) ? p.y : p.x;
}

// Adds the taps of |zp| = B on the D columns of one plane to the distances of
// plane q - B (its taps zp = +B, LO) and q + B (zp = -B, HI), in the
// reference's (yp, xp) order. A product w * D serves both planes and, mirrored
// in y, the taps +yp and -yp of different voxels: each is formed once (plain
// form). The fused form adds by fused multiply-adds and shares nothing.
template <int RX, int RY, int RZ, int B, bool LO, bool HI, bool FUSED>
__device__ __forceinline__ void plane_taps(const f32x2 (&D)[PairGeom<RX, RY, RZ>::NV2],
                                           f32x2 (&lo)[kPairRows / 2], f32x2 (&hi)[kPairRows / 2], f32x2 neg0,
                                           const PairArgs& a) {
    using G = PairGeom<RX, RY, RZ>;
    constexpr int YM = G::ymax(B);
    constexpr int NP = kPairRows / 2;
    f32x2 P[RY + 1][2 * RX + 1][NP + RY];
    static_for<0, NP>([&](auto pc) {
        constexpr int p = pc;
        static_for<-YM, YM + 1>([&](auto yc) {
            constexpr int yp = yc;
            constexpr int A = yp < 0 ? -yp : yp;
            static_for<-RX, RX + 1>([&](auto xc) {
                constexpr int xp = xc;
                constexpr int C = xp < 0 ? -xp : xp;
                if constexpr (G::member(B, A, C) && !(B == 0 && A == 0 && C == 0)) {
                    constexpr int j = yp > 0 ? p + A : p;  // pair of D rows (2j - A, 2j - A + 1)
                    constexpr int i = 2 * j - A + G::lead(C);  // its first value in the column
                    constexpr int f = 2 * G::first(xp);
                    const float w = a.w[G::weight(B, A, C)];
                    const float v0 = element(D, f + i), v1 = element(D, f + i + 1);
                    if constexpr (FUSED) {
                        const f32x2 v = pack2(v0, v1), ww = splat2(w);
                        if constexpr (LO) lo[p] = fma2(v, ww, lo[p]);
                        if constexpr (HI) hi[p] = fma2(v, ww, hi[p]);
                    } else {
                        // first use: the upper tap of any pair, or the lower
                        // tap of the first A pairs
                        if constexpr (yp >= 0 || p < A)
                            P[A][xp + RX][j] = (i & 1) ? mul_pair(v0, v1, w)
                                                       : mul2_to_add(D[(f + i) / 2], splat2(w), neg0);
                        if constexpr (LO) lo[p] = add2(lo[p], P[A][xp + RX][j]);
                        if constexpr (HI) hi[p] = add2(hi[p], P[A][xp + RX][j]);
                    }
                }
            });
        });
    });
}

// Taps of D plane q on the distances of the planes around it; planes outside
// [z0, z1) are not formed.
template <int RX, int RY, int RZ, bool FUSED>
__device__ __forceinline__ void all_taps(const f32x2 (&D)[PairGeom<RX, RY, RZ>::NV2],
                                         f32x2 (&acc)[2 * RZ + 1][kPairRows / 2], int q, int z0, int z1, f32x2 neg0,
                                         const PairArgs& a) {
    static_for<0, RZ + 1>([&](auto bc) {
        constexpr int B = bc;
        const bool l = q - B >= z0 && q - B < z1, u = q + B >= z0 && q + B < z1;
        if constexpr (B == 0) {
            if (l) plane_taps<RX, RY, RZ, 0, true, false, FUSED>(D, acc[RZ], acc[RZ], neg0, a);
        } else {
            if (l && u)
                plane_taps<RX, RY, RZ, B, true, true, FUSED>(D, acc[RZ - B], acc[RZ + B], neg0, a);
            else if (l)
                plane_taps<RX, RY, RZ, B, true, false, FUSED>(D, acc[RZ - B], acc[RZ + B], neg0, a);
            else if (u)
                plane_taps<RX, RY, RZ, B, false, true, FUSED>(D, acc[RZ - B], acc[RZ + B], neg0, a);
        }
    });
}

// Squared differences of rows y, y + 1 of one column (c0: unshifted, c1: shifted).
template <int PBX>
__device__ __forceinline__ f32x2 square_pair(const float* c0, const float* c1, int y) {
    const f32x2 v = sub2(pack2(c1[y * PBX], c1[(y + 1) * PBX]), pack2(c0[y * PBX], c0[(y + 1) * PBX]));
    return mul2_to_mul(v, v);  // feeds only products
}

// What bounds it: FP32 lanes, shared-memory reads and issue slots together (64 %,
// 81 % and 70 % busy at patch radius 2; about 54 lane operations per distance
// for 33 taps, against 66 without the sharing). At 256 x 256 x 96, search radius
// 5, it takes 4.94 ms and the weight kernel 2.76 ms; the warp-specialised
// kernel, which sums the patches of all offsets, takes 13.4 ms. Forming the
// columns of patch radius 2 directly took 5.61 ms; at patch radius 1 staging
// moves more through shared memory than it saves (9.9 against 6.7 ms for
// 192 x 192 x 64, search radius 10), and at radius 3 the staged planes would
// leave no room for the box.
//
// A warp takes offsets of the CTA's tile (32 x 8 x tz voxels, prev box staged by
// one TMA load); a thread owns one x column of 8 y voxels and walks the z
// planes with the 2 RZ + 1 planes of distances that a D plane touches in
// registers: a D plane is formed once, and its products serve every plane and
// mirrored tap they belong to. Finished planes leave by TMA.
//
// Patch radius 2 (staged): the warp forms each D plane once over its 32
// columns and the patch halo, into a ring of RZ + 1 planes of its own in shared
// memory, column-major so that a thread reads a neighbour column's 12 rows as
// three 16-byte words (the 48-byte column pitch spreads 8 lanes over all
// banks). The tap w_0 D that opens the sum of plane q + RZ is taken from the
// thread's own column while it is staged.
template <int RX, int RY, int RZ, int PBX, bool FUSED>
__global__ void __launch_bounds__(32 * PairSmem<RX, RZ>::kWarps, 1)
    nlm_pair_dist_kernel(const __grid_constant__ CUtensorMap tm_prev, const __grid_constant__ CUtensorMap tm_out,
                         const __grid_constant__ PairArgs a, int z_first) {
    using G = PairGeom<RX, RY, RZ>;
    using M = PairSmem<RX, RZ>;
    constexpr int NP = kPairRows / 2;
    constexpr int LIVE = 2 * RZ + 1;
    constexpr bool STAGED = pair_staged(RX);
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
    int* next = reinterpret_cast<int*>(smem + 64);
    float* prevb = reinterpret_cast<float*>(smem + M::kBox);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int t = blockIdx.x;
    const int split = t % a.splits;
    t /= a.splits;
    const int X0 = a.xs + (t % a.tiles_x) * 32;
    t /= a.tiles_x;
    const int Y0 = a.ys + (t % a.tiles_y) * kPairRows;
    const int Z0 = z_first + (t / a.tiles_y) * a.tz;
    if (tid == 0) {
        prefetch_tmap(&tm_prev);
        prefetch_tmap(&tm_out);
        mbar_init(bar, 1);
        fence_mbar_init();
        *next = split;
    }
    __syncthreads();
    if (tid == 0) {
        mbar_arrive_expect_tx(bar, (uint32_t)(PBX * a.pby * a.pbz) * 4u);
        // voxel (X0 - px, Y0 - py, Z0 - szc - RZ) in padded coordinates
        tma_load_3d(prevb, &tm_prev, X0, Y0, Z0, bar);
    }
    const bool arrived = mbar_wait_bounded(bar, 0);
    if (!__syncthreads_and(arrived)) {
        if (tid == 0) {
            set_error(a.err, DEV_TMA_TIMEOUT);
            mbar_wait_bounded(bar, 0);  // let the copy land before the CTA's memory goes away
        }
        return;
    }
    const int pplane = PBX * a.pby;
    const f32x2 neg0 = splat2(a.neg0);
    const f32x2 w0 = splat2(a.w[0]);
    const int tz = min(a.tz, a.nz + a.szc - Z0);  // planes of this tile that are ever read
    const bool own = X0 < a.x1 && X0 + 32 > a.x0 && Y0 < a.y1 && Y0 + kPairRows > a.y0 && Z0 < a.nz;
    float* out = reinterpret_cast<float*>(smem + 128 + warp * M::kWarp);
    float* stage = out + M::kOut / 4;
    // voxel (lane, row 0) on plane 0 of the tile
    const float* org0 = prevb + (a.szc + RZ) * pplane + a.py * PBX + a.px + lane;
    // halo columns of a staged plane: lane -> (column, pair of rows)
    constexpr int NH = 2 * RX * (kStageRows / 2);
    const int hc = lane / (kStageRows / 2), hp = lane % (kStageRows / 2);
    const int hx = hc < RX ? hc - RX : 32 + hc - RX;

    // whole offsets first; the last ones, fewer than the warps of the CTAs that
    // share the tile, are cut in z so that every warp has a part
    const int lanes = M::kWarps * a.splits;
    const int rest = a.H % lanes;
    const int parts = rest ? max(1, min(lanes / rest, tz / (2 * RZ + 2))) : 1;
    const int whole = a.H - rest, items = whole + rest * parts;
    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(next, a.splits);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= items) break;
        int h = item, z0 = 0, z1 = tz;
        if (item >= whole) {
            const int j = item - whole;
            h = whole + j / parts;
            z0 = (j % parts) * tz / parts;
            z1 = (j % parts + 1) * tz / parts;
        }
        const PairOffset o = a.offsets[h];
        // a tile outside the block serves only the offsets that lead into it
        if (!own && !(X0 + o.x < a.x1 && X0 + 32 + o.x > a.x0 && Y0 + o.y < a.y1 && Y0 + kPairRows + o.y > a.y0 &&
                      Z0 + o.z < a.nz))
            continue;
        f32x2 acc[LIVE][NP];
#pragma unroll
        for (int i = 0; i < LIVE; i++)
#pragma unroll
            for (int p = 0; p < NP; p++) acc[i][p] = 0ull;
        int zr = (Z0 + z0) % a.ring;
        // the finished plane q - RZ: its rows to shared memory, then out
        auto put = [&]() {
#pragma unroll
            for (int p = 0; p < NP; p++) {
                const float2 d = unpack2(acc[0][p]);
                out[2 * p * 32 + lane] = d.x;
                out[(2 * p + 1) * 32 + lane] = d.y;
            }
            fence_proxy_async_smem();
        };
        auto send = [&]() {
            if (lane == 0) tma_store_4d(&tm_out, out, X0 - a.xs, Y0 - a.ys, zr, h);
            if (++zr == a.ring) zr = 0;
        };
        auto shift = [&]() {
#pragma unroll
            for (int i = 0; i + 1 < LIVE; i++)
#pragma unroll
                for (int p = 0; p < NP; p++) acc[i][p] = acc[i + 1][p];
        };
        if constexpr (STAGED) {
            const float* c0 = org0 + (z0 - RZ) * pplane;
            const float* h0 = c0 - lane + hx + (2 * hp - 2) * PBX;
            int wslot = 0, rslot = 0;  // staged plane written and read next
#pragma unroll 1
            for (int k = z0 - RZ; k < z1 + 2 * RZ; k++) {
                if (k < z1 + RZ) {  // stage plane k
                    float* col = stage + wslot * M::kPlane;
                    const float* c1 = c0 + o.prev;
                    f32x2 v[kStageRows / 2];
#pragma unroll
                    for (int i = 0; i < kStageRows / 2; i++) v[i] = square_pair<PBX>(c0, c1, 2 * i - 2);
                    ulonglong2* dst = reinterpret_cast<ulonglong2*>(col + (lane + RX) * kStageRows);
#pragma unroll
                    for (int i = 0; i < kStageRows / 4; i++) dst[i] = make_ulonglong2(v[2 * i], v[2 * i + 1]);
                    if (lane < NH)
                        *reinterpret_cast<f32x2*>(col + (hx + RX) * kStageRows + 2 * hp) =
                            square_pair<PBX>(h0, h0 + o.prev, 0);
                    // the centre tap opens the sum of plane k
#pragma unroll
                    for (int p = 0; p < NP; p++) acc[LIVE - 1][p] = mul2_to_add(v[p + 1], w0, neg0);
                    c0 += pplane;
                    h0 += pplane;
                    if (++wslot == RZ + 1) wslot = 0;
                }
                if (lane == 0) tma_store_wait_read();  // `out` may be written again
                __syncwarp();
                const int q = k - RZ;
                if (q >= z0 - RZ) {
                    f32x2 D[G::NV2];
                    const float* col = stage + rslot * M::kPlane + lane * kStageRows;
                    static_for<-RX, RX + 1>([&](auto xc) {
                        constexpr int xp = xc;
                        const ulonglong2* src = reinterpret_cast<const ulonglong2*>(col + (xp + RX) * kStageRows);
#pragma unroll
                        for (int i = 0; i < kStageRows / 4; i++) {
                            const ulonglong2 u = src[i];
                            D[G::first(xp) + 2 * i] = u.x;
                            D[G::first(xp) + 2 * i + 1] = u.y;
                        }
                    });
                    all_taps<RX, RY, RZ, FUSED>(D, acc, q, z0, z1, neg0, a);
                    if (q - RZ >= z0) put();
                    if (++rslot == RZ + 1) rslot = 0;
                }
                __syncwarp();
                if (q - RZ >= z0) send();
                shift();
            }
        } else {
            const float* org = org0 + (z0 - RZ) * pplane;
            // the own column of the next plane, whose centre tap opens its sum
            constexpr bool CARRY = RZ == 1;
            f32x2 ahead[CARRY ? G::pairs(0) : 1];
            if constexpr (CARRY) {
#pragma unroll
                for (int i = 0; i < G::pairs(0); i++) ahead[i] = square_pair<PBX>(org, org + o.prev, 2 * i - G::lead(0));
            }
#pragma unroll 1
            for (int q = z0 - RZ; q < z1 + RZ; q++) {
                // D columns of plane q; the planes outside the range need only
                // the columns that reach into it
                const int bmin = q < z0 ? z0 - q : q >= z1 ? q - z1 + 1 : 0;
                f32x2 D[G::NV2];
                static_for<-RX, RX + 1>([&](auto xc) {
                    constexpr int xp = xc;
                    constexpr int C = xp < 0 ? -xp : xp;
                    if constexpr (CARRY && xp == 0) {
#pragma unroll
                        for (int i = 0; i < G::pairs(0); i++) D[G::first(0) + i] = ahead[i];
                    } else if (G::bmax(C) >= RZ || bmin <= G::bmax(C)) {
                        const float* c0 = org + xp;
#pragma unroll
                        for (int i = 0; i < G::pairs(C); i++)
                            D[G::first(xp) + i] = square_pair<PBX>(c0, c0 + o.prev, 2 * i - G::lead(C));
                    }
                });
                // the centre tap opens the sum of plane q + RZ
                if constexpr (CARRY) {
                    if (q + 1 < z1 + RZ) {
                        const float* c0 = org + pplane;
#pragma unroll
                        for (int i = 0; i < G::pairs(0); i++)
                            ahead[i] = square_pair<PBX>(c0, c0 + o.prev, 2 * i - G::lead(0));
                    }
#pragma unroll
                    for (int p = 0; p < NP; p++) {
                        if constexpr (G::lead(0) % 2 == 0) {
                            acc[LIVE - 1][p] = mul2_to_add(ahead[p + G::lead(0) / 2], w0, neg0);
                        } else {
                            const float2 u = unpack2(ahead[p + G::lead(0) / 2]), v = unpack2(ahead[p + G::lead(0) / 2 + 1]);
                            acc[LIVE - 1][p] = mul_pair(u.y, v.x, a.w[0]);
                        }
                    }
                } else if (q + RZ < z1) {
                    const float* c0 = org + RZ * pplane;
#pragma unroll
                    for (int p = 0; p < NP; p++)
                        acc[LIVE - 1][p] = mul2_to_add(square_pair<PBX>(c0, c0 + o.prev, 2 * p), w0, neg0);
                }
                all_taps<RX, RY, RZ, FUSED>(D, acc, q, z0, z1, neg0, a);
                if (q - RZ >= z0) {
                    if (lane == 0) tma_store_wait_read();
                    __syncwarp();
                    put();
                    __syncwarp();
                    send();
                }
                shift();
                org += pplane;
            }
        }
    }
    if (lane == 0) tma_store_wait();
}

template <int RX, int RY, int RZ, int PBX>
cudaError_t launch_dist_pitch(bool fused, const PairMaps& m, const PairArgs& a, int z0, cudaStream_t st) {
    const size_t smem = pair_smem_bytes(RX, RZ, a);
    auto kern = fused ? nlm_pair_dist_kernel<RX, RY, RZ, PBX, true> : nlm_pair_dist_kernel<RX, RY, RZ, PBX, false>;
    cudaError_t e = allow_shared_memory(kern, smem);
    if (e != cudaSuccess) return e;
    kern<<<a.tiles_x * a.tiles_y * a.tiles_z * a.splits, 32 * PairSmem<RX, RZ>::kWarps, smem, st>>>(m.prev, m.out, a, z0);
    return cudaGetLastError();
}

template <int RX, int RY, int RZ>
cudaError_t launch_dist_shape(bool fused, const PairMaps& m, const PairArgs& a, int z0, cudaStream_t st) {
    switch (a.pbx) {
        case 44: return launch_dist_pitch<RX, RY, RZ, 44>(fused, m, a, z0, st);
        case 52: return launch_dist_pitch<RX, RY, RZ, 52>(fused, m, a, z0, st);
        case 60: return launch_dist_pitch<RX, RY, RZ, 60>(fused, m, a, z0, st);
        default: return cudaErrorInvalidConfiguration;
    }
}

template <int RX, int RY, int RZ>
bool symmetric_shape(const float* w) {
    constexpr PairPatch g = make_pair_patch(RX, RY, RZ);
    for (int z = -RZ; z <= RZ; z++)
        for (int y = -RY; y <= RY; y++)
            for (int x = -RX; x <= RX; x++) {
                const int t = g.tap[z + 3][y + 3][x + 3];
                const int m = g.tap[(z < 0 ? -z : z) + 3][(y < 0 ? -y : y) + 3][(x < 0 ? -x : x) + 3];
                if ((t < 0) != (m < 0)) return false;
                if (t >= 0 && !(w[t] == w[m])) return false;
            }
    return true;
}

}  // namespace

#define INLM_PAIR_SHAPES(X) \
    X(1, 1, 1) X(1, 1, 2) X(1, 1, 3) X(2, 2, 1) X(2, 2, 2) X(3, 3, 1) X(3, 3, 2) X(3, 3, 3)

bool pair_kernel_available(int rx, int ry, int rz) {
#define X(A, B, C) \
    if (rx == A && ry == B && rz == C) return true;
    INLM_PAIR_SHAPES(X)
#undef X
    return false;
}

bool pair_weights_symmetric(int rx, int ry, int rz, const float* w) {
#define X(A, B, C) \
    if (rx == A && ry == B && rz == C) return symmetric_shape<A, B, C>(w);
    INLM_PAIR_SHAPES(X)
#undef X
    return false;
}

int pair_kernel_warps(int rx) { return rx <= 2 ? PairSmem<1, 1>::kWarps : PairSmem<3, 1>::kWarps; }

// Pitches of 4 (mod 8) floats: eight rows of a column lie in different banks.
int pair_box_pitch(int px) {
    const int w = 32 + 2 * px;
    return w <= 44 ? 44 : w <= 52 ? 52 : w <= 60 ? 60 : 0;
}

size_t pair_smem_bytes(int rx, int rz, const PairArgs& a) {
    size_t head = 0;
    if (rx == 1) head = rz == 1 ? PairSmem<1, 1>::kBox : rz == 2 ? PairSmem<1, 2>::kBox : PairSmem<1, 3>::kBox;
    if (rx == 2) head = rz == 1 ? PairSmem<2, 1>::kBox : PairSmem<2, 2>::kBox;
    if (rx == 3) head = PairSmem<3, 1>::kBox;
    return head + (size_t)a.pbx * a.pby * a.pbz * 4;
}

cudaError_t launch_pair_dist(int rx, int ry, int rz, bool fused, const PairMaps& m, const PairArgs& a, int z0,
                             cudaStream_t st) {
#define X(A, B, C) \
    if (rx == A && ry == B && rz == C) return launch_dist_shape<A, B, C>(fused, m, a, z0, st);
    INLM_PAIR_SHAPES(X)
#undef X
    return cudaErrorInvalidConfiguration;
}

}  // namespace inlm
