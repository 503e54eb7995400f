// Host side of the paired-offset FP32 form (filter_pair.cu): when it applies,
// the workspace and how a volume is cut into blocks and z chunks that fit it.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <mutex>

#include "api_internal.hpp"
#include "common.cuh"

using namespace inlm;

namespace {

// A workspace takes at most an eighth of the device's memory, and half of what
// is free when a handle plans its passes. A deeper z chunk means fewer launches
// with a partly filled last wave: 256^3, patch radius 1, search radius 10 takes
// 95 ms with an eighth and 101 ms with a sixteenth.
constexpr int kWorkspaceShare = 8;

// Workspaces are not the handles': a call borrows one and hands it back when
// its work on the GPU has ended, so handles that take turns share one buffer.
// Per device the pool holds as many as calls in flight need, up to the share
// above in total; from then on a call joins a buffer that is out, and the passes
// on it run one after another (each fills the GPU). Nothing is allocated or freed
// between the passes of such calls. None is left once the last handle that
// borrowed is gone.
struct Pool {
    std::vector<PairBuf*> bufs;
    int users = 0;
    size_t share = 0;  // bytes kept in total
};
constexpr int kMaxDevices = 64;
Pool g_pool[kMaxDevices];
std::recursive_mutex g_pool_mutex;  // device_malloc may call pair_trim under it
std::atomic<long long> g_pool_bound{0};  // a test's bound in place of the share

// (a batch's own does not count: it would leave the calls beside it nothing)
size_t pool_bytes(const Pool& pool) {
    size_t n = 0;
    for (const PairBuf* b : pool.bufs)
        if (!b->alone) n += b->bytes;
    return n;
}

size_t pool_share(const Pool& pool) {
    const long long bound = g_pool_bound.load();
    return bound > 0 ? (size_t)bound : pool.share;
}

// Frees the smallest idle buffer; false if there is none.
bool free_idle(Pool& pool) {
    PairBuf* least = nullptr;
    for (PairBuf* b : pool.bufs)
        if (b->users == 0 && (!least || b->bytes < least->bytes)) least = b;
    if (!least) return false;
    pool.bufs.erase(std::find(pool.bufs.begin(), pool.bufs.end(), least));
    device_free(least->p);
    cudaEventDestroy(least->done);
    delete least;
    return true;
}

PairBuf* borrow(int device, size_t bytes, bool alone) {
    std::lock_guard<std::recursive_mutex> lock(g_pool_mutex);
    Pool& pool = g_pool[device];
    if (pool.share == 0) {
        size_t free_b = 0, total_b = 0;
        if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return nullptr;
        pool.share = total_b / kWorkspaceShare;
    }
    PairBuf *idle = nullptr, *out = nullptr;
    for (PairBuf* b : pool.bufs) {
        if (b->bytes < bytes) continue;
        if (b->users == 0 && (!idle || b->bytes < idle->bytes)) idle = b;
        if (b->users > 0 && !b->alone && !alone && (!out || b->users < out->users)) out = b;
    }
    if (!idle) {
        while (pool_bytes(pool) + bytes > pool_share(pool) && free_idle(pool)) {
        }
        if (pool_bytes(pool) + bytes <= pool_share(pool) || !out) {
            PairBuf* b = new PairBuf();
            b->device = device;
            b->bytes = bytes;
            if (device_malloc(&b->p, bytes) == cudaSuccess &&
                cudaEventCreateWithFlags(&b->done, cudaEventDisableTiming) == cudaSuccess) {
                pool.bufs.push_back(b);
                idle = b;
            } else {
                cudaGetLastError();
                device_free(b->p);
                delete b;
            }
        }
    }
    PairBuf* b = idle ? idle : out;
    if (!b) return nullptr;
    b->alone = alone;
    b->users++;
    return b;
}

void hand_back(PairBuf* b) {
    std::lock_guard<std::recursive_mutex> lock(g_pool_mutex);
    Pool& pool = g_pool[b->device];
    if (--b->users > 0) return;
    b->last = nullptr;
    b->alone = false;
    while ((pool.users == 0 || pool_bytes(pool) > pool_share(pool)) && free_idle(pool)) {
    }
}

void count_user(int device, int change) {
    std::lock_guard<std::recursive_mutex> lock(g_pool_mutex);
    Pool& pool = g_pool[device];
    pool.users += change;
    while (pool.users == 0 && free_idle(pool)) {
    }
}

size_t idle_bytes(int device) {
    std::lock_guard<std::recursive_mutex> lock(g_pool_mutex);
    size_t n = 0;
    for (const PairBuf* b : g_pool[device].bufs)
        if (b->users == 0) n += b->bytes;
    return n;
}

int round_up(int v, int m) { return (v + m - 1) / m * m; }

// CTAs that share one tile's offsets: as many as leave the least of the last
// wave empty (one CTA runs per SM), each costing another load of the tile's
// box (about a fiftieth of a tile's work), and at most one per round of warps.
int offset_splits(int tiles, int sms, int most) {
    int best = 1;
    double best_cost = 0;
    for (int n = 1; n <= std::max(1, std::min(most, 64)); n++) {
        const double cost = (double)((tiles * (long long)n + sms - 1) / sms) / n * (1.0 + 0.02 * n);
        if (n == 1 || cost < best_cost) {
            best = n;
            best_cost = cost;
        }
    }
    return best;
}

// Plane steps of the longest-working warp of a launch (the kernel's split of
// whole offsets and of the rest among its warps).
double warp_steps(int tiles, int splits, int sms, int warps, int H, int tz, int rz) {
    const int lanes = warps * splits, rest = H % lanes;
    const int parts = rest ? std::max(1, std::min(lanes / rest, tz / (2 * rz + 2))) : 1;
    const double rounds = (double)(H / lanes) * (tz + 2 * rz) + (rest ? (double)tz / parts + 2 * rz : 0.0);
    return rounds * ((tiles * (long long)splits + sms - 1) / sms);
}

// A volume cut into blocks (whole rows and columns where they fit) and each block
// into z chunks, so that one chunk's distances and the search halo fit a
// workspace.
struct Plan {
    int bx = 0, by = 0;          // voxels per block in x and y
    int chunk = 0;               // planes per pair of launches
    int tz = 0;                  // planes per tile
    int tiles_x = 0, tiles_y = 0;
    int ring = 0;                // workspace planes per offset
    double cost = 0;             // 0: not even the smallest block fits
    size_t bytes(int H) const { return (size_t)H * ring * tiles_x * 32 * tiles_y * 8 * 4; }
};

// The cheapest plan for a workspace of `budget` bytes; a.tz is the deepest tile.
Plan plan_blocks(const PairArgs& a, const int* pr, int sms, int warps, size_t budget) {
    Plan best;
    const int depth = a.nz + a.szc;  // planes whose distances are read
    const int tz_most = a.tz, rz = pr[2];
    // weight kernel's time over distance kernel's (measured: 1.2, 0.6, 0.25)
    const double weights_share = pr[0] == 1 ? 1.2 : pr[0] == 2 ? 0.6 : 0.25;
    for (int nby = 1; nby <= 32; nby++)
        for (int nbx = 1; nbx <= 32; nbx++) {
            const int bx = round_up((a.nx + nbx - 1) / nbx, 32), by = round_up((a.ny + nby - 1) / nby, 8);
            if ((nbx > 1 && bx * (nbx - 1) >= a.nx) || (nby > 1 && by * (nby - 1) >= a.ny)) continue;
            const int tiles_x = (round_up(a.sxr, 8) + std::min(bx, a.nx) + a.sxr + 31) / 32;
            const int tiles_y = (2 * a.syr + std::min(by, a.ny) + 7) / 8;
            const size_t plane = (size_t)tiles_x * 32 * tiles_y * 8 * a.H * 4;
            const int ring_max = (int)std::min<size_t>(budget / plane, 1 << 20);
            // the whole volume where it fits, else chunks of k layers of tiles
            // of any depth down to half the deepest
            const bool whole = depth <= ring_max;
            for (int k = 1; k <= (whole ? 1 : 64) && (whole || (k - 1) * std::max(4, tz_most / 2) < depth); k++)
                for (int tz = tz_most; tz >= (whole ? tz_most : std::max(4, tz_most / 2)); tz--) {
                    const int chunk = whole ? depth : std::min(depth, k * tz), ring = whole ? depth : chunk + a.szc;
                    if (ring > ring_max) continue;
                    const int n_chunks = (depth + chunk - 1) / chunk;
                    // distances: tiles of all launches (a tile of tz planes
                    // walks tz + 2 RZ), and a third of a wave of tiles lost per
                    // launch; weights: whole waves of CTAs (four per SM), at the
                    // share of the time that they take
                    const double layers = (double)((chunk + tz - 1) / tz) * n_chunks;
                    const double walk = (double)tiles_x * tiles_y * layers / sms * (tz + 2 * rz) +
                                        0.3 * n_chunks * (tz_most + 2 * rz);
                    const double ctas = (double)((std::min(bx, a.nx) + 31) / 32) * ((std::min(by, a.ny) + 31) / 32) *
                                        std::min(chunk, a.nz) / (4.0 * sms);
                    const double cost = walk * (1.0 + weights_share * std::ceil(ctas) / ctas) * nbx * nby;
                    if (best.cost == 0 || cost < best.cost) best = Plan{bx, by, chunk, tz, tiles_x, tiles_y, ring, cost};
                }
        }
    // a volume that leaves SMs idle even with its offsets shared out: shallower
    // tiles, whose walks are shorter
    const int most = (a.H + warps - 1) / warps;
    if (best.cost > 0 && best.chunk == depth &&
        best.tiles_x * best.tiles_y * ((depth + best.tz - 1) / best.tz) * most < sms) {
        double least = 0;
        for (int tz = tz_most; tz >= 4; tz--) {
            const int tiles = best.tiles_x * best.tiles_y * ((depth + tz - 1) / tz);
            const double steps = warp_steps(tiles, offset_splits(tiles, sms, most), sms, warps, a.H, tz, rz);
            if (least == 0 || steps < least) {
                least = steps;
                best.tz = tz;
            }
        }
    }
    return best;
}

// A plan's time in units of a plane step of a tile on one SM. Unlike the cost that
// plans are chosen by, it counts the weight kernel's CTAs in the rows per thread
// that a chunk gets: within 15 % of the measured ratio up to half again the time of
// the whole volume in one chunk, above it beyond.
double plan_time(const PairArgs& a, const int* pr, int sms, const Plan& p) {
    const int depth = a.nz + a.szc, rz = pr[2], wx = std::min(p.bx, a.nx), wy = std::min(p.by, a.ny);
    const double weights_share = pr[0] == 1 ? 1.2 : pr[0] == 2 ? 0.6 : 0.25;
    const int blocks = (a.nx + p.bx - 1) / p.bx * ((a.ny + p.by - 1) / p.by), n_chunks = (depth + p.chunk - 1) / p.chunk;
    const double layers = (double)((p.chunk + p.tz - 1) / p.tz) * n_chunks;
    const double dist = (double)p.tiles_x * p.tiles_y * layers / sms * (p.tz + 2 * rz) + 0.3 * n_chunks * (a.tz + 2 * rz);
    const int columns = (wx + 31) / 32, planes = std::min(p.chunk, a.nz);
    const int rows = pair_weight_rows(pair_weight_small((long long)columns * ((wy + 7) / 8) * planes, sms));
    const double ctas = (double)columns * ((wy + rows - 1) / rows) * planes / (4.0 * sms);
    const double weights = weights_share * columns * ((wy + 7) / 8) * a.nz / sms * std::ceil(ctas) / ctas;
    return (dist + weights) * blocks;
}

// Whether a plan is worth running. With few offsets the two launches and the
// distances' way through memory cost more than the pairs save: single-pass over
// paired time at patch radius 1, 2 offsets 0.60 to 0.68, 6 offsets 0.83 to 0.88, 8
// offsets 0.93 to 1.08, 14 to 18 offsets 0.96 to 1.45, from 28 on at least 1.17; at
// patch radius 2 and 3, 2 offsets 0.67 to 1.11, 4 offsets 0.89 to 1.43, from 6 on
// 1.09 to 1.6; fused, 8 offsets 0.81 and 0.97 on 24 x 64 x 64 (five volumes of 23
// thousand to 16.8 million voxels). And with little workspace: the single-pass kernels take kSingle times as
// long as the whole volume in one chunk, so a plan that is cut up further is slower
// than they are. Measured at 256^3 as workspace: paired (single-pass), ms. Patch
// radius 1, search radius 10, 22 GB: 92.9, 16: 96.8, 8: 113.7, 4: 130.9, 2: 149, 1:
// 296 (102.6); search radius 5, 22 GB: 13.9, 2: 16.1, 1: 20.0 (17.1). Patch radius
// 2, search radius 5, 22 GB: 19.7, 1: 27.3, 0.5: 30.8, 0.25: 42.5 (36.1). Patch
// radius 3, search radius 7, 22 GB: 112, 2: 138, 1: 167, 0.5: 221, 0.25: 396 (262).
// Where the column form does not fit (patch radius 1, search radius 13: 174 against
// 389 ms) the tile kernels set the line.
bool plan_pays(const PairArgs& a, const int* pr, bool fused, bool column, int sms, int warps, const Plan& p) {
    if (a.S < (pr[0] == 1 ? 14 : fused ? 10 : 6)) return false;
    const double kSingle = column ? 1.18 : pr[0] <= 2 ? 1.85 : 2.3;
    return p.cost > 0 && plan_time(a, pr, sms, p) <= kSingle * plan_time(a, pr, sms, plan_blocks(a, pr, sms, warps, SIZE_MAX));
}

// Extents of the form's kernels for a volume: false where they do not cover it.
// a->tz is the deepest tile whose box fits beside the warps' buffers.
bool pair_extents(const Geometry& g, const int shape[3], int nslices, size_t smem_max, PairArgs* a) {
    const int* pr = g.patch_radius;
    *a = PairArgs{};
    a->nx = shape[0];
    a->ny = shape[1];
    a->nz = shape[2];
    a->px = g.pad[0];
    a->py = g.pad[1];
    a->pz = g.pad[2];
    a->sxr = g.search_radius[0];
    a->syr = g.search_radius[1];
    a->szc = std::min(nslices / 2, g.search_radius[2]);
    a->S = (int)g.search.size();
    a->H = a->S / 2;
    a->pbx = pair_box_pitch(a->px);
    if (a->pbx == 0) return false;
    a->pby = 8 + 2 * a->py;
    for (int tz = 24; tz >= 4 && a->tz == 0; tz--) {
        a->pbz = tz + 2 * pr[2] + a->szc;
        if (pair_smem_bytes(pr[0], pr[2], *a) <= smem_max) a->tz = tz;
    }
    return a->tz > 0 && a->pbx <= 256 && a->pby <= 256 && a->pbz <= 256;
}

}  // namespace

// Plans the handle's passes for the memory there is; the handle runs the form where
// the plan is faster than the single-pass kernel.
int inlm::pair_plan(inlm_denoiser* d) {
    PairRun& r = d->pair;
    PairArgs& a = r.args;
    const int* pr = d->geo.patch_radius;
    size_t free_b = 0, total_b = 0;
    CUDA_TRY(cudaMemGetInfo(&free_b, &total_b));
    size_t budget = std::min(total_b / kWorkspaceShare, (free_b + idle_bytes(d->device)) / 2);
    if (r.limit > 0) budget = std::min(budget, r.limit);
    PairArgs deepest = a;  // (without a new plan the old one stays whole)
    deepest.tz = r.tz;
    const Plan plan = plan_blocks(deepest, pr, r.sms, r.warps, budget);
    r.active = false;
    const bool fused = d->p.precision == INLM_PRECISION_F32_FMA;
    if (plan.cost == 0 || (!r.forced && !plan_pays(deepest, pr, fused, d->tcfg.column, r.sms, r.warps, plan)))
        return INLM_OK;
    a.dist = nullptr;  // no tensor maps yet
    r.bx = plan.bx;
    r.by = plan.by;
    r.chunk = plan.chunk;
    a.tz = plan.tz;
    a.pbz = a.tz + 2 * pr[2] + a.szc;
    a.tiles_x = plan.tiles_x;
    a.tiles_y = plan.tiles_y;
    a.ex = plan.tiles_x * 32;
    a.ey = plan.tiles_y * 8;
    a.ring = plan.ring;
    r.bytes = plan.bytes(a.H);
    r.active = true;
    return INLM_OK;
}

// Whether the paired form covers the handle's configuration: an instantiated
// patch shape whose taps the tile kernel checked, weights that depend on
// |x|, |y|, |z| alone, and offsets in central symmetry with the first half
// at z <= 0 (the reference's z-major order always is).
int inlm::pair_configure(inlm_denoiser* d) {
    PairRun& r = d->pair;
    pair_idle(d);  // a workspace left by a call that failed may not fit the new plan
    r.active = false;
    const Geometry& g = d->geo;
    const int* pr = g.patch_radius;
    const int S = (int)g.search.size();
    if (!d->use_tile || d->device >= kMaxDevices || S < 2 || S % 2 || !pair_kernel_available(pr[0], pr[1], pr[2]))
        return INLM_OK;
    if (!pair_weights_symmetric(pr[0], pr[1], pr[2], d->targs.w)) return INLM_OK;
    for (int s = 0; s < S / 2; s++) {
        const Offset3 &o = g.search[s], &m = g.search[S - 1 - s];
        if (o.x != -m.x || o.y != -m.y || o.z != -m.z || o.z > 0) return INLM_OK;
    }
    for (int s = 1; s < S; s++)
        if (g.search[s].z < g.search[s - 1].z) return INLM_OK;
    // The fused column form (patch radius 1) sums its 7 taps by fused multiply-
    // adds in less time than the distances take to go through memory: 66 against
    // 84 ms at 256^3, search radius 10, 0.87 against 1.11 ms at 128 x 128 x 64,
    // radius 5. Where its CTAs leave a quarter of the SMs idle the paired form
    // wins by sharing out the offsets: 0.21 against 0.46 ms at 48 x 40 x 12.
    if (d->p.precision == INLM_PRECISION_F32_FMA && d->tcfg.column) {
        int sms = 0;
        CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, d->device));
        const long long ctas = (long long)d->targs.tiles_x * d->targs.tiles_y * ((d->shape[2] + d->tcfg.tz - 1) / d->tcfg.tz);
        if (4 * ctas >= 3ll * sms) return INLM_OK;
    }
    PairArgs& a = r.args;
    int smem_max = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, d->device));
    if (!pair_extents(g, d->shape, d->p.nslices, smem_max, &a)) return INLM_OK;
    for (int t = 0; t < (int)g.taps.size(); t++) a.w[t] = g.weights[t];
    r.tz = a.tz;
    CUDA_TRY(cudaDeviceGetAttribute(&r.sms, cudaDevAttrMultiProcessorCount, d->device));
    r.warps = pair_kernel_warps(pr[0]);
    std::vector<PairOffset> t(S);
    for (int s = 0; s < S; s++) {
        const Offset3& o = g.search[s];
        t[s].x = o.x;
        t[s].y = o.y;
        t[s].z = o.z;
        t[s].prev = (o.z * a.pby + o.y) * a.pbx + o.x;
    }
    std::vector<int> zs(2 * a.szc + 2, S);  // first offset of every z
    for (int s = S - 1; s >= 0; s--) zs[g.search[s].z + a.szc] = s;
    for (int i = 2 * a.szc; i >= 0; i--) zs[i] = std::min(zs[i], zs[i + 1]);
    CUDA_TRY(r.offsets.ensure(S * sizeof(PairOffset)));
    CUDA_TRY(r.z_start.ensure(zs.size() * sizeof(int)));
    CUDA_TRY(cudaMemcpyAsync(r.offsets.p, t.data(), S * sizeof(PairOffset), cudaMemcpyHostToDevice, d->stream));
    CUDA_TRY(cudaMemcpyAsync(r.z_start.p, zs.data(), zs.size() * sizeof(int), cudaMemcpyHostToDevice, d->stream));
    CUDA_TRY(cudaStreamSynchronize(d->stream));  // the host vectors go out of scope
    a.offsets = r.offsets.as<PairOffset>();
    a.z_start = r.z_start.as<int>();
    a.neg0 = -0.0f;
    a.raw_pad = d->d_raw_pad;
    a.gpitch_y = d->pitch_y;
    a.gpitch_z = d->pitch_z;
    a.out = d->d_next;
    a.mult = d->d_mult;
    a.err = d->d_err;
    return pair_plan(d);
}

// Points the handle's kernels at a workspace of at least r.bytes.
static int pair_bind(inlm_denoiser* d, void* ws) {
    PairRun& r = d->pair;
    PairArgs& a = r.args;
    if (a.dist == ws) return INLM_OK;  // the tensor maps are this buffer's
    a.dist = nullptr;
    const long long pad_dims[3] = {d->nxp, d->nyp, d->nzp}, pad_pitch[2] = {d->pitch_y, d->pitch_z};
    const int box[3] = {a.pbx, a.pby, a.pbz};
    int rc = encode_map_f32(&r.maps.prev, d->d_prev_pad, 3, pad_dims, pad_pitch, box);
    const int obox[4] = {32, 8, 1, 1};
    const long long dims[4] = {a.ex, a.ey, a.ring, a.H};
    const long long pitch[3] = {a.ex, (long long)a.ex * a.ey, (long long)a.ex * a.ey * a.ring};
    if (rc == INLM_OK) rc = encode_map_f32(&r.maps.out, ws, 4, dims, pitch, obox);
    for (int i = 0; i < 2 && rc == INLM_OK; i++) {
        const int dbox[4] = {kPairDistBox, pair_weight_rows(i), 1, 1};
        const int rbox[3] = {a.pbx, pair_weight_rows(i) + 2 * a.syr, 1};
        rc = encode_map_f32(&r.maps.dist[i], ws, 4, dims, pitch, dbox);
        if (rc == INLM_OK) rc = encode_map_f32(&r.maps.raw[i], d->d_raw_pad, 3, pad_dims, pad_pitch, rbox);
    }
    if (rc) return rc;
    a.dist = static_cast<float*>(ws);
    return INLM_OK;
}

// Borrows a workspace for the handle's next passes; *ok = false where there is
// no room for one. Where memory has become scarce since the handle was configured,
// the passes are planned anew for what is left.
static int pair_borrow(inlm_denoiser* d, bool* ok) {
    PairRun& r = d->pair;
    *ok = true;
    if (r.dist) return INLM_OK;
    if (!r.user) {
        count_user(d->device, 1);
        r.user = true;
    }
    r.dist = borrow(d->device, r.bytes, false);
    if (!r.dist) {
        const size_t wanted = r.bytes;
        const int rc = pair_plan(d);
        if (rc) return rc;
        if (r.active && r.bytes < wanted) r.dist = borrow(d->device, r.bytes, false);
        r.active = true;  // a later call may find room again
    }
    *ok = r.dist != nullptr;
    return r.dist ? pair_bind(d, r.dist->p) : INLM_OK;
}

// Borrows the workspace of the handle's passes; *ready = false when the form does
// not run here.
int inlm::pair_prepare(inlm_denoiser* d, bool* ready) {
    *ready = false;
    return d->pair.active ? pair_borrow(d, ready) : INLM_OK;
}

static int pair_launches(inlm_denoiser* d) {
    const PairRun& r = d->pair;
    const int* pr = d->geo.patch_radius;
    const bool fused = d->p.precision == INLM_PRECISION_F32_FMA;
    PairArgs a = r.args;
    const int depth = a.nz + a.szc;
    for (int y0 = 0; y0 < a.ny; y0 += r.by)
        for (int x0 = 0; x0 < a.nx; x0 += r.bx) {
            a.x0 = x0;
            a.x1 = std::min(a.nx, x0 + r.bx);
            a.y0 = y0;
            a.y1 = std::min(a.ny, y0 + r.by);
            a.xs = x0 - round_up(a.sxr, 8);
            a.ys = y0 - a.syr;
            a.tiles_x = (a.x1 + a.sxr - a.xs + 31) / 32;
            a.tiles_y = (a.y1 + a.syr - a.ys + 7) / 8;
            for (int z = 0; z < depth; z += r.chunk) {
                const int z1 = std::min(depth, z + r.chunk);
                a.tiles_z = (z1 - z + a.tz - 1) / a.tz;
                a.splits = offset_splits(a.tiles_x * a.tiles_y * a.tiles_z, r.sms, (a.H + r.warps - 1) / r.warps);
                CUDA_TRY(launch_pair_dist(pr[0], pr[1], pr[2], fused, r.maps, a, z, d->stream));
                const int w0 = std::max(0, z - a.szc), w1 = std::min(a.nz, z1 - a.szc);
                CUDA_TRY(launch_pair_weights(fused, r.maps, a, w0, w1, r.sms, d->stream));
                d->launches += 1 + (std::max(0, w1 - w0) + kPairGridZ - 1) / kPairGridZ;
            }
        }
    return INLM_OK;
}

// Enqueues one filter pass, after the last pass of another handle on the same
// workspace.
int inlm::pair_filter(inlm_denoiser* d) {
    PairBuf* b = d->pair.dist;
    if (b->alone) return pair_launches(d);
    std::lock_guard<std::mutex> lock(b->enqueue);
    if (b->last && b->last != d) CUDA_TRY(cudaStreamWaitEvent(d->stream, b->done, 0));
    const int rc = pair_launches(d);
    b->last = d;  // (whatever was enqueued counts)
    CUDA_TRY(cudaEventRecord(b->done, d->stream));
    return rc;
}

int inlm::pair_share(inlm_denoiser* d, PairBuf* b) {
    pair_idle(d);
    d->pair.shared = true;
    d->pair.dist = b;
    return pair_bind(d, b->p);
}

PairBuf* inlm::pair_take(int device, size_t bytes, bool alone) {
    count_user(device, 1);
    PairBuf* b = borrow(device, bytes, alone);
    if (!b) count_user(device, -1);
    return b;
}

void inlm::pair_give_back(PairBuf* b) {
    if (!b) return;
    const int device = b->device;
    hand_back(b);
    count_user(device, -1);
}

bool inlm::pair_trim(int device) {
    std::lock_guard<std::recursive_mutex> lock(g_pool_mutex);
    if (device < 0 || device >= kMaxDevices) return false;
    bool any = false;
    while (free_idle(g_pool[device])) any = true;
    return any;
}

void inlm::pair_idle(inlm_denoiser* d) {
    PairRun& r = d->pair;
    if (!r.dist || r.shared) return;
    hand_back(r.dist);
    r.dist = nullptr;
}

void inlm::pair_release(inlm_denoiser* d) {
    PairRun& r = d->pair;
    pair_idle(d);
    if (r.user) count_user(d->device, -1);
    r.user = false;
    r.offsets.release();
    r.z_start.release();
    r.active = false;
}

extern "C" int inlm_trim_memory(int device) {
    if (device < 0) return fail(INLM_ERR_ARG, "device %d", device);
    pair_trim(device);
    return INLM_OK;
}

extern "C" int inlm_debug_pair_workspace(inlm_denoiser* d, int64_t bytes) {
    if (!d) return fail(INLM_ERR_ARG, "null handle");
    if (!d->pair.offsets.p) return fail(INLM_ERR_UNSUPPORTED, "the paired form does not cover this handle");
    CUDA_TRY(cudaSetDevice(d->device));
    CUDA_TRY(cudaStreamSynchronize(d->stream));
    pair_idle(d);
    d->pair.limit = (size_t)std::llabs(bytes);
    d->pair.forced = bytes > 0;
    return pair_plan(d);
}

extern "C" int inlm_debug_pair_pool(int64_t bytes) {
    if (bytes < 0) return fail(INLM_ERR_ARG, "bad argument");
    g_pool_bound.store(bytes);
    return INLM_OK;
}

extern "C" int inlm_debug_pair_plan(const int shape[3], const inlm_params* p, int64_t bytes, double out[8]) {
    if (!shape || !p || !out || bytes < 0) return fail(INLM_ERR_ARG, "bad argument");
    const int* pr = p->patch_radius;
    if (!pair_kernel_available(pr[0], pr[1], pr[2])) return fail(INLM_ERR_UNSUPPORTED, "no kernels of this patch shape");
    const int pz = std::min(p->nslices / 2, p->search_radius[2]) + pr[2];
    const Geometry g = make_geometry(p->search_radius, pr, p->nslices, p->z_anisotropy, p->weight_table, shape[2] + 2 * pz);
    PairArgs a;
    if (!pair_extents(g, shape, p->nslices, 227 * 1024, &a)) return fail(INLM_ERR_UNSUPPORTED, "the box does not fit");
    const int sms = 148, warps = pair_kernel_warps(pr[0]);
    const Plan most = plan_blocks(a, pr, sms, warps, SIZE_MAX);
    const Plan plan = plan_blocks(a, pr, sms, warps, (size_t)bytes);
    TileArgs t{};
    const int depth = column_kernel_depth(pr[0], pr[1], pr[2]);
    t.pbx = (32 + 2 * a.px + 3) / 4 * 4;
    t.pby = 8 + 2 * a.py;
    t.pbz = depth + 2 * a.pz;
    const bool column = depth > 0 && column_smem_bytes(t) <= 227 * 1024;
    const bool runs = plan_pays(a, pr, p->precision == INLM_PRECISION_F32_FMA, column, sms, warps, plan);
    out[0] = runs ? 1.0 : 0.0;
    out[1] = plan.cost > 0 ? plan_time(a, pr, sms, plan) : 0.0;
    out[2] = plan_time(a, pr, sms, most);
    out[3] = (double)plan.bytes(a.H);
    out[4] = plan.bx;
    out[5] = plan.by;
    out[6] = plan.chunk;
    out[7] = plan.tz;
    return INLM_OK;
}

// Runs a check that leaves one 64-bit value on the device (from zero).
template <class T, class F>
static int device_check(T* out, F launch) {
    static_assert(sizeof(T) == 8, "one 64-bit value");
    T* p = nullptr;
    CUDA_TRY(dalloc(&p, 1));
    cudaError_t e = cudaMemset(p, 0, sizeof(T));
    if (e == cudaSuccess) e = launch(p);
    if (e == cudaSuccess) e = cudaMemcpy(out, p, sizeof(T), cudaMemcpyDeviceToHost);
    device_free(p);
    CUDA_TRY(e);
    return INLM_OK;
}

extern "C" int inlm_debug_weight_mismatches(int64_t* n) {
    if (!n) return fail(INLM_ERR_ARG, "null argument");
    unsigned long long h = 0;
    const int rc = device_check(&h, [](unsigned long long* p) { return launch_weight_mismatches(p, -0.0f, nullptr); });
    if (rc == INLM_OK) *n = (int64_t)h;
    return rc;
}

extern "C" int inlm_debug_fused_weight_error(double* worst) {
    if (!worst) return fail(INLM_ERR_ARG, "null argument");
    return device_check(worst, [](double* p) { return launch_fused_weight_error(p, nullptr); });
}
