// Paired-offset form of the plain and fused FP32 filter (filter_pair.cu):
// launch arguments and entry points.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "filter_kernels.cuh"

namespace inlm {

// One search offset s as both kernels read it.
struct __align__(16) PairOffset {
    int x, y, z;  // s
    int prev;     // distance kernel: delta of s inside the staged prev box
};

constexpr int kPairGridZ = 65535;  // planes per launch of the weight kernel: the largest grid.z
constexpr int kPairDistBox = 36;  // columns of a distance tile: 32 and the misalignment of its start

struct PairArgs {
    int nz;                    // planes of the volume
    int x0, x1, y0, y1;        // voxels this block filters
    int xs, ys;                // first column and row of the block's workspace planes
    int px, py, pz;            // padding of the volume per side
    int syr, sxr, szc;         // search radius, z clipped
    int S, H;                  // offsets, and the first half of them
    int tz;                    // planes per tile of the distance kernel
    int ring;                  // workspace planes per offset (z modulo ring)
    int ex, ey;                // workspace plane extents
    int tiles_x, tiles_y, tiles_z;
    int splits;                // CTAs that share a tile's offsets
    int pbx, pby, pbz;         // staged prev box
    const PairOffset* __restrict__ offsets;
    const int* __restrict__ z_start;  // first offset of z = -szc, ..., szc; then S
    float neg0;                // -0.0f, unknown to the compiler (pair_math.cuh)
    float* __restrict__ dist;  // [H][ring][ey][ex] patch distances
    const float* __restrict__ raw_pad;
    long long gpitch_y, gpitch_z;
    float* __restrict__ out;
    int nx, ny;                // pitches of out
    const float* __restrict__ mult;
    int* err;
    float w[kMaxTaps];         // patch weights, reference tap order
};

// Patch shapes the form is instantiated for.
bool pair_kernel_available(int rx, int ry, int rz);
// Whether the weights depend on |x|, |y|, |z| of a tap alone (the kernel shares
// their products between mirrored taps).
bool pair_weights_symmetric(int rx, int ry, int rz, const float* w);
// Warps per CTA of the distance kernel; one CTA runs per SM.
int pair_kernel_warps(int rx);
// Row pitch of the staged prev box for a padding of px columns (0: too wide).
int pair_box_pitch(int px);
size_t pair_smem_bytes(int rx, int rz, const PairArgs& a);
// Tensor maps: the padded previous iterate (prev box), the workspace in tiles
// of 32 x 8 (stored by the distance kernel), and for the weight kernel's two
// tile heights the workspace in tiles of kPairDistBox columns and the padded
// raw volume in tiles of pbx columns.
struct PairMaps {
    CUtensorMap prev, out, dist[2], raw[2];
};
// Distances of the planes [z0, z0 + tiles_z * tz) into the ring.
cudaError_t launch_pair_dist(int rx, int ry, int rz, bool fused, const PairMaps& m, const PairArgs& a, int z0,
                             cudaStream_t st);
int pair_weight_rows(int i);  // rows per CTA: i 0 (8 rows per thread), 1 (2 rows)
int pair_weight_small(long long warps, int sms);  // that i, for a launch of so many warps of 32 x 8 voxels
// Weights, sums and results of the planes [z0, z1) from the ring.
cudaError_t launch_pair_weights(bool fused, const PairMaps& m, const PairArgs& a, int z0, int z1, int sms,
                                cudaStream_t st);

// Counts the x in [-3.6, -0] whose exact_weight_pair_fast step differs from
// exact_weight_pair's.
cudaError_t launch_weight_mismatches(unsigned long long* n, float neg0, cudaStream_t st);
// Raises *worst to the largest relative error of fused_weight_pair over the x that
// it weighs (1e300: an x past the cutoff weighs something).
cudaError_t launch_fused_weight_error(double* worst, cudaStream_t st);

}  // namespace inlm
