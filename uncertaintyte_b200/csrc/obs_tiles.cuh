// obs_tiles.cuh - the observations of a camera in tiles, shared by the camera
// block kernels (assembly.cu) and the point covariances (points.cu).
#pragma once
#include "internal.h"

namespace unc {

// Observations are numbered by position in the camera order: those of camera c
// are the positions [cam_ptr[c], cam_ptr[c+1]), cut into tiles of kObsTile.
// Camera c owns the tile slots [base(c), base(c+1)) with base(c) = c +
// cam_ptr[c] / kObsTile: never fewer than its tiles, since
// ceil((B - A) / T) <= floor(B / T) - floor(A / T) + 1. Slots past a camera's
// last tile are empty. The slot count base(C) is bounded on the host by
// C + num_obs / kObsTile, so the grids need no read-back; a CTA finds its
// camera by binary search over cam_ptr.
constexpr int kObsTile = 256;

__device__ __forceinline__ int tile_base(const int* __restrict__ cam_ptr, int c) {
    return c + cam_ptr[c] / kObsTile;
}

struct ObsTile {
    int cam, begin, end;
};

__device__ __forceinline__ bool find_tile(const int* __restrict__ cam_ptr, int num_cams, int k, ObsTile& t) {
    if (k >= tile_base(cam_ptr, num_cams)) return false;
    int lo = 0, hi = num_cams;  // tile_base(lo) <= k < tile_base(hi)
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (tile_base(cam_ptr, mid) <= k)
            lo = mid;
        else
            hi = mid;
    }
    t.cam = lo;
    t.end = cam_ptr[lo + 1];
    t.begin = min(cam_ptr[lo] + (k - tile_base(cam_ptr, lo)) * kObsTile, t.end);
    t.end = min(t.begin + kObsTile, t.end);
    return true;
}

// The tile's Jacobian records (24 doubles: row 0's 9 camera and 3 point values,
// then row 1's) into shared memory, kRecStride doubles apart, by all kObsTile
// threads: the records are scattered, so twelve threads take one record's
// twelve 16-byte pieces side by side (a thread per record would touch as many
// cache lines per load as there are threads). ids: kObsTile shared ints.
constexpr int kRecStride = 26;  // 16-byte aligned records, two-way bank conflicts when a thread reads its own
__device__ __forceinline__ void stage_records(double* sj, int* ids, const double* __restrict__ J,
                                              const int* __restrict__ cam_obs, const ObsTile& tile) {
    const int n = tile.end - tile.begin, t = threadIdx.x;
    if (t < n) ids[t] = cam_obs[tile.begin + t];
    __syncthreads();
    for (int k = t; k < 12 * n; k += kObsTile) {
        const int i = k / 12, q = k - 12 * i;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                         static_cast<unsigned>(__cvta_generic_to_shared(sj + i * kRecStride + 2 * q))),
                     "l"(J + 24L * ids[i] + 2 * q)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
}

}  // namespace unc
