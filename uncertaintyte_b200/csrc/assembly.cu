// assembly.cu - sparse-Jacobian ingest, J^T J block assembly, point 3x3
// inverses and the camera Schur-complement scatter (sm_100a).
//
// Replaces, for the TAYLOR_EXPANSION path of uncertaintyTE:
//   fixPts                       compute.cpp:283-368
//   SSM::scaleMat(RIGHT)         ScaledSparseMatrix.cpp:334-358, compute.cpp:77-82
//   J^T J + splitTo3Blocks       compute.cpp:86-96, ScaledSparseMatrix.cpp:238-299,517-539
//   inv3x3blockSymmDiag          ScaledSparseMatrix.cpp:210-230
//   Z = U - W iV W^T (dense)     compute.cpp:108-112
//
// Device layout: the Jacobian values are used in place. With the reference's
// layout (every row 12 entries) observation o occupies values[24o, 24o+24):
// [row0: 9 camera, 3 point | row1: 9 camera, 3 point], a 192-byte record
// read with 128-bit loads. Fixed-point observations are masked (obs_pt = -1)
// instead of compacted; the reference deletes those rows (compute.cpp:337-366).
#include <algorithm>

#include "obs_tiles.cuh"

namespace unc {

// ------------------------------------------------------------------------
// validation / ids
// ------------------------------------------------------------------------
__global__ void k_validate_obs(int num_obs, int num_cams, int num_points, int3 fix, int has_fix,
                               long nnz, const int* __restrict__ rows, const int* __restrict__ cols,
                               int* __restrict__ obs_cam, int* __restrict__ obs_pt, int* err) {
    int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= num_obs) return;
    const long base = 24L * o;
    bool bad = rows[2 * o] != base || rows[2 * o + 1] != base + 12 || rows[2 * o + 2] != base + 24 ||
               base + 24 > nnz;
    int cam = -1, pt = -1;
    if (!bad) {
        const int4* c4 = reinterpret_cast<const int4*>(cols + base);
        int c[24];
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            int4 v = c4[q];
            c[4 * q] = v.x;
            c[4 * q + 1] = v.y;
            c[4 * q + 2] = v.z;
            c[4 * q + 3] = v.w;
        }
        cam = c[0] / kCamParams;
        const int cam_off = kCamParams * num_cams;
        pt = (c[9] - cam_off) / 3;
        bad |= c[0] < 0 || cam >= num_cams || c[9] < cam_off || pt >= num_points;
#pragma unroll
        for (int j = 0; j < 9; ++j) bad |= (c[j] != cam * 9 + j) | (c[12 + j] != cam * 9 + j);
#pragma unroll
        for (int j = 0; j < 3; ++j)
            bad |= (c[9 + j] != cam_off + 3 * pt + j) | (c[21 + j] != cam_off + 3 * pt + j);
    }
    if (bad) {
        atomicOr(err, ERRBIT_LAYOUT);
        cam = pt = -1;
    } else if (has_fix && (pt == fix.x || pt == fix.y || pt == fix.z)) {
        cam = pt = -1;  // all rows of a fixed point are deleted (compute.cpp:337-366)
    }
    obs_cam[o] = cam;
    obs_pt[o] = pt;
}

void launch_validate_obs(const SceneDev& s, cudaStream_t st) {
    if (s.num_obs == 0) return;
    int3 fix = make_int3(s.fix[0], s.fix[1], s.fix[2]);
    k_validate_obs<<<(s.num_obs + 255) / 256, 256, 0, st>>>(s.num_obs, s.num_cams, s.num_points,
                                                            fix, s.has_fix, s.nnz, s.rows, s.cols,
                                                            s.obs_cam, s.obs_pt, s.err);
    count_launch();
}

// Generic repack for J^T J export: rows of 12 (camera + point) or 9 (camera
// only) entries; writes the 24-value observation record with zero point part.
__global__ void k_repack_generic(int num_obs, int num_cams, int num_points, const int* __restrict__ rows,
                                 const int* __restrict__ cols, const double* __restrict__ vals,
                                 double* __restrict__ J, int* obs_cam, int* obs_pt, int* err) {
    int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= num_obs) return;
    int r0 = rows[2 * o], r1 = rows[2 * o + 1], r2 = rows[2 * o + 2];
    int n0 = r1 - r0, n1 = r2 - r1;
    bool bad = n0 != n1 || (n0 != 12 && n0 != 9);
    int cam = -1, pt = -1;
    double* out = J + 24L * o;
    const int cam_off = kCamParams * num_cams;
    if (!bad) {
        cam = cols[r0] / kCamParams;
        bad = cols[r0] < 0 || cam >= num_cams;
        for (int j = 0; j < 9; ++j) {
            bad |= cols[r0 + j] != cam * 9 + j || cols[r1 + j] != cam * 9 + j;
            out[j] = vals[r0 + j];
            out[12 + j] = vals[r1 + j];
        }
        if (n0 == 12) {
            pt = (cols[r0 + 9] - cam_off) / 3;
            bad |= cols[r0 + 9] < cam_off || pt >= num_points;
            for (int j = 0; j < 3; ++j) {
                bad |= cols[r0 + 9 + j] != cam_off + 3 * pt + j || cols[r1 + 9 + j] != cam_off + 3 * pt + j;
                out[9 + j] = vals[r0 + 9 + j];
                out[21 + j] = vals[r1 + 9 + j];
            }
        } else {
            for (int j = 0; j < 3; ++j) out[9 + j] = out[21 + j] = 0.0;
        }
    }
    if (bad) {
        atomicOr(err, ERRBIT_LAYOUT);
        cam = pt = -1;
    }
    obs_cam[o] = cam;
    obs_pt[o] = pt;
}

void launch_repack_generic(int num_obs, int num_cams, int num_points, const int* rows, const int* cols,
                           const double* vals, double* J, int* obs_cam, int* obs_pt, int* err,
                           cudaStream_t st) {
    if (num_obs == 0) return;
    k_repack_generic<<<(num_obs + 255) / 256, 256, 0, st>>>(num_obs, num_cams, num_points, rows, cols, vals, J,
                                                            obs_cam, obs_pt, err);
    count_launch();
}

// ------------------------------------------------------------------------
// observation index by camera and by point
// ------------------------------------------------------------------------
// A stable counting sort by camera (ascending observation id within a camera)
// without sorting a segment: the observations are cut into chunks, one per CTA,
// a chunk into eight contiguous parts, one per warp, and a warp places its
// observations in order, 32 at a time. Counts and positions live in shared
// memory, so that a few cameras do not serialise on their counters in L2
// (342k observations of 200 cameras: 48 us to count and 50 us to place with
// global atomics). The points' lists (short, many) are placed with global
// atomics and brought into order by rank: an entry counts the smaller positions
// of its list. Cameras are taken kIndexCams at a time (one pass up to that many).
constexpr int kIndexCams = 5120;
constexpr int kIndexThreads = 256, kIndexWarps = kIndexThreads / 32;
constexpr int kIndexChunks = 148;   // at most
constexpr int kScanItems = 2048;    // point counts per block of the scan
constexpr int kScanGroup = 32;      // cameras per block of the scan

struct IndexShape {
    int chunks, per_chunk, point_blocks, cam_blocks;  // per_chunk: a multiple of 32 * kIndexWarps
};
IndexShape index_shape(int num_obs, int num_points, int range) {
    IndexShape x;
    const int step = 32 * kIndexWarps;
    x.chunks = std::max(1, std::min(kIndexChunks, (num_obs + 4 * step - 1) / (4 * step)));
    x.per_chunk = ((num_obs + x.chunks - 1) / x.chunks + step - 1) / step * step;
    x.point_blocks = (num_points + kScanItems - 1) / kScanItems;
    x.cam_blocks = (range + kScanGroup - 1) / kScanGroup;
    return x;
}

// hist[chunk][c] = observations of camera c0 + c in the chunk; the points'
// counts in the first pass.
__global__ void __launch_bounds__(kIndexThreads)
    k_index_count(int num_obs, int per_chunk, int c0, int range, const int* __restrict__ obs_cam,
                  const int* __restrict__ obs_pt, int* __restrict__ hist, int* pt_cnt) {
    extern __shared__ int counts[];
    for (int c = threadIdx.x; c < range; c += kIndexThreads) counts[c] = 0;
    __syncthreads();
    const int b = blockIdx.x * per_chunk, e = min(num_obs, b + per_chunk);
    for (int o = b + threadIdx.x; o < e; o += kIndexThreads) {
        const unsigned c = (unsigned)(obs_cam[o] - c0);
        if (c < (unsigned)range) atomicAdd(counts + c, 1);
        if (c0 == 0) {
            const int p = obs_pt[o];
            if (p >= 0) atomicAdd(pt_cnt + p, 1);
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < range; c += kIndexThreads) hist[(long)blockIdx.x * range + c] = counts[c];
}

// In-place exclusive scan of a[0, n) in shared memory by the block; the total.
__device__ int block_scan(int* a, int n, int* tmp) {
    const int per = (n + kIndexThreads - 1) / kIndexThreads;
    const int b = min(n, (int)threadIdx.x * per), e = min(n, b + per);
    int s = 0;
    for (int i = b; i < e; ++i) s += a[i];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = s;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) tmp[w] = x;
    __syncthreads();
    int base = x - s, total = 0;
    for (int q = 0; q < kIndexWarps; ++q) {
        if (q < w) base += tmp[q];
        total += tmp[q];
    }
    for (int i = b; i < e; ++i) {
        const int v = a[i];
        a[i] = base;
        base += v;
    }
    __syncthreads();
    return total;
}

// Blocks [0, point_blocks): the sum of their points' counts. The others: per
// camera the exclusive scan of its counts over the chunks (in place) and its
// total; the last of them to finish turns the totals into cam_ptr[c0 ..].
__global__ void __launch_bounds__(kIndexThreads)
    k_index_scan(int point_blocks, int num_points, const int* __restrict__ pt_cnt, int* __restrict__ pt_sums, int chunks,
                 int c0, int range, int* __restrict__ hist, int* totals, int* cam_ptr, int* ticket) {
    extern __shared__ int buf[];
    __shared__ int tmp[kIndexWarps], last;
    const int t = threadIdx.x;
    if ((int)blockIdx.x < point_blocks) {
        int s = 0;
        for (int i = t; i < kScanItems; i += kIndexThreads) {
            const int p = blockIdx.x * kScanItems + i;
            s += p < num_points ? pt_cnt[p] : 0;
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        if ((t & 31) == 0) tmp[t >> 5] = s;
        __syncthreads();
        if (t == 0) {
            int v = 0;
            for (int q = 0; q < kIndexWarps; ++q) v += tmp[q];
            pt_sums[blockIdx.x] = v;
        }
        return;
    }
    // eight threads per camera, each a contiguous share of the chunks
    const int c = (blockIdx.x - point_blocks) * kScanGroup + (t & 31), part = t >> 5;
    const int k0 = chunks * part / kIndexWarps, k1 = chunks * (part + 1) / kIndexWarps;
    int s = 0;
    if (c < range)
#pragma unroll 8
        for (int k = k0; k < k1; ++k) s += hist[(long)k * range + c];
    buf[t] = s;
    __syncthreads();
    int run = 0;
    for (int q = 0; q < part; ++q) run += buf[32 * q + (t & 31)];
    if (c < range) {
        if (part == kIndexWarps - 1) totals[c0 + c] = run + s;
#pragma unroll 8
        for (int k = k0; k < k1; ++k) {
            const int v = hist[(long)k * range + c];
            hist[(long)k * range + c] = run;
            run += v;
        }
    }
    __threadfence();
    __syncthreads();
    if (t == 0) last = atomicAdd(ticket, 1) == (int)gridDim.x - point_blocks - 1;
    __syncthreads();
    if (!last) return;
    for (int i = t; i < range; i += kIndexThreads) buf[i] = __ldcg(totals + c0 + i);
    __syncthreads();
    const int total = block_scan(buf, range, tmp);
    const int base = c0 ? __ldcg(cam_ptr + c0) : 0;
    for (int i = t; i < range; i += kIndexThreads) cam_ptr[c0 + i] = base + buf[i];
    if (t == 0) {
        cam_ptr[c0 + range] = base + total;
        *ticket = 0;
    }
}

// pt_ptr (and a copy of it, advanced by the placing) from the counts and the blocks' sums.
__global__ void __launch_bounds__(kIndexThreads)
    k_index_points(int num_points, const int* __restrict__ pt_sums, int* pt_cnt, int* __restrict__ pt_ptr, int* err) {
    __shared__ int buf[kScanItems], tmp[kIndexWarps];
    const int t = threadIdx.x, p0 = blockIdx.x * kScanItems;
    int before = 0;
    for (int i = t; i < (int)blockIdx.x; i += kIndexThreads) before += pt_sums[i];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) before += __shfl_xor_sync(0xffffffffu, before, d);
    if ((t & 31) == 0) tmp[t >> 5] = before;
    for (int i = t; i < kScanItems; i += kIndexThreads) {
        const int cnt = p0 + i < num_points ? pt_cnt[p0 + i] : 0;
        buf[i] = cnt;
        if (cnt > kSchurMaxList) atomicOr(err, ERRBIT_SCHUR_CAP);
    }
    __syncthreads();
    before = 0;
    for (int q = 0; q < kIndexWarps; ++q) before += tmp[q];
    __syncthreads();
    const int total = block_scan(buf, kScanItems, tmp);
    for (int i = t; i < kScanItems; i += kIndexThreads)
        if (p0 + i < num_points) {
            pt_ptr[p0 + i] = before + buf[i];
            pt_cnt[p0 + i] = before + buf[i];
        }
    if (t == 0 && blockIdx.x == gridDim.x - 1) pt_ptr[num_points] = before + total;
}

// cam_obs (the observation at each position) and the points' lists in arrival order.
__global__ void __launch_bounds__(kIndexThreads)
    k_index_place(int num_obs, int per_chunk, int c0, int range, const int* __restrict__ obs_cam,
                  const int* __restrict__ obs_pt, const int* __restrict__ hist, const int* __restrict__ cam_ptr,
                  int* pt_cur, int* __restrict__ cam_obs, int2* __restrict__ pt_tmp) {
    extern __shared__ int counts[];  // [warp][range]
    for (int c = threadIdx.x; c < kIndexWarps * range; c += kIndexThreads) counts[c] = 0;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, per_warp = per_chunk / kIndexWarps;
    const int b = min(num_obs, (int)blockIdx.x * per_chunk + warp * per_warp), e = min(num_obs, b + per_warp);
    int* const mine = counts + warp * range;
    for (int o = b + lane; o < e; o += 32) {
        const unsigned c = (unsigned)(obs_cam[o] - c0);
        if (c < (unsigned)range) atomicAdd(mine + c, 1);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < range; c += kIndexThreads) {
        int run = cam_ptr[c0 + c] + hist[(long)blockIdx.x * range + c];
        for (int w = 0; w < kIndexWarps; ++w) {
            const int v = counts[w * range + c];
            counts[w * range + c] = run;
            run += v;
        }
    }
    __syncthreads();
    for (int o0 = b; o0 < e; o0 += 32) {
        const int o = o0 + lane;
        const int cam = o < e ? obs_cam[o] : -1;
        const unsigned c = (unsigned)(cam - c0);
        const bool in = cam >= 0 && c < (unsigned)range;
        const unsigned same = __match_any_sync(0xffffffffu, in ? (int)c : -1);
        const int rank = __popc(same & ((1u << lane) - 1u));
        const int pos = in ? mine[c] + rank : 0;
        __syncwarp();
        if (in && rank == 0) mine[c] = pos + __popc(same);
        __syncwarp();
        if (in) {
            cam_obs[pos] = o;
            const int p = obs_pt[o];
            if (p >= 0) pt_tmp[atomicAdd(pt_cur + p, 1)] = make_int2(pos, cam);
        }
    }
}

// Every list entry to its rank in its point's list (ascending positions, so
// ascending cameras); per position: its list's start and its rank in it. The count
// is quadratic, so lists of more than kSchurMaxList entries are left alone: a solve
// refuses them, J^T J and the SVD algorithms place them by k_index_long.
__global__ void __launch_bounds__(kIndexThreads)
    k_index_rank(int num_cams, const int* __restrict__ cam_ptr, const int* __restrict__ cam_obs,
                 const int* __restrict__ obs_cam, const int* __restrict__ obs_pt, const int* __restrict__ pt_ptr,
                 const int2* __restrict__ pt_tmp, int2* __restrict__ pt_list, int2* __restrict__ pos_list) {
    const int i = blockIdx.x * kIndexThreads + threadIdx.x;
    if (i >= cam_ptr[num_cams]) return;
    const int o = cam_obs[i], p = obs_pt[o];
    if (p < 0) {
        pos_list[i] = make_int2(0, 0);
        return;
    }
    const int b = pt_ptr[p], e = pt_ptr[p + 1];
    if (e - b > kSchurMaxList) {
        pos_list[i] = make_int2(0, 0);
        return;
    }
    int rank = 0;
    for (int k = b; k < e; ++k) rank += pt_tmp[k].x < i;
    pt_list[b + rank] = make_int2(i, obs_cam[o]);
    pos_list[i] = make_int2(b, rank);
}

// The lists that k_index_rank leaves: one CTA walks the positions in order and keeps
// those of the point. There are at most num_obs / kSchurMaxList such lists.
__global__ void __launch_bounds__(kIndexThreads)
    k_index_long(int num_cams, int num_points, const int* __restrict__ cam_ptr, const int* __restrict__ cam_obs,
                 const int* __restrict__ obs_cam, const int* __restrict__ obs_pt, const int* __restrict__ pt_ptr,
                 int2* __restrict__ pt_list) {
    __shared__ int lists[kIndexThreads], count, found[kIndexWarps];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, n = cam_ptr[num_cams];
    for (long p0 = (long)blockIdx.x * kIndexThreads; p0 < num_points; p0 += (long)gridDim.x * kIndexThreads) {
        if (t == 0) count = 0;
        __syncthreads();
        if (p0 + t < num_points && pt_ptr[p0 + t + 1] - pt_ptr[p0 + t] > kSchurMaxList)
            lists[atomicAdd(&count, 1)] = (int)p0 + t;
        __syncthreads();
        for (int q = 0; q < count; ++q) {
            const int p = lists[q];
            int at = pt_ptr[p];
            for (int i0 = 0; i0 < n; i0 += kIndexThreads) {
                const int i = i0 + t, o = i < n ? cam_obs[i] : -1;
                const bool mine = o >= 0 && obs_pt[o] == p;
                const unsigned votes = __ballot_sync(0xffffffffu, mine);
                if (lane == 0) found[warp] = __popc(votes);
                __syncthreads();
                int before = at;
                for (int w = 0; w < kIndexWarps; ++w) {
                    before += w < warp ? found[w] : 0;
                    at += found[w];
                }
                if (mine) pt_list[before + __popc(votes & ((1u << lane) - 1u))] = make_int2(i, obs_cam[o]);
                __syncthreads();  // found is rewritten
            }
        }
        __syncthreads();  // count is rewritten
    }
}

size_t index_scratch_ints(int num_cams, int num_points) {
    const size_t range = std::min(num_cams, kIndexCams);
    return 1 + (size_t)num_points + (size_t)num_cams + (num_points + kScanItems - 1) / kScanItems + kIndexChunks * range;
}

void launch_build_index(SceneDev& s, cudaStream_t st) {
    const int C = s.num_cams, P = s.num_points, n = s.num_obs;
    // scratch: ticket, the points' counts, camera totals, the scan's block sums, the chunks' histograms
    int* ticket = s.index_tmp;
    int* pt_cnt = ticket + 1;
    int* totals = pt_cnt + P;
    int* pt_sums = totals + C;
    int* hist = pt_sums + (P + kScanItems - 1) / kScanItems;
    cudaMemsetAsync(ticket, 0, sizeof(int) * ((size_t)P + 1), st);
    if (P == 0) cudaMemsetAsync(s.pt_ptr, 0, sizeof(int), st);
    prepare_assembly_kernels();
    for (int c0 = 0; c0 < C; c0 += kIndexCams) {
        const int range = std::min(kIndexCams, C - c0);
        const IndexShape x = index_shape(n, c0 == 0 ? P : 0, range);
        k_index_count<<<x.chunks, kIndexThreads, sizeof(int) * range, st>>>(n, x.per_chunk, c0, range, s.obs_cam, s.obs_pt,
                                                                            hist, pt_cnt);
        k_index_scan<<<x.point_blocks + x.cam_blocks, kIndexThreads, sizeof(int) * std::max(range, kIndexThreads), st>>>(
            x.point_blocks, P, pt_cnt, pt_sums, x.chunks, c0, range, hist, totals, s.cam_ptr, ticket);
        if (x.point_blocks) k_index_points<<<x.point_blocks, kIndexThreads, 0, st>>>(P, pt_sums, pt_cnt, s.pt_ptr, s.err);
        k_index_place<<<x.chunks, kIndexThreads, sizeof(int) * kIndexWarps * range, st>>>(
            n, x.per_chunk, c0, range, s.obs_cam, s.obs_pt, hist, s.cam_ptr, pt_cnt, s.cam_obs, s.pt_tmp);
        count_launch(x.point_blocks ? 4 : 3);
    }
    if (n > 0) {
        k_index_rank<<<(n + kIndexThreads - 1) / kIndexThreads, kIndexThreads, 0, st>>>(
            C, s.cam_ptr, s.cam_obs, s.obs_cam, s.obs_pt, s.pt_ptr, s.pt_tmp, s.pt_list, s.pos_list);
        count_launch();
    }
}

void launch_long_lists(const SceneDev& s, cudaStream_t st) {
    if (s.num_obs <= kSchurMaxList || s.num_points == 0) return;
    const int blocks = std::min((s.num_points + kIndexThreads - 1) / kIndexThreads, 4 * device_sms());
    k_index_long<<<blocks, kIndexThreads, 0, st>>>(s.num_cams, s.num_points, s.cam_ptr, s.cam_obs, s.obs_cam, s.obs_pt,
                                                   s.pt_ptr, s.pt_list);
    count_launch();
}

// ------------------------------------------------------------------------
// J^T J blocks
// ------------------------------------------------------------------------
// upper-triangle index of (j,k), j <= k < 9, row-major: t = j*9 - j*(j-1)/2 + (k-j)
__host__ __device__ constexpr int ut9(int j, int k) { return j * 9 - (j * (j - 1)) / 2 + (k - j); }

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}

// Load the 18 camera values of observation o (row0 c0..c8, row1 c0..c8) with
// 128-bit loads from the 24-double record.
__device__ __forceinline__ void load_cam_rows(const double* __restrict__ J, int o, double r0[9],
                                              double r1[9]) {
    const double2* q = reinterpret_cast<const double2*>(J + 24L * o);
    double2 a0 = __ldg(q + 0), a1 = __ldg(q + 1), a2 = __ldg(q + 2), a3 = __ldg(q + 3),
            a4 = __ldg(q + 4);
    double2 b0 = __ldg(q + 6), b1 = __ldg(q + 7), b2 = __ldg(q + 8), b3 = __ldg(q + 9),
            b4 = __ldg(q + 10);
    r0[0] = a0.x; r0[1] = a0.y; r0[2] = a1.x; r0[3] = a1.y; r0[4] = a2.x;
    r0[5] = a2.y; r0[6] = a3.x; r0[7] = a3.y; r0[8] = a4.x;
    r1[0] = b0.x; r1[1] = b0.y; r1[2] = b1.x; r1[3] = b1.y; r1[4] = b2.x;
    r1[5] = b2.y; r1[6] = b3.x; r1[7] = b3.y; r1[8] = b4.x;
}

__device__ __forceinline__ void load_pt_rows(const double* __restrict__ J, int o, double p0[3],
                                             double p1[3]) {
    const double* r = J + 24L * o;
    double2 a = __ldg(reinterpret_cast<const double2*>(r + 8));   // c8, p0
    double2 b = __ldg(reinterpret_cast<const double2*>(r + 10));  // p1, p2
    double2 c = __ldg(reinterpret_cast<const double2*>(r + 20));  // c8', p0'
    double2 d = __ldg(reinterpret_cast<const double2*>(r + 22));  // p1', p2'
    p0[0] = a.y; p0[1] = b.x; p0[2] = b.y;
    p1[0] = c.y; p1[1] = d.x; p1[2] = d.y;
}

// Per-tile partial sums of a camera are combined in slot order: a fixed
// summation order, bitwise repeatable.
size_t camera_tile_slots(int num_cams, int num_obs) { return (size_t)num_cams + num_obs / kObsTile + 1; }

// (j, k), j <= k, of upper-triangle element el (inverse of ut9)
__device__ __forceinline__ void ut9_inv(int el, int& j, int& k) {
    j = 0;
    while (j < 8 && ut9(j + 1, j + 1) <= el) ++j;
    k = j + (el - ut9(j, j));
}

// One pass over the tile's Jacobian records:
//   * the partial sums of U = sum_o Jc_o^T Jc_o;
//   * Q_o = W_o M_p, W_o = Jc_o^T Jp_o, M_p M_p^T = the inverse of the point's
//     block (k_point_blocks): the record the Schur complement reads, not yet
//     scaled by the camera's column norms. Written in position order, so the
//     tile's records are one contiguous store of 27 doubles each;
//   * the partial sums of Q_o Q_o^T, the self terms of the Schur complement's
//     diagonal block (formed here, where the records are in shared memory, and
//     not in the column kernel: 29 us of a column's first CTA at 200 cameras).
// Shared-memory instructions and the latency of the scattered records bound the
// kernel (192 bytes in and 216 out per observation are 22 us at 342,000), so both
// sums are outer products on the FP64 tensor cores: a third of the reads (57 us at
// that size; as much for U alone with ordinary multiply-adds).
constexpr size_t kCamTileSmem = sizeof(double) * kObsTile * 27;
static_assert(27 >= kRecStride, "the staged records fit the Q records' space");

// sum_k x_k x_k^T over k in [k0, k1), a multiple of 4 apart, x_k in R^9, by one warp:
// x(k, e) is element e of x_k. out: the 45 upper elements.
template <class F>
__device__ __forceinline__ void outer_sum(int k0, int k1, F&& x, double* out) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    double c[2] = {0.0, 0.0}, row = 0.0, corner = 0.0;
#pragma unroll 4
    for (int k = k0 + t; k < k1; k += 4) {
        const double a = x(k, g), a8 = x(k, 8);
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                     : "+d"(c[0]), "+d"(c[1])
                     : "d"(a), "d"(a));
        row = fma(a8, a, row);
        corner = fma(a8, a8, corner);
    }
#pragma unroll
    for (int d = 1; d < 4; d <<= 1) {
        row += __shfl_xor_sync(0xffffffffu, row, d);
        corner += __shfl_xor_sync(0xffffffffu, corner, d);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
        if (g >= 2 * t + h) out[ut9(2 * t + h, g)] = c[h];
    if (t == 0) out[ut9(g, 8)] = row;
    if (lane == 0) out[ut9(8, 8)] = corner;
}

__global__ void __launch_bounds__(kObsTile, 2)
    k_camera_tiles(int num_cams, const double* __restrict__ J, const int* __restrict__ cam_ptr,
                   const int* __restrict__ cam_obs, const int* __restrict__ obs_pt, const double* __restrict__ Mp,
                   double* __restrict__ part, double* __restrict__ Q) {
    extern __shared__ __align__(16) double sj[];
    __shared__ int ids[kObsTile];
    __shared__ double red[kObsTile / 32][2][45];
    ObsTile tile;
    if (!find_tile(cam_ptr, num_cams, blockIdx.x, tile)) return;
    const int n = tile.end - tile.begin, t = threadIdx.x, warp = t >> 5;
    stage_records(sj, ids, J, cam_obs, tile);
    double m[6] = {0, 0, 0, 0, 0, 0};
    if (t < n) {
        const int p = obs_pt[ids[t]];
        const double2* src = reinterpret_cast<const double2*>(Mp + 6L * (p < 0 ? 0 : p));
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double2 v = __ldg(src + k);
            m[2 * k] = v.x;
            m[2 * k + 1] = v.y;
        }
    }
    // U: k = 2 observation + row
    const int i0 = 32 * warp;
    outer_sum(2 * i0, 2 * (i0 + 32), [&](int k, int e) {
        const int i = k >> 1;
        return i < n ? sj[i * kRecStride + 12 * (k & 1) + e] : 0.0;
    }, red[warp][0]);
    double q[27];
    if (t < n) {
        const double* r = sj + t * kRecStride;
        const double a0 = r[9], a1 = r[10], a2 = r[11], b0 = r[21], b1 = r[22], b2 = r[23];
#pragma unroll
        for (int j = 0; j < 9; ++j) {
            const double u = r[j], v = r[12 + j];
            const double w0 = u * a0 + v * b0, w1 = u * a1 + v * b1, w2 = u * a2 + v * b2;
            q[3 * j] = w0 * m[0];
            q[3 * j + 1] = fma(w1, m[2], w0 * m[1]);
            q[3 * j + 2] = fma(w2, m[5], fma(w1, m[4], w0 * m[3]));
        }
    }
    __syncthreads();
    if (t < n) {
#pragma unroll
        for (int e = 0; e < 27; ++e) sj[27 * t + e] = q[e];
    }
    __syncthreads();
    double* out = Q + 27L * tile.begin;
    for (int i = t; i < 27 * n; i += kObsTile) out[i] = sj[i];
    // the self terms: k = 3 observation + component
    outer_sum(3 * i0, 3 * (i0 + 32), [&](int k, int e) {
        const int i = k / 3;
        return i < n ? sj[24 * i + k + 3 * e] : 0.0;
    }, red[warp][1]);
    __syncthreads();
    if (t < 90) {
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < kObsTile / 32; ++w) v += red[w][t / 45][t % 45];
        part[90L * blockIdx.x + t] = v;
    }
}

// One warp per camera: U = sum of the camera's tile partials, column norms
// s = sqrt(diag U), scaled block U/(s s) less the scaled self terms, written as a
// full 9 x 9 block (column-major, 81 per camera). J <- J diag(1/s) skips s == 0
// (ScaledSparseMatrix.cpp:352-356).
__global__ void __launch_bounds__(128) k_camera_gram_reduce(int num_cams, const int* __restrict__ cam_ptr,
                                                            const double* __restrict__ part, double* __restrict__ s_cam,
                                                            double* __restrict__ is_cam, double* __restrict__ U,
                                                            double* __restrict__ zero_record) {
    __shared__ double sh[4][90];
    if (blockIdx.x == 0 && threadIdx.x < 27) zero_record[threadIdx.x] = 0.0;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cam = blockIdx.x * 4 + w;
    if (cam >= num_cams) return;
    const int k0 = tile_base(cam_ptr, cam), k1 = tile_base(cam_ptr, cam + 1);
    double a[3] = {0.0, 0.0, 0.0};
    for (int k = k0; k < k1; ++k)
#pragma unroll
        for (int q = 0; q < 3; ++q)
            if (32 * q + lane < 90) a[q] += part[90L * k + 32 * q + lane];
    double* u = sh[w];
#pragma unroll
    for (int q = 0; q < 3; ++q)
        if (32 * q + lane < 90) u[32 * q + lane] = a[q];
    __syncwarp();
    if (lane < 9) {
        const double v = sqrt(u[ut9(lane, lane)]);
        s_cam[9L * cam + lane] = v;
        is_cam[9L * cam + lane] = v != 0 ? 1.0 / v : 1.0;
    }
    for (int el = lane; el < 45; el += 32) {
        int j, k;
        ut9_inv(el, j, k);
        const double sj = sqrt(u[ut9(j, j)]), sk = sqrt(u[ut9(k, k)]);
        double v = u[el], self = u[45 + el];
        if (sj != 0) v *= 1.0 / sj, self *= 1.0 / sj;
        if (sk != 0) v *= 1.0 / sk, self *= 1.0 / sk;
        v -= self;
        U[81L * cam + j + 9 * k] = v;
        U[81L * cam + k + 9 * j] = v;
    }
}

void launch_camera_blocks(const SceneDev& s, cudaStream_t st) {
    if (s.num_cams == 0) return;
    prepare_assembly_kernels();
    const unsigned slots = (unsigned)camera_tile_slots(s.num_cams, s.num_obs);
    k_camera_tiles<<<slots, kObsTile, kCamTileSmem, st>>>(s.num_cams, s.J, s.cam_ptr, s.cam_obs, s.obs_pt, s.Mp, s.cam_part,
                                                          s.Q);
    k_camera_gram_reduce<<<(s.num_cams + 3) / 4, 128, 0, st>>>(s.num_cams, s.cam_ptr, s.cam_part, s.s_cam, s.is_cam,
                                                                s.Ucam, s.Q + 27L * s.num_obs);
    count_launch(2);
}

// One thread per point: V_p = sum Jp^T Jp (unscaled) and M_p (3 x 3 upper
// triangular, by columns: 00 | 01 11 | 02 12 22) with M_p M_p^T = V_p^{-1}:
// the block scaled to unit diagonal (s = sqrt(diag), as the reference scales
// it), its Cholesky factor L, M_p = diag(1/s) L^{-T}. The reference inverts the
// scaled block by its adjugate (ScaledSparseMatrix.cpp:219-228) and multiplies
// W V^{-1} W^T; with the factor one record Q = W M per observation gives the
// same product as Q Q^T.
// A singular block (a point seen once, or only along one ray) sets
// ERRBIT_SINGULAR: the scaled block's last pivot, taken in the order that puts the
// larger second pivot first, is at most (64 + n) eps for n observations. In that
// order rounding leaves at most about 16 eps of a zero pivot (200,000 blocks of
// rank two, rows up to 1e-6 from parallel), besides n eps of the block's sums; in
// the fixed order it can leave any size, of either sign, when the first two
// columns are close. 64 eps is where k_point_cov drops an eigenvalue.
__global__ void k_point_blocks(int num_points, const double* __restrict__ J, const int* __restrict__ pt_ptr,
                               const int2* __restrict__ pt_list, const int* __restrict__ cam_obs,
                               double* __restrict__ Vraw, double* __restrict__ Mp, int* err) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= num_points) return;
    double v00 = 0, v01 = 0, v02 = 0, v11 = 0, v12 = 0, v22 = 0;
    const int b = pt_ptr[p];
    int n = pt_ptr[p + 1] - b;
    if (Mp && n > kSchurMaxList) n = 0;  // refused (ERRBIT_SCHUR_CAP): its list was not placed
    for (int i0 = 0; i0 < n; i0 += 4) {  // four records in flight
        int o[4];
        double x[4][3], y[4][3];
#pragma unroll
        for (int q = 0; q < 4; ++q) o[q] = i0 + q < n ? pt_list[b + i0 + q].x : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q) o[q] = o[q] >= 0 ? cam_obs[o[q]] : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            x[q][0] = x[q][1] = x[q][2] = y[q][0] = y[q][1] = y[q][2] = 0.0;
            if (o[q] >= 0) load_pt_rows(J, o[q], x[q], y[q]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            v00 += x[q][0] * x[q][0] + y[q][0] * y[q][0];
            v01 += x[q][0] * x[q][1] + y[q][0] * y[q][1];
            v02 += x[q][0] * x[q][2] + y[q][0] * y[q][2];
            v11 += x[q][1] * x[q][1] + y[q][1] * y[q][1];
            v12 += x[q][1] * x[q][2] + y[q][1] * y[q][2];
            v22 += x[q][2] * x[q][2] + y[q][2] * y[q][2];
        }
    }
    double* V = Vraw + 6L * p;
    V[0] = v00; V[1] = v01; V[2] = v02; V[3] = v11; V[4] = v12; V[5] = v22;
    if (!Mp) return;
    double* o = Mp + 6L * p;
    if (n == 0) {  // unobserved, fixed or refused point: unused
        o[0] = o[1] = o[2] = o[3] = o[4] = o[5] = 0.0;
        return;
    }
    const double s0 = sqrt(v00), s1 = sqrt(v11), s2 = sqrt(v22);
    const double i0 = s0 != 0 ? 1.0 / s0 : 1.0, i1 = s1 != 0 ? 1.0 / s1 : 1.0, i2 = s2 != 0 ? 1.0 / s2 : 1.0;
    // scaled block entries a b c / . e f / . . k
    const double a = v00 * i0 * i0, bb = v01 * i0 * i1, c = v02 * i0 * i2;
    const double e = v11 * i1 * i1, f = v12 * i1 * i2, k = v22 * i2 * i2;
    const double r0 = 1.0 / sqrt(a), l10 = bb * r0, l20 = c * r0;
    {
        const double p1 = e - l10 * l10, p2 = k - l20 * l20, g = f - l20 * l10;
        const double top = fmax(p1, p2), least = (64.0 + n) * 2.220446049250313e-16;
        // the last pivot min(p1, p2) - g^2 / top > least (false for a NaN)
        if (!(top > least && fma(fmin(p1, p2), top, -(g * g)) > least * top)) atomicOr(err, ERRBIT_SINGULAR);
    }
    const double r1 = 1.0 / sqrt(e - l10 * l10), l21 = (f - l20 * l10) * r1;
    const double r2 = 1.0 / sqrt(k - l20 * l20 - l21 * l21);
    o[0] = r0 * i0;
    o[1] = -l10 * r0 * r1 * i0;
    o[2] = r1 * i1;
    o[3] = (l10 * l21 * r1 - l20) * r0 * r2 * i0;
    o[4] = -l21 * r1 * r2 * i1;
    o[5] = r2 * i2;
}

void launch_point_blocks(const SceneDev& s, cudaStream_t st) {
    if (s.num_points == 0) return;
    k_point_blocks<<<(s.num_points + 127) / 128, 128, 0, st>>>(s.num_points, s.J, s.pt_ptr, s.pt_list, s.cam_obs, s.Vraw,
                                                               s.Mp, s.err);
    count_launch();
}

void prepare_assembly_kernels() {
    prepare_schur_columns();
    static std::atomic<unsigned long long> attr{0};
    once_per_device(attr, [] {
        return cudaFuncSetAttribute(k_camera_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCamTileSmem) ==
                   cudaSuccess &&
               cudaFuncSetAttribute(k_index_place, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(int) * kIndexWarps * kIndexCams) == cudaSuccess;
    });
}

// Unscaled blocks for the J^T J export: U (9x9 per camera, column-major
// inside a (9C x 9C) dense buffer is too large, so U is written per camera as
// 81 values) and W_o per observation (27 values, row-major 9x3).
__global__ void __launch_bounds__(128) k_camera_blocks_raw(int num_cams, const double* __restrict__ J,
                                                           const int* __restrict__ cam_ptr,
                                                           const int* __restrict__ cam_obs,
                                                           double* __restrict__ U) {
    int cam = blockIdx.x * 4 + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    if (cam >= num_cams) return;
    double acc[45];
#pragma unroll
    for (int t = 0; t < 45; ++t) acc[t] = 0.0;
    for (int i = cam_ptr[cam] + lane; i < cam_ptr[cam + 1]; i += 32) {
        double r0[9], r1[9];
        load_cam_rows(J, cam_obs[i], r0, r1);
#pragma unroll
        for (int j = 0; j < 9; ++j)
#pragma unroll
            for (int k = j; k < 9; ++k) acc[ut9(j, k)] += r0[j] * r0[k] + r1[j] * r1[k];
    }
#pragma unroll
    for (int t = 0; t < 45; ++t) acc[t] = warp_sum(acc[t]);
#pragma unroll
    for (int j = 0; j < 9; ++j)
#pragma unroll
        for (int k = j; k < 9; ++k)
            if (lane == ut9(j, k) || lane + 32 == ut9(j, k)) {
                U[81L * cam + 9 * j + k] = acc[ut9(j, k)];
                U[81L * cam + 9 * k + j] = acc[ut9(j, k)];
            }
}

__global__ void k_obs_blocks_raw(int num_obs, const double* __restrict__ J,
                                 const int* __restrict__ obs_cam, const int* __restrict__ obs_pt,
                                 double* __restrict__ W) {
    int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= num_obs) return;
    if (obs_cam[o] < 0 || obs_pt[o] < 0) return;
    double r0[9], r1[9], a[3], b[3];
    load_cam_rows(J, o, r0, r1);
    load_pt_rows(J, o, a, b);
#pragma unroll
    for (int j = 0; j < 9; ++j)
#pragma unroll
        for (int k = 0; k < 3; ++k) W[27L * o + 3 * j + k] = r0[j] * a[k] + r1[j] * b[k];
}

void launch_unscaled_blocks(const SceneDev& s, double* U, double* W, cudaStream_t st) {
    if (s.num_cams > 0) {
        k_camera_blocks_raw<<<(s.num_cams + 3) / 4, 128, 0, st>>>(s.num_cams, s.J, s.cam_ptr,
                                                                  s.cam_obs, U);
        count_launch();
    }
    if (s.num_obs > 0) {
        k_obs_blocks_raw<<<(s.num_obs + 127) / 128, 128, 0, st>>>(s.num_obs, s.J, s.obs_cam,
                                                                  s.obs_pt, W);
        count_launch();
    }
}

}  // namespace unc
