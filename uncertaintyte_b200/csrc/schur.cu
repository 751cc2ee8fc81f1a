// schur.cu - the camera Schur complement Z = U - W V^-1 W^T (compute.cpp:108-118),
// one camera column per CTA, without a global pair list.
//
// With Q_o = W_o M_p, M_p M_p^T = V_p^-1 (k_point_blocks, k_camera_tiles),
//   Z(ca, cb) = U(ca, cb) - S_ca (sum of Q_o Q_o'^T) S_cb
// over the points seen by both cameras, o the observation of the point by camera
// ca and o' by cb, S the inverse column norms. The CTA of camera cb forms the
// blocks ca <= cb of column cb and writes each one twice, in place (upper
// triangle) and transposed (Z(cb, ca)), so Z comes out exactly symmetric:
//  1. the observations of cb (consecutive positions) are taken in chunks. A
//     point's list is ordered by camera, so an observation's partners are the
//     entries before its own; they are copied into shared memory, one list
//     entry per thread;
//  2. the partner cameras get slots (ascending camera); a bit mask per slot
//     marks the chunk's observations with a partner in that camera, so the
//     set bits walk the terms of one block in a fixed order;
//  3. one warp per slot sums its block, four terms (k = 12) per step, on the FP64
//     tensor cores: the leading 8 x 8 part by DMMA, the ninth row and column by
//     ordinary multiply-adds on the operands already loaded. A load instruction
//     covers the rows of one or two records (216 bytes each), where a thread per
//     row of a record made each touch thirty cache lines: the record loads bound
//     the kernel. The block is stored (subtracted from U on the diagonal, read
//     back and updated for the second and later chunks). U comes with the self
//     terms Q_o' Q_o'^T of the diagonal block already subtracted
//     (k_camera_tiles); only a camera that sees a point twice adds to it here.
// Scenes with few cameras split every column over several CTAs (camera ca's
// block to CTA (cb - ca) mod parts, in every chunk), so that the grid covers
// the SMs.
// No floating-point atomics, no device-to-host round trip: the result is
// bitwise repeatable and the stage can be captured in a graph. A camera that
// observes a point more than once gives more than one term per (slot,
// observation): a run of neighbouring entries, since the lists are ordered by
// camera. A chunk that has such a run expands it where the terms are staged, so
// the work is the number of terms whatever the multiplicities.
#include "internal.h"

namespace unc {
namespace {

constexpr int kSzThreads = 256;       // 8 warps, two CTAs per SM (up to about 3000 cameras)
constexpr int kSzWarps = kSzThreads / 32;
constexpr int kSzChunk = 2048;        // owner observations per chunk, at most
constexpr int kSzParts = 8192;        // partner entries per chunk, at most
constexpr int kSzMaskWords = 6144;    // run-mask words (also the entries' owners and the camera scan)
constexpr int kSzPad = 16;            // terms past the end of a run that its steps read
constexpr int kSzSegCap = 256 - kSzPad;  // run entries staged per warp at a time
constexpr unsigned short kNoSlot = 0xFFFF;

static_assert(kSzMaskWords >= kSchurMaxCams, "the camera scan reuses the mask words");
static_assert(kSzMaskWords * 2 >= kSzParts, "the entries' owners (16-bit) reuse the mask words");
static_assert(kSzWarps * (kSzSegCap + kSzPad) * 2 >= kSzChunk, "the point-list starts reuse the run buffers");
static_assert(kSzParts <= 65536 && kSzChunk <= 65536, "owners are 16-bit");
static_assert(kSchurMaxCams < kNoSlot, "slot ids are 16-bit");

struct SzShared {
    int* off;             // [kSzChunk + 1] partner-entry offsets of the chunk's observations
    int* part_o;          // [kSzParts] partner positions
    unsigned short* part_c;  // [kSzParts] partner cameras
    unsigned* mask;       // [kSzMaskWords] slot x word run masks; camera scan buffer before
    unsigned short* slot_of;      // [C] slot of a camera, kNoSlot when none
    unsigned short* cam_of_slot;  // [C]
    int* tmp;             // [kSzWarps + 4] scan scratch and broadcast words
    uint2* runbuf;        // [kSzWarps][kSzSegCap + kSzPad] staged terms (partner, owner), one buffer per warp
    int* sb;              // [kSzChunk] start of each observation's partners (aliases runbuf)
    unsigned short* seg;  // [kSzParts] observation of each entry (aliases mask)
};

// Shared-memory layout (byte offsets; every array starts 16-byte aligned).
struct SzOffsets {
    size_t mask, off, part_o, tmp, runbuf, part_c, slot_of, cam_of_slot, total;
};
__host__ __device__ constexpr size_t sz_align(size_t x) { return (x + 15) & ~size_t(15); }
__host__ __device__ inline SzOffsets sz_offsets(int C) {
    SzOffsets o{};
    o.mask = 0;
    o.off = sz_align(o.mask + sizeof(unsigned) * kSzMaskWords);
    o.part_o = sz_align(o.off + sizeof(int) * (kSzChunk + 1));
    o.tmp = sz_align(o.part_o + sizeof(int) * kSzParts);
    o.runbuf = sz_align(o.tmp + sizeof(int) * (kSzWarps + 4));
    o.part_c = sz_align(o.runbuf + sizeof(uint2) * kSzWarps * (kSzSegCap + kSzPad));
    o.slot_of = sz_align(o.part_c + sizeof(unsigned short) * kSzParts);
    o.cam_of_slot = sz_align(o.slot_of + sizeof(unsigned short) * (size_t)C);
    o.total = sz_align(o.cam_of_slot + sizeof(unsigned short) * (size_t)C);
    return o;
}

__device__ __forceinline__ SzShared sz_layout(char* base, int C) {
    const SzOffsets o = sz_offsets(C);
    SzShared s;
    s.mask = reinterpret_cast<unsigned*>(base + o.mask);
    s.off = reinterpret_cast<int*>(base + o.off);
    s.part_o = reinterpret_cast<int*>(base + o.part_o);
    s.tmp = reinterpret_cast<int*>(base + o.tmp);
    s.runbuf = reinterpret_cast<uint2*>(base + o.runbuf);
    s.part_c = reinterpret_cast<unsigned short*>(base + o.part_c);
    s.slot_of = reinterpret_cast<unsigned short*>(base + o.slot_of);
    s.cam_of_slot = reinterpret_cast<unsigned short*>(base + o.cam_of_slot);
    s.sb = reinterpret_cast<int*>(s.runbuf);
    s.seg = reinterpret_cast<unsigned short*>(s.mask);
    return s;
}

// In-place exclusive scan of a[0, n) over the block; returns the total.
__device__ int sz_scan(int* a, int n, int* tmp) {
    const int per = (n + kSzThreads - 1) / kSzThreads;
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
#pragma unroll
    for (int q = 0; q < kSzWarps; ++q) {
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

// The sum of Q_P Q_O^T over the terms of a run, by one warp: lane (g, t) holds
// C(g, 2t), C(g, 2t + 1) in c, and its share (its k) of C(8, g), C(g, 8) and
// C(8, 8) in row, col, corner. Four terms are k = 12: three DMMA steps, lane t's
// k of step s being 4 s + t (component k % 3 of term k / 3). A term is the two
// records' positions; terms past the end of a run name the zero record, so that a
// load is one address and no test. The loads' latency bounds a run: two steps are
// in flight while one is summed (200 cameras, 60 terms per block: the kernel
// 230 -> 202 us with the tests gone, the second step ahead and the self terms summed
// where the records are made).
struct SzSum {
    int g, t, q[3];
    const double *at[3], *at8[3];  // per step: the lane's element of row g and of row 8 of record 0
    double c[2] = {0.0, 0.0}, row = 0.0, col = 0.0, corner = 0.0;

    __device__ SzSum(int lane, const double* Q) : g(lane >> 2), t(lane & 3) {
#pragma unroll
        for (int s = 0; s < 3; ++s) {
            const int k = 4 * s + t;
            q[s] = k / 3;
            at[s] = Q + 3 * g + k % 3;
            at8[s] = Q + 24 + k % 3;
        }
    }
    template <class F>
    __device__ void load(int e0, F&& term, double (&a)[3], double (&b)[3], double (&a8)[3], double (&b8)[3]) const {
#pragma unroll
        for (int s = 0; s < 3; ++s) {
            const uint2 po = term(e0 + q[s]);
            a[s] = __ldg(at[s] + 27L * po.x);
            b[s] = __ldg(at[s] + 27L * po.y);
            a8[s] = __ldg(at8[s] + 27L * po.x);
            b8[s] = __ldg(at8[s] + 27L * po.y);
        }
    }
    __device__ void add(const double (&a)[3], const double (&b)[3], const double (&a8)[3], const double (&b8)[3]) {
#pragma unroll
        for (int s = 0; s < 3; ++s) {
            asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                         : "+d"(c[0]), "+d"(c[1])
                         : "d"(a[s]), "d"(b[s]));
            row = fma(a8[s], b[s], row);
            col = fma(a[s], b8[s], col);
            corner = fma(a8[s], b8[s], corner);
        }
    }
    // terms 0 .. n - 1 (term(e) answers up to e < n + kSzPad)
    template <class F>
    __device__ void run(int n, F&& term) {
        double a[3][3], b[3][3], a8[3][3], b8[3][3];
        load(0, term, a[0], b[0], a8[0], b8[0]);
        load(4, term, a[1], b[1], a8[1], b8[1]);
        for (int e = 0; e < n; e += 12) {
            load(e + 8, term, a[2], b[2], a8[2], b8[2]);
            add(a[0], b[0], a8[0], b8[0]);
            if (e + 4 >= n) break;
            load(e + 12, term, a[0], b[0], a8[0], b8[0]);
            add(a[1], b[1], a8[1], b8[1]);
            if (e + 8 >= n) break;
            load(e + 16, term, a[1], b[1], a8[1], b8[1]);
            add(a[2], b[2], a8[2], b8[2]);
        }
    }
    // the shares of row 8 and column 8 added over the k lanes
    __device__ void finish() {
#pragma unroll
        for (int d = 1; d < 4; d <<= 1) {
            row += __shfl_xor_sync(0xffffffffu, row, d);
            col += __shfl_xor_sync(0xffffffffu, col, d);
            corner += __shfl_xor_sync(0xffffffffu, corner, d);
        }
    }
    // f(r, c, value) over this lane's elements of the 9 x 9 block
    template <class F>
    __device__ void elements(F&& f) const {
        f(g, 2 * t, c[0]);
        f(g, 2 * t + 1, c[1]);
        if (t == 0) f(8, g, row);
        if (t == 1) f(g, 8, col);
        if (g == 0 && t == 2) f(8, 8, corner);
    }
};

// The first partner of camera c among observation j's (one exists; ordered by camera).
__device__ __forceinline__ int sz_first(const SzShared& sh, int j, int c) {
    int t = sh.off[j], end = sh.off[j + 1];
    while (end - t > 16) {
        const int m = (t + end) >> 1;
        if (sh.part_c[m] < c) t = m + 1; else end = m + 1;
    }
    while (t < end && sh.part_c[t] != c) ++t;
    return t;
}

// The end of the run of equal cameras that starts at entry t of observation j.
__device__ __forceinline__ int sz_run_end(const SzShared& sh, int j, int t) {
    int lo = t + 1, hi = sh.off[j + 1];
    while (lo < hi) {
        const int m = (lo + hi) >> 1;
        if (sh.part_c[m] == sh.part_c[t]) lo = m + 1; else hi = m;
    }
    return lo;
}

// One block: the terms of slot s (camera ca <= cb) over the chunk, then the block
// stored in both triangles (the diagonal: U minus the terms, both ways round). The
// run is staged in the warp's buffer segment by segment. repeats: some observation
// of the chunk has several partners in a camera; the segments are at most 32
// observations then, one per lane, and a segment whose terms do not fit is staged
// again for the next of them, so that only its start and `skip` stay in registers
// over the sum (200 cameras: the kernel 208 us without repeats, 210 so, 218 with the
// lanes' entries kept). first: the position of the chunk's observation 0; zero: the
// zero record's position. Warp-level.
__device__ void sz_block(const SzShared& sh, uint2* buf, int s, int ca, int cb, int first, int zero, int W, bool repeats,
                         bool store, const double* __restrict__ Q, const double* __restrict__ is_cam,
                         const double* __restrict__ U, double* Z, long ldz) {
    const int lane = threadIdx.x & 31;
    const unsigned* mk = sh.mask + (size_t)s * W;
    SzSum sum(lane, Q);
    const uint2 none = make_uint2((unsigned)zero, (unsigned)zero);
    for (int wi = 0, skip = 0; wi < W;) {
        // stage a segment of the run: the marked observations j in order (32
        // mask words per step, a prefix scan of their bit counts gives every
        // lane its place), then each entry's partner, one entry per lane
        const int cap = repeats ? 32 : kSzSegCap;
        int nseg = 0, next = wi;
        while (next < W && nseg <= cap - 32) {
            const int nw = min(32, W - next);
            const unsigned word = lane < nw ? mk[next + lane] : 0u;
            const int c = __popc(word);
            int incl = c;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += y;
            }
            // whole words that fit (a prefix of the lanes: incl grows with the lane)
            const int take = __popc(__ballot_sync(0xffffffffu, lane < nw && nseg + incl <= cap));
            if (lane < take) {
                int pos = nseg + incl - c;
                for (unsigned bb = word; bb; bb &= bb - 1u) buf[pos++].y = 32u * (next + lane) + (__ffs(bb) - 1);
            }
            nseg += __shfl_sync(0xffffffffu, incl, take - 1);
            next += take;
        }
        __syncwarp();
        if (!repeats) {
            for (int e = lane; e < nseg; e += 32) {
                const int j = (int)buf[e].y;
                buf[e] = make_uint2((unsigned)sh.part_o[sz_first(sh, j, ca)], (unsigned)(first + j));
            }
        } else {
            int j = 0, t = 0, n = 0;  // this lane's observation and its entries [t, t + n) of camera ca
            if (lane < nseg) {
                j = (int)buf[lane].y;
                t = sz_first(sh, j, ca);
                n = sz_run_end(sh, j, t) - t;
            }
            int incl = n;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += y;
            }
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            __syncwarp();
            nseg = min(kSzSegCap, total - skip);  // the segment's terms [skip, skip + nseg)
            for (int x = skip + lane; x - lane < skip + nseg; x += 32) {
                int from = 0;  // the lane whose entries hold term x: as many lanes end at or before it
#pragma unroll
                for (int d = 16; d > 0; d >>= 1)
                    if (__shfl_sync(0xffffffffu, incl, from + d - 1) <= x) from += d;
                const int at = __shfl_sync(0xffffffffu, t + n - incl, from) + x;
                const int owner = first + __shfl_sync(0xffffffffu, j, from);
                if (x < skip + nseg) buf[x - skip] = make_uint2((unsigned)sh.part_o[at], (unsigned)owner);
            }
            skip += nseg;
            if (skip < total) next = wi;
            else skip = 0;
        }
        wi = next;
        if (lane < kSzPad) buf[nseg + lane] = none;
        __syncwarp();
        sum.run(nseg, [&](int e) { return buf[e]; });
        __syncwarp();  // the buffer is refilled next
    }
    sum.finish();
    sum.elements([&](int r, int q, double v) {
        const long row = 9L * ca + r, col = 9L * cb + q;
        if (ca < cb) {
            v *= __ldg(is_cam + row) * __ldg(is_cam + col);
            double* up = Z + row + col * ldz;
            v = store ? -v : *up - v;
            *up = v;
            Z[col + row * ldz] = v;
        }
    });
    if (ca != cb) return;
    // the diagonal block, kept symmetric: both orders of a pair of observations of cb
    double* blk = reinterpret_cast<double*>(buf);  // 81 of the buffer's doubles
    __syncwarp();
    sum.elements([&](int r, int q, double v) { blk[9 * r + q] = v; });
    __syncwarp();
    for (int e = lane; e < 81; e += 32) {
        const int r = e % 9, q = e / 9;
        if (r > q) continue;
        const long row = 9L * cb + r, col = 9L * cb + q;
        double v = blk[9 * r + q] + blk[9 * q + r];
        v *= __ldg(is_cam + row) * __ldg(is_cam + col);
        double* up = Z + row + col * ldz;
        v = (store ? U[81L * cb + e] : *up) - v;
        *up = v;
        Z[col + row * ldz] = v;
    }
    __syncwarp();
}

// The run masks of the chunk's entries; true when some camera has two entries at one
// observation. Where the lists are long (one of more than 32 entries on average), the
// block's threads share each of them. Block-level.
__device__ bool sz_masks(const SzShared& sh, int len, int K, int W) {
    for (int k = threadIdx.x; k < K * W; k += kSzThreads) sh.mask[k] = 0u;
    __syncthreads();
    const bool shared_list = sh.off[len] > 32 * len;
    int more = 0;
    for (int j = shared_list ? 0 : threadIdx.x; j < len; j += shared_list ? 1 : kSzThreads) {
        const int t0 = sh.off[j], t1 = sh.off[j + 1], step = shared_list ? kSzThreads : 1;
        for (int t = t0 + (shared_list ? threadIdx.x : 0); t < t1; t += step) {
            const unsigned short c = sh.part_c[t];
            atomicOr(sh.mask + (size_t)sh.slot_of[c] * W + (j >> 5), 1u << (j & 31));
            more |= t > t0 && sh.part_c[t - 1] == c;
        }
    }
    return __syncthreads_or(more) != 0;
}

__global__ void __launch_bounds__(kSzThreads, 2)
    k_schur_columns(int C, const int* __restrict__ cam_ptr, const int2* __restrict__ pt_list,
                    const int2* __restrict__ pos_list, const double* __restrict__ Q, const double* __restrict__ is_cam,
                    const double* __restrict__ U, double* Z, long ldz, int parts, int zero,
                    const int* __restrict__ err) {
    if (*err & ERRBIT_SCHUR_CAP) return;
    extern __shared__ __align__(16) char sz_smem[];
    const SzShared sh = sz_layout(sz_smem, C);
    const int cb = C - 1 - (int)(blockIdx.x / parts);  // the most partners (cameras <= cb) first
    const int part = (int)(blockIdx.x % parts);        // this CTA's share of the column's slots
    const int base = cam_ptr[cb], n = cam_ptr[cb + 1] - base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (n == 0) {  // no observations: the diagonal block is U alone
        if (part == 0 && tid < 81) Z[9L * cb + tid % 9 + (9L * cb + tid / 9) * ldz] = U[81L * cb + tid];
        return;
    }
    for (int c = tid; c <= cb; c += kSzThreads) sh.slot_of[c] = kNoSlot;
    __syncthreads();
    bool first_chunk = true;
    // skip: entries of observation j0 that earlier chunks took (an observation with more
    // partners than a chunk holds is taken in pieces)
    for (int j0 = 0, skip = 0; j0 < n;) {
        const int jn = min(n, j0 + kSzChunk) - j0;
        for (int j = tid; j < jn; j += kSzThreads) {
            int2 l = pos_list[base + j0 + j];
            if (j == 0) l = make_int2(l.x + skip, l.y - skip);
            sh.sb[j] = l.x;
            sh.off[j] = l.y;
        }
        __syncthreads();
        const int total = sz_scan(sh.off, jn, sh.tmp);
        if (tid == 0) {
            sh.off[jn] = total;
            int lo = 0, hi = jn;  // the longest prefix whose lists fit
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (sh.off[mid] <= kSzParts) lo = mid; else hi = mid - 1;
            }
            sh.tmp[kSzWarps] = lo;
        }
        __syncthreads();
        int len = sh.tmp[kSzWarps];
        const bool piece = len == 0;  // one observation's first kSzParts entries
        if (piece) {
            len = 1;
            if (tid == 0) sh.off[1] = kSzParts;
            __syncthreads();
        }
        // every entry: its observation (then its partner and camera, in parallel)
        const int E = sh.off[len];
        if (E > 32 * len) {  // long lists: the block's threads share each
            for (int j = 0; j < len; ++j)
                for (int i = sh.off[j] + tid; i < sh.off[j + 1]; i += kSzThreads) sh.seg[i] = (unsigned short)j;
        } else {
            for (int j = tid; j < len; j += kSzThreads)
                for (int i = sh.off[j]; i < sh.off[j + 1]; ++i) sh.seg[i] = (unsigned short)j;
        }
        __syncthreads();
        for (int i = tid; i < E; i += 4 * kSzThreads) {  // four entries per thread in flight
            int2 l[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int k = i + q * kSzThreads;
                int j = 0;
                if (k < E) j = sh.seg[k];
                l[q] = k < E ? pt_list[sh.sb[j] + (k - sh.off[j])] : make_int2(0, 0);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int k = i + q * kSzThreads;
                if (k < E) {
                    sh.part_o[k] = l[q].x;
                    sh.part_c[k] = (unsigned short)l[q].y;
                    sh.slot_of[l[q].y] = 0;
                }
            }
        }
        if (tid == 0) sh.slot_of[cb] = 0;  // the diagonal block always has a slot (U)
        __syncthreads();
        int K = 0, W = 0;
        for (;;) {
            int* scan = reinterpret_cast<int*>(sh.mask);
            for (int c = tid; c <= cb; c += kSzThreads) scan[c] = sh.slot_of[c] != kNoSlot;
            __syncthreads();
            K = sz_scan(scan, cb + 1, sh.tmp);
            W = (len + 31) >> 5;
            if (K * W <= kSzMaskWords) break;
            // too many slots for the masks: the first half of the chunk, its cameras again
            for (int c = tid; c <= cb; c += kSzThreads) sh.slot_of[c] = kNoSlot;
            len = (len + 1) >> 1;
            __syncthreads();
            for (int i = tid; i < sh.off[len]; i += kSzThreads) sh.slot_of[sh.part_c[i]] = 0;
            if (tid == 0) sh.slot_of[cb] = 0;
            __syncthreads();
        }
        {
            const int* scan = reinterpret_cast<const int*>(sh.mask);
            for (int c = tid; c <= cb; c += kSzThreads)
                if (sh.slot_of[c] != kNoSlot) {
                    const int s = scan[c];
                    sh.slot_of[c] = (unsigned short)s;
                    sh.cam_of_slot[s] = (unsigned short)c;
                }
        }
        __syncthreads();
        if (tid == 0) sh.tmp[kSzWarps + 1] = 0;  // slot cursor: warps take slots as they finish
        const bool repeats = sz_masks(sh, len, K, W);
        for (;;) {  // this CTA's blocks: cameras ca with (cb - ca) mod parts == part, the same in
                    // every chunk (slot numbers are not), so no block is updated by two CTAs
            int q = 0;
            if (lane == 0) q = atomicAdd(sh.tmp + kSzWarps + 1, 1);
            q = __shfl_sync(0xffffffffu, q, 0);
            const int s = K - 1 - q;
            if (s < 0) break;
            const int ca = sh.cam_of_slot[s];
            if ((cb - ca) % parts != part) continue;
            sz_block(sh, sh.runbuf + warp * (kSzSegCap + kSzPad), s, ca, cb, base + j0, zero, W, repeats, first_chunk, Q,
                     is_cam, U, Z, ldz);
        }
        __syncthreads();
        for (int s = tid; s < K; s += kSzThreads) sh.slot_of[sh.cam_of_slot[s]] = kNoSlot;
        __syncthreads();
        first_chunk = false;
        if (piece) {
            skip += kSzParts;  // the rest of this observation's entries next
        } else {
            j0 += len;
            skip = 0;
        }
    }
}

}  // namespace

size_t schur_columns_smem(int C) { return sz_offsets(C).total; }

void prepare_schur_columns() {
    static std::atomic<unsigned long long> attr{0};
    once_per_device(attr, [] {
        return cudaFuncSetAttribute(k_schur_columns, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)schur_columns_smem(kSchurMaxCams)) == cudaSuccess;
    });
}

int launch_schur_columns(const SceneDev& s, double* Z, int ldz, cudaStream_t st) {
    const int C = s.num_cams;
    if (C == 0) return UNC_OK;
    if (C > kSchurMaxCams) return UNC_ERR_TOO_LARGE;
    const size_t smem = schur_columns_smem(C);
    prepare_schur_columns();
    // few cameras: split every column so that the grid covers about two waves of CTAs (every part
    // stages the column's entries again; whole solve at 200 cameras with 2, 3 and 4 parts: 1475,
    // 1435 and 1458 us)
    const int parts = std::max(1, std::min(8, (4 * device_sms() + C - 1) / C));
    k_schur_columns<<<C * parts, kSzThreads, smem, st>>>(C, s.cam_ptr, s.pt_list, s.pos_list, s.Q, s.is_cam, s.Ucam, Z,
                                                         ldz, parts, s.num_obs, s.err);
    count_launch();
    return UNC_OK;
}

}  // namespace unc
