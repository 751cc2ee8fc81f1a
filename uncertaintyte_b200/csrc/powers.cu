// powers.cu - the Taylor series of teInverse (compute.cpp:141-160) evaluated
// from a few powers of X instead of one product per iteration.
//
// The reference forms add = X^(i+1) by one product per iteration, stops when
// change = |k_i max|add|| falls below 1e-5 or grows (k_i = lambda^i / (i-1)!,
// the 32-bit factorial of compute.cpp:57-62), and sums iZ = X + sum_i k_i add_i.
// Here:
//   * X is SPD, so every power X^j is SPD and its largest |entry| is its
//     largest diagonal entry; diag(X^(a+b))_c is the dot product of column c
//     of X^a and of X^b. From X, X^2, X^3, X^4, X^8, X^12 (and X^16) every
//     j = 2..20 is such a pair, so the stop rule runs on the device from
//     O(N^2) column dot products;
//   * only the 9 x 9 diagonal camera blocks of iZ are read after the series (the
//     camera output, compute.cpp:168-183, and the point stage's block-diagonal
//     camera covariance, compute.cpp:422-441), and the camera blocks of
//     X^(4q + r + 1), q = 1..4, r = 0..3, are products of 9 columns of X^(4q)
//     and of X^(r+1): formed once, they give both the diagonal entries of the
//     stop rule and, with the coefficients that it decides (c_0 = 1, c_i = k_i
//     for the performed iterations and 0 after), the sum.
// Products: X^2, X^3, X^4, X^8, X^12 (X^16 past 15 iterations): 5 for the
// 12..15 iterations of the reference scenes, instead of 13..16. The
// polynomial, its coefficients and the stop decisions are the reference's;
// the results differ from the one-product-per-iteration order at the
// rounding level. Every kernel here has a fixed summation order, so the
// results are bitwise repeatable.
#include <cfloat>

#include "internal.h"

namespace unc {
namespace {

constexpr int kBlkThreads = 256;
constexpr int kBlkPairs = kPowerPairs;

// Element p = r (r + 1) / 2 + s of a lower triangle.
__device__ __forceinline__ void lower_pair(int p, int& r, int& s) {
    r = 0;
    s = p;
    while (s > r) s -= ++r;
}

// The camera's blocks of X^(4q) X^(r+1) for q in [Q0, Q0 + NQ) and r = 0..3,
// lower triangles, into ps.blk; their diagonals, and with Q0 = 1 those of X^2,
// X^3, X^4, into the maxima ps.dmax (over the non-negative values; a non-finite
// one becomes +inf). One CTA per camera: the camera's nine columns of every
// power are streamed through shared memory, kBlkK rows at a time in kBlkStages
// asynchronous stages (reading each power once bounds the kernel; with loads
// straight into registers its latency did: 110 us at n = 1800, 9.0 ms at 18000;
// now 67 us and 4.0 ms, 59 % of the copy bandwidth). Eight warps:
// warp (r, half) multiplies the columns of X^(r+1) with those of the NQ powers over
// every other 8 rows: a DMMA per power for the leading 8 x 8 part, ordinary
// multiply-adds for row 8. A lane's 16-byte read holds the rows k = 8 j + 2 t
// and the next, which go to two DMMA steps.
constexpr int kBlkK = 32, kBlkStages = 4, kBlkStride = kBlkK + 8;  // column stride: conflict-free 16-byte reads
template <int NQ>
constexpr int blk_slots() { return 4 + (NQ == 3 ? 2 : 1); }  // X .. X^4, then the powers that are not X^4
template <int NQ>
constexpr size_t blk_smem() { return sizeof(double) * kBlkStages * blk_slots<NQ>() * 9 * kBlkStride; }

template <int Q0, int NQ>
__device__ __forceinline__ void power_blocks(const PowerSet& ps, int cam, double* sm, double (*red)[4][NQ][kBlkPairs],
                                             double (*dia)[3][9], unsigned long long* top) {
    static_assert((Q0 == 1 && NQ == 3) || (Q0 == 4 && NQ == 1), "X^4, X^8, X^12 or X^16");
    constexpr int kSlots = blk_slots<NQ>(), kStage = kSlots * 9 * kBlkStride;
    const int n = ps.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int r = warp & 3, half = warp >> 2;
    const long ld = ps.ld, c0 = 9L * cam;
    const int stages = (n + kBlkK - 1) / kBlkK;
    auto issue = [&](int s) {
        if (s < stages) {
            double* st = sm + (s % kBlkStages) * kStage;
            for (int q = tid; q < kSlots * 9 * (kBlkK / 2); q += kBlkThreads) {
                const int col = q / (kBlkK / 2), k2 = q % (kBlkK / 2) * 2, slot = col / 9;
                const double* M = ps.M[slot < 4 ? slot : (Q0 == 1 ? slot : 6)];
                const int left = n - (s * kBlkK + k2), bytes = left >= 2 ? 16 : (left == 1 ? 8 : 0);
                const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(st + col * kBlkStride + k2));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst),
                             "l"(bytes ? M + (c0 + col - 9 * slot) * ld + s * kBlkK + k2 : M), "r"(bytes)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    double c[NQ][2], row[NQ], corner[NQ], d[2][2];  // d: diagonals of X X (X^2 X^2 in warp r = 1) and X X^2
#pragma unroll
    for (int q = 0; q < NQ; ++q) c[q][0] = c[q][1] = row[q] = corner[q] = 0.0;
    d[0][0] = d[0][1] = d[1][0] = d[1][1] = 0.0;
#pragma unroll
    for (int s = 0; s < kBlkStages - 1; ++s) issue(s);
    for (int s = 0; s < stages; ++s) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kBlkStages - 2) : "memory");
        __syncthreads();
        issue(s + kBlkStages - 1);
        const double* st = sm + (s % kBlkStages) * kStage;
#pragma unroll
        for (int j = 0; j < kBlkK / 16; ++j) {
            const double* at = st + 8 * (2 * j + half) + 2 * t;
            auto read = [&](int slot, int col) {
                return *reinterpret_cast<const double2*>(at + (9 * slot + col) * kBlkStride);
            };
            const double2 a = read(r, g), a8 = read(r, 8);
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const int slot = Q0 == 1 ? 3 + q : 4;
                const double2 b = read(slot, g), b8 = read(slot, 8);
                asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                             : "+d"(c[q][0]), "+d"(c[q][1])
                             : "d"(a.x), "d"(b.x));
                asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                             : "+d"(c[q][0]), "+d"(c[q][1])
                             : "d"(a.y), "d"(b.y));
                row[q] = fma(a8.y, b.y, fma(a8.x, b.x, row[q]));
                corner[q] = fma(a8.y, b8.y, fma(a8.x, b8.x, corner[q]));
            }
            if (Q0 == 1 && r < 2) {
                d[0][0] = fma(a.y, a.y, fma(a.x, a.x, d[0][0]));
                d[0][1] = fma(a8.y, a8.y, fma(a8.x, a8.x, d[0][1]));
                if (r == 0) {
                    const double2 x = read(1, g), x8 = read(1, 8);
                    d[1][0] = fma(a.y, x.y, fma(a.x, x.x, d[1][0]));
                    d[1][1] = fma(a8.y, x8.y, fma(a8.x, x8.x, d[1][1]));
                }
            }
        }
    }
#pragma unroll
    for (int m = 1; m < 4; m <<= 1) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            row[q] += __shfl_xor_sync(0xffffffffu, row[q], m);
            corner[q] += __shfl_xor_sync(0xffffffffu, corner[q], m);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) d[i][j] += __shfl_xor_sync(0xffffffffu, d[i][j], m);
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        double* out = red[half][r][q];
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (2 * t + h <= g) out[g * (g + 1) / 2 + 2 * t + h] = c[q][h];
        if (t == 0) out[36 + g] = row[q];
        if (lane == 0) out[44] = corner[q];
    }
    if (Q0 == 1 && r < 2 && t == 0) {  // rows of dia: X^2, X^3 (both from warp r = 0), X^4
        dia[half][r == 0 ? 0 : 2][g] = d[0][0];
        if (r == 0) dia[half][1][g] = d[1][0];
        if (g == 0) {
            dia[half][r == 0 ? 0 : 2][8] = d[0][1];
            if (r == 0) dia[half][1][8] = d[1][1];
        }
    }
    if (tid < 32) top[tid] = 0ULL;
    __syncthreads();
    auto fold = [&](int j, double v) {  // a diagonal entry of X^j
        v = v <= DBL_MAX ? fmax(v, 0.0) : __longlong_as_double(0x7ff0000000000000LL);  // NaN -> inf
        atomicMax(top + j, (unsigned long long)__double_as_longlong(v));
    };
    for (int e = tid; e < NQ * 4 * kBlkPairs; e += kBlkThreads) {
        const int p = e % kBlkPairs, rr = e / kBlkPairs % 4, q = e / (4 * kBlkPairs);
        const double v = red[0][rr][q][p] + red[1][rr][q][p];
        ps.blk[((long)cam * 16 + 4 * (Q0 - 1 + q) + rr) * kBlkPairs + p] = v;
        int i, j;
        lower_pair(p, i, j);
        if (i == j) fold(4 * (Q0 + q) + rr + 1, v);
    }
    if (Q0 == 1 && tid < 27) fold(2 + tid / 9, dia[0][tid / 9][tid % 9] + dia[1][tid / 9][tid % 9]);
    __syncthreads();
    constexpr int jlo = Q0 == 1 ? 2 : 4 * Q0 + 1, jhi = 4 * (Q0 + NQ);
    if (tid <= jhi - jlo) atomicMax(ps.dmax + jlo + tid, top[jlo + tid]);
}

template <int Q0, int NQ>
__global__ void __launch_bounds__(kBlkThreads, 2) k_power_blocks(PowerSet ps, const int* skip) {
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[2][4][NQ][kBlkPairs], dia[2][3][9];
    __shared__ unsigned long long top[32];
    if (skip && *skip) return;
    power_blocks<Q0, NQ>(ps, blockIdx.x, sm, red, dia, top);
}

__device__ __forceinline__ int set_of_block(const long* __restrict__ blk, int nsets, long b) {
    int lo = 0, hi = nsets - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (blk[mid] <= b) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// The same over the cameras of many sets: cols holds the sets' column offsets
// (multiples of 9), so set m owns the cameras [cols[m] / 9, cols[m + 1] / 9).
template <int Q0, int NQ>
__global__ void __launch_bounds__(kBlkThreads, 2)
    k_power_blocks_grouped(const PowerSet* __restrict__ sets, int nsets, const long* __restrict__ cols) {
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[2][4][NQ][kBlkPairs], dia[2][3][9];
    __shared__ unsigned long long top[32];
    const int m = set_of_block(cols, nsets, 9L * blockIdx.x);
    const PowerSet ps = sets[m];
    if (Q0 > 1 && ps.te->skip[0]) return;
    power_blocks<Q0, NQ>(ps, (int)(blockIdx.x - cols[m] / 9), sm, red, dia, top);
}

// The reference's stop rule (compute.cpp:145-155) over iterations ilo..ihi.
__device__ __forceinline__ void power_decide_one(TeState* s, const unsigned long long* dmax, const double* k, int ilo,
                                                 int ihi) {
    if (ilo == 1) s->c[0] = 1.0;
    for (int i = ilo; i <= ihi && !s->done; ++i) {
        double amax = __longlong_as_double((long long)dmax[i + 1]);
        amax = fmax(amax, 2.2250738585072014e-308);  // absMax starts at DBL_MIN (ScaledDenseMatrix.cpp:208)
        if (!(amax <= 1.7976931348623157e308)) s->bad = 1;
        const double change = fabs(k[i - 1] * amax);
        if (change < 1e-5 || change > s->old_change) {  // compute.cpp:150-152
            s->done = 1;
            break;
        }
        s->old_change = change;
        if (s->iters < 20) s->change[s->iters] = change;
        s->iters += 1;
        s->c[i] = k[i - 1];
    }
    if (ihi == 15) s->skip[0] = s->done;  // X^16 is needed only past iteration 15
    if (ihi == 19)
        for (int q = 1; q <= 4; ++q) s->skip[q] = s->iters < 4 * q;
}

__global__ void k_power_decide(TeState* s, const unsigned long long* dmax, TaylorCoefs k, int ilo, int ihi) {
    if (threadIdx.x == 0 && blockIdx.x == 0) power_decide_one(s, dmax, k.k, ilo, ihi);
}

__global__ void k_power_decide_grouped(const PowerSet* __restrict__ sets, int nsets, const double* __restrict__ k,
                                       int ilo, int ihi) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < nsets) power_decide_one(sets[m].te, sets[m].dmax, k + 19L * m, ilo, ihi);
}

// The camera's block of iZ = sum_i c_i X^(i+1) and the outputs that read it:
// cam_unc = (iZ(j,k) + iZ(k,j) / 2) d_j d_k, d = 1 / s (compute.cpp:176), and
// the unscaled covariance block sig (compute.cpp:435). One CTA per camera, a
// thread per element of the lower triangle.
__global__ void __launch_bounds__(64) k_power_output(PowerSet ps, const double* __restrict__ s_cam,
                                                     double* __restrict__ cam_unc, double* __restrict__ sig) {
    const int p = threadIdx.x;
    if (p >= kBlkPairs) return;
    const long cam = blockIdx.x, c0 = 9 * cam;
    int r, s;
    lower_pair(p, r, s);
    const double* c = ps.te->c;
    const long at = (c0 + r) + (c0 + s) * ps.ld;
    double v = c[0] * ps.M[0][at];
    v += c[1] * ps.M[1][at];
    v += c[2] * ps.M[2][at];
    v += c[3] * ps.M[3][at];
    for (int q = 1; q <= 4; ++q) {
        if (ps.te->skip[q]) continue;
        const double* b = ps.blk + (cam * 16 + 4 * (q - 1)) * kBlkPairs + p;
        double t = c[4 * q] * b[0];
        t += c[4 * q + 1] * b[kBlkPairs];
        t += c[4 * q + 2] * b[2 * kBlkPairs];
        t += c[4 * q + 3] * b[3 * kBlkPairs];
        v += t;
    }
    const double dr = 1.0 / s_cam[c0 + r], ds = 1.0 / s_cam[c0 + s];
    sig[81 * cam + 9 * r + s] = v * dr * ds;
    sig[81 * cam + 9 * s + r] = v * ds * dr;
    cam_unc[45 * cam + s * 9 - (s * (s - 1)) / 2 + (r - s)] = (v + v / 2) * ds * dr;  // row s, column r
}

}  // namespace

void prepare_power_kernels() {
    static std::atomic<unsigned long long> attr{0};
    once_per_device(attr, [] {
        auto set = [](const void* f, size_t bytes) {
            return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess;
        };
        return set((const void*)k_power_blocks<1, 3>, blk_smem<3>()) && set((const void*)k_power_blocks<4, 1>, blk_smem<1>()) &&
               set((const void*)k_power_blocks_grouped<1, 3>, blk_smem<3>()) &&
               set((const void*)k_power_blocks_grouped<4, 1>, blk_smem<1>());
    });
}

void launch_power_blocks(const PowerSet& ps, bool past_15, const int* skip, cudaStream_t st) {
    if (past_15)
        k_power_blocks<4, 1><<<ps.n / 9, kBlkThreads, blk_smem<1>(), st>>>(ps, skip);
    else
        k_power_blocks<1, 3><<<ps.n / 9, kBlkThreads, blk_smem<3>(), st>>>(ps, skip);
    count_launch();
}

void launch_power_blocks_grouped(const PowerSet* d_sets, int nsets, const long* d_blk_cols, long nblk_cols, bool past_15,
                                 cudaStream_t st) {
    if (nsets <= 0 || nblk_cols < 9) return;
    const unsigned cams = (unsigned)(nblk_cols / 9);
    if (past_15)
        k_power_blocks_grouped<4, 1><<<cams, kBlkThreads, blk_smem<1>(), st>>>(d_sets, nsets, d_blk_cols);
    else
        k_power_blocks_grouped<1, 3><<<cams, kBlkThreads, blk_smem<3>(), st>>>(d_sets, nsets, d_blk_cols);
    count_launch();
}

void launch_power_decide(TeState* te, const unsigned long long* dmax, const TaylorCoefs& k, int ilo, int ihi,
                         cudaStream_t st) {
    k_power_decide<<<1, 32, 0, st>>>(te, dmax, k, ilo, ihi);
    count_launch();
}

void launch_power_decide_grouped(const PowerSet* d_sets, int nsets, const double* d_k, int ilo, int ihi,
                                 cudaStream_t st) {
    if (nsets <= 0) return;
    k_power_decide_grouped<<<(nsets + 127) / 128, 128, 0, st>>>(d_sets, nsets, d_k, ilo, ihi);
    count_launch();
}

void launch_power_output(const PowerSet& ps, const double* s_cam, double* cam_unc, double* sig, cudaStream_t st) {
    k_power_output<<<ps.n / 9, 64, 0, st>>>(ps, s_cam, cam_unc, sig);
    count_launch();
}

}  // namespace unc
