// dense.cu - FP64 dense kernels for the inverse of the camera Schur
// complement (sm_100a):
//   * gemm_f64      : C = alpha*A*B + beta*C on DMMA (mma.sync m8n8k4 f64),
//                     4-stage cp.async pipeline of 16-deep K tiles, optional fused max|C| for the
//                     Taylor stop rule (ScaledDenseMatrix.cpp:207-216,314-353),
//                     lower-tile and triangular-operand (k range per tile) modes.
//   * spd_inverse   : SPD inverse by recursive Cholesky that forms T = L^{-1}
//                     on the way, then A^{-1} = T^T T; every step is a GEMM above
//                     the blocks that the tile tasks (dag.cu) take
//                     (replaces dgetrf+dgetri in SDM::inv, ScaledDenseMatrix.cpp:232-279).
//   * shift/equilibrate, un-equilibrate, axpy (iZupdate, compute.cpp:64-71),
//     camera output with the reference's (a + b/2) quirk (compute.cpp:168-183).
#include <algorithm>

#include "chol_leaf.cuh"
#include "internal.h"

namespace unc {

// ------------------------------------------------------------------------
// GEMM
// ------------------------------------------------------------------------
namespace {
// Output tile 2W x 2W by four warps of W x W (fragments of the 8 x 8 DMMA
// result), k stages of 16, three CTAs per SM. The FP64 pipe bounds the kernel
// (one DMMA is 16 cycles of a quarter SM), so what counts is that some warp
// always has one to issue: three independent CTAs cover each other's barriers
// and fragment loads. W = 32; W = 16 where 64 x 64 tiles are fewer than the SMs
// (a tile's time is its k range on one SM's FP64 pipe, so smaller tiles finish
// four times sooner).
constexpr int BK = 16, STAGES = 4, GEMM_THREADS = 128, GEMM_CTAS = 3;
template <int W>
struct GemmTile {
    static constexpr int B = 2 * W, F = W / 8;
    // Shared-memory operand tiles. Operands contiguous along m (n): rows of k, pitch
    // B + 4 doubles; a thread reads two neighbouring m (n) of one k as 16 bytes.
    // Operands contiguous along k: rows of m (n), pitch 18. Both pitches make the
    // fragment reads conflict-free (rows 2 g of a group at 8 g words).
    static constexpr int LDM = B + 4, LDK = BK + 2;
    static_assert((2 * LDM) % 32 == 8 && (4 * LDK) % 32 == 8, "conflict-free fragment rows");
    static constexpr int OP_STAGE = B * LDK > BK * LDM ? B * LDK : BK * LDM;  // doubles of one operand tile
    static constexpr size_t SMEM = sizeof(double) * 2 * STAGES * OP_STAGE;
    static constexpr int COPIES = B * BK / 2 / GEMM_THREADS;  // 16-byte copies per thread and operand tile
};

// 16-byte asynchronous copy of `bytes` (0, 8 or 16) valid bytes, the rest zero
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int bytes) {
    unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// Accumulation. By default the products accumulate in the MMA's own C
// operand over the whole k range: one rounding per k step at the size of the
// running sum. With GEMM_SHORT_ACC they accumulate there over 32 steps of k
// (two stages), starting from zero, and those partial sums are added to the
// running sums: k / 32 roundings at that size. The SPD inverse's last Cholesky
// pivots (~lambda, formed by cancellation from O(1) entries) set the inverse's
// largest, gauge, components, so the products that feed pivots
// (L21 = A21 T11^T and A22 -= L21 L21^T) take it. A partial sum is added when
// its registers are needed again, one k step of other fragments later, so that
// no addition waits for an MMA in flight (n = 6144: 32.1 TFLOP/s; 25.5 with
// partial sums of 8 added at once).
__device__ __forceinline__ void dmma0(double& t0, double& t1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%4,%4};\n"
                 : "=d"(t0), "=d"(t1)
                 : "d"(a), "d"(b), "d"(0.0));
}
__device__ __forceinline__ void dmma_acc(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// This thread's copies of one operand's tiles: B rows (m or n) from r0, BK
// steps of k at a time, of an operand with extent R x K. kAlongK: X(r, k) =
// X[k + r ld], else X[r + k ld]. Everything past K is zero. Along m (n) the
// 16-byte pair at R - 1 may include one element past R, which only reaches
// results that are not stored.
template <int W, bool kAlongK>
struct OperandCopy {
    using T = GemmTile<W>;
    const double* src;
    long step, next;   // between this thread's copies of a tile, from one tile to the next
    int dst, rows_ok;  // rows_ok: bit q set when copy q's row exists
    int k;             // k of the first copy in the next tile

    __device__ __forceinline__ OperandCopy(const double* X, long ld, int R, int r0, int kt, int tid) {
        rows_ok = 0;
        if (kAlongK) {
            const int r = tid / (BK / 2);
            k = kt * BK + (tid % (BK / 2)) * 2;
            src = X + k + (long)(r0 + r) * ld;
            step = (long)(GEMM_THREADS / (BK / 2)) * ld;
            next = BK;
            dst = r * T::LDK + (tid % (BK / 2)) * 2;
#pragma unroll
            for (int q = 0; q < T::COPIES; ++q) rows_ok |= (r0 + r + q * (GEMM_THREADS / (BK / 2)) < R) << q;
        } else {
            const int r2 = (tid % W) * 2;
            k = kt * BK + tid / W;
            src = X + (r0 + r2) + (long)k * ld;
            step = (long)(GEMM_THREADS / W) * ld;
            next = (long)BK * ld;
            dst = (tid / W) * T::LDM + r2;
            rows_ok = r0 + r2 < R ? (1 << T::COPIES) - 1 : 0;
        }
    }
    __device__ __forceinline__ void tile(double* sm, const double* __restrict__ X, int K) {
#pragma unroll
        for (int q = 0; q < T::COPIES; ++q) {
            const int left = K - (kAlongK ? k : k + q * (GEMM_THREADS / W));
            const int bytes = !((rows_ok >> q) & 1) || left <= 0 ? 0 : (kAlongK && left == 1 ? 8 : 16);
            cp_async16(sm + dst + q * (kAlongK ? GEMM_THREADS / (BK / 2) * T::LDK : GEMM_THREADS / W * T::LDM),
                       bytes ? src + q * step : X, bytes);
        }
        src += next;
        k += BK;
    }
};

// The fragments of one operand at k step kk (this thread's k: kk + t).
// Fragment f holds rows 16 (f / 2) + 2 g + f % 2 of the warp's W: a pair of
// fragments reads neighbouring rows.
template <int W, bool kAlongK>
__device__ __forceinline__ void load_fragments(const double* sm, int w0, int kk, int g, int t, double (&f)[W / 8]) {
    using T = GemmTile<W>;
#pragma unroll
    for (int i = 0; i < W / 8; i += 2) {
        const int r = w0 + 8 * i + 2 * g;
        if (kAlongK) {
            f[i] = sm[r * T::LDK + kk + t];
            f[i + 1] = sm[(r + 1) * T::LDK + kk + t];
        } else {
            const double2 v = *reinterpret_cast<const double2*>(sm + (kk + t) * T::LDM + r);
            f[i] = v.x;
            f[i + 1] = v.y;
        }
    }
}

__device__ __forceinline__ double finite_abs(double v) {  // |v|, infinity for a NaN
    const double a = fabs(v);
    return a <= 1.7976931348623157e308 ? a : __longlong_as_double(0x7ff0000000000000LL);
}

// X[0], X[stride] = v0, v1 (one 16-byte store when wide)
__device__ __forceinline__ void store_pair(double* X, double v0, double v1, bool wide) {
    if (wide) {
        *reinterpret_cast<double2*>(X) = make_double2(v0, v1);
    } else {
        X[0] = v0;
        X[1] = v1;
    }
}
}  // namespace

// kTransA: A(m, k) = A[k + m lda]; kTransB: B(k, n) = B[n + k ldb].
template <int W, bool kTransA, bool kTransB, bool kShortAcc>
__global__ void __launch_bounds__(GEMM_THREADS, GEMM_CTAS)
    k_gemm_f64(int M, int N, int K, double alpha, const double* __restrict__ A, long lda,
               const double* __restrict__ B, long ldb, double beta, double* C, long ldc,
               unsigned long long* amax, int mode, double* part, const int* skip) {
    using T = GemmTile<W>;
    constexpr int BM = T::B, BN = T::B, FM = T::F, FN = T::F;
    if (skip && *skip) return;
    // Tile order: groups of kGroup tile rows, each walked column by column, so that
    // the CTAs running together share a few rows of A and columns of B in L2. Where
    // the k range grows with m or n the walk starts at the long end (short tiles last).
    constexpr int kGroup = 16;
    const int gy = (M + BM - 1) / BM, gx = (N + BN - 1) / BN;
    const int band = (int)(blockIdx.x / (unsigned)(kGroup * gx)), in = (int)(blockIdx.x - (unsigned)band * (kGroup * gx));
    const int rows = min(kGroup, gy - band * kGroup);
    int ty = band * kGroup + in % rows, tx = in / rows;
    if (mode & GEMM_KHI_M) ty = gy - 1 - ty;
    if (mode & GEMM_KHI_N) tx = gx - 1 - tx;
    const int m0 = ty * BM, n0 = tx * BN;
    // GEMM_LOWER: tiles strictly above the diagonal of C are skipped (SYRK-style update)
    if ((mode & GEMM_LOWER) && n0 > m0 + BM - 1) return;
    extern __shared__ __align__(16) double smem[];
    double* As = smem;
    double* Bs = smem + STAGES * T::OP_STAGE;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp & 1) * W, wn = (warp >> 1) * W;
    const int g = lane >> 2, t = lane & 3;
    const bool wact = (m0 + wm < M) && (n0 + wn < N);
    // triangular operands: the k range of this tile outside which a product term is zero
    int kbeg = 0, kend = K;
    if (mode & GEMM_KLO_M) kbeg = max(kbeg, m0);
    if (mode & GEMM_KLO_N) kbeg = max(kbeg, n0);
    if (mode & GEMM_KHI_M) kend = min(kend, m0 + BM);
    if (mode & GEMM_KHI_N) kend = min(kend, n0 + BN);
    int kt0 = kbeg / BK;
    int KT = kend > kbeg ? (kend + BK - 1) / BK - kt0 : 0;  // k tiles of this output tile
    if (gridDim.y > 1) {  // split-K: a contiguous share of the k tiles, partial sums to part
        const int chunk = (KT + gridDim.y - 1) / gridDim.y;
        const int b0 = min(KT, (int)blockIdx.y * chunk);
        KT = min(KT, b0 + chunk) - b0;
        kt0 += b0;
    }

    double acc[FM][FN][2], p[FM][FN][2];
#pragma unroll
    for (int i = 0; i < FM; ++i)
#pragma unroll
        for (int j = 0; j < FN; ++j) acc[i][j][0] = acc[i][j][1] = p[i][j][0] = p[i][j][1] = 0.0;

    OperandCopy<W, kTransA> copy_a(A, lda, M, m0, kt0, tid);
    OperandCopy<W, !kTransB> copy_b(B, ldb, N, n0, kt0, tid);
    auto load_stage = [&](int s) {
        copy_a.tile(As + s * T::OP_STAGE, A, K);
        copy_b.tile(Bs + s * T::OP_STAGE, B, K);
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < KT) load_stage(s);
        cp_async_commit();
    }
    constexpr int kUnroll = kShortAcc ? 2 : 1;  // a partial sum spans two stages
    auto stage = [&](int kt, bool opens) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        if (kt + STAGES - 1 < KT) load_stage((kt + STAGES - 1) % STAGES);
        cp_async_commit();
        if (!wact) return;  // this warp's sub-tile lies outside C
        const double* as = As + (kt % STAGES) * T::OP_STAGE;
        const double* bs = Bs + (kt % STAGES) * T::OP_STAGE;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            double af[FM], bf[FN];
            load_fragments<W, kTransA>(as, wm, kk, g, t, af);
            load_fragments<W, !kTransB>(bs, wn, kk, g, t, bf);
#pragma unroll
            for (int i = 0; i < FM; ++i)
#pragma unroll
                for (int j = 0; j < FN; ++j) {
                    if (!kShortAcc) {
                        dmma_acc(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
                    } else if (kk == 0 && opens) {  // a new partial sum; the finished one is added
                        acc[i][j][0] += p[i][j][0];
                        acc[i][j][1] += p[i][j][1];
                        dmma0(p[i][j][0], p[i][j][1], af[i], bf[j]);
                    } else {
                        dmma_acc(p[i][j][0], p[i][j][1], af[i], bf[j]);
                    }
                }
        }
    };
    for (int kt = 0; kt < KT; kt += kUnroll) {
        stage(kt, true);
        if (kUnroll == 2 && kt + 1 < KT) stage(kt + 1, false);
    }
    cp_async_wait<0>();
    if (kShortAcc) {
#pragma unroll
        for (int i = 0; i < FM; ++i)
#pragma unroll
            for (int j = 0; j < FN; ++j) {
                acc[i][j][0] += p[i][j][0];
                acc[i][j][1] += p[i][j][1];
            }
    }

    if (part) {  // raw partial tile of split blockIdx.y (M x N slab, leading dimension M)
        double* P = part + (size_t)blockIdx.y * M * N;
#pragma unroll
        for (int i = 0; i < FM; ++i) {
            const int row = m0 + wm + 16 * (i / 2) + 2 * g + i % 2;
#pragma unroll
            for (int j = 0; j < FN; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int col = n0 + wn + 16 * (j / 2) + 2 * (2 * t + h) + j % 2;
                    if (row < M && col < N) P[row + (size_t)col * M] = acc[i][j][h];
                }
        }
        return;
    }

    // each 2 x 2 group of fragment elements (rows r, r + 1, columns c, c + 1)
    const bool wide = ((reinterpret_cast<uintptr_t>(C) | (uintptr_t)(ldc * 8)) & 15) == 0;
    const bool mirror = (mode & GEMM_MIRROR) != 0;
    double mx = 0.0;
#pragma unroll
    for (int i = 0; i < FM; i += 2)
#pragma unroll
        for (int j = 0; j < FN; j += 2)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = m0 + wm + 8 * i + 2 * g, c = n0 + wn + 8 * j + 2 * (2 * t + h);
                double v[2][2];  // [row][column]
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        const bool in_c = r + a < M && c + b < N && (!mirror || r + a >= c + b);
                        v[a][b] = alpha * acc[i + a][j + b][h];
                        if (in_c && beta != 0.0) v[a][b] += beta * C[(r + a) + (long)(c + b) * ldc];
                        if (in_c) mx = fmax(mx, finite_abs(v[a][b]));
                    }
                if (r + 1 < M && c + 1 < N && (!mirror || r > c + 1)) {  // the whole group, strictly below the diagonal
#pragma unroll
                    for (int b = 0; b < 2; ++b) store_pair(C + r + (long)(c + b) * ldc, v[0][b], v[1][b], wide);
                    if (mirror) {
#pragma unroll
                        for (int a = 0; a < 2; ++a) store_pair(C + c + (long)(r + a) * ldc, v[a][0], v[a][1], wide);
                    }
                } else {
#pragma unroll
                    for (int a = 0; a < 2; ++a)
#pragma unroll
                        for (int b = 0; b < 2; ++b)
                            if (r + a < M && c + b < N && (!mirror || r + a >= c + b)) {
                                C[(r + a) + (long)(c + b) * ldc] = v[a][b];
                                if (mirror && r + a > c + b) C[(c + b) + (long)(r + a) * ldc] = v[a][b];
                            }
                }
            }
    if (amax) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, d));
        if (lane == 0) atomicMax(amax, (unsigned long long)__double_as_longlong(mx));
    }
}

// C = alpha * sum_s part[s] + beta * C over the tiles the GEMM computed
// (tiles of b x b), the splits summed in a fixed order (deterministic),
// max|C| folded into amax.
__global__ void k_splitk_reduce(int M, int N, int splits, const double* __restrict__ part, double alpha,
                                double beta, double* C, long ldc, unsigned long long* amax, int mode, int b,
                                const int* skip) {
    if (skip && *skip) return;
    const long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
    double mx = 0.0;
    if (idx < (long)M * N) {
        const int col = (int)(idx / M), row = (int)(idx - (long)col * M);
        if (!((mode & GEMM_LOWER) && col / b > row / b) &&
            !((mode & GEMM_MIRROR) && row < col)) {
            double v = 0.0;
            for (int s = 0; s < splits; ++s) v += part[(size_t)s * M * N + idx];
            double* c = C + row + (long)col * ldc;
            v *= alpha;
            if (beta != 0.0) v += beta * *c;
            *c = v;
            if ((mode & GEMM_MIRROR) && row > col) C[col + (long)row * ldc] = v;
            const double av = fabs(v);
            mx = av <= 1.7976931348623157e308 ? av : __longlong_as_double(0x7ff0000000000000LL);
        }
    }
    if (amax) {
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, d));
        if (lane == 0 && mx > 0.0) atomicMax(amax, (unsigned long long)__double_as_longlong(mx));
    }
}

namespace {
int active_tiles(int M, int N, int b, int mode) {
    const int gy = (M + b - 1) / b, gx = (N + b - 1) / b;
    if (!(mode & GEMM_LOWER)) return gy * gx;
    int tiles = 0;
    for (int y = 0; y < gy; ++y) tiles += std::min(gx, y + 1);
    return tiles;
}

template <int W, bool kTransA, bool kTransB, bool kShortAcc>
bool gemm_smem() {
    return cudaFuncSetAttribute(k_gemm_f64<W, kTransA, kTransB, kShortAcc>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GemmTile<W>::SMEM) == cudaSuccess;
}

template <int W>
void gemm_attr() {
    static std::atomic<unsigned long long> attr{0};
    once_per_device(attr, [] {
        return gemm_smem<W, false, false, false>() && gemm_smem<W, false, true, false>() &&
               gemm_smem<W, false, true, true>() && gemm_smem<W, true, false, false>();
    });
}

template <int W>
void launch_gemm(int M, int N, int K, double alpha, const double* A, int lda, const double* B, int ldb, double beta,
                 double* C, int ldc, unsigned long long* amax, int mode, cudaStream_t st, double* ws,
                 size_t ws_doubles, const int* skip) {
    gemm_attr<W>();
    // split-K when the output has too few tiles to fill the SMs: each split
    // keeps at least kMinSplitTiles k tiles, the partial slabs fit in ws
    constexpr int B_ = GemmTile<W>::B;
    const int tiles = active_tiles(M, N, B_, mode);
    constexpr int kMinSplitTiles = 6, kMaxSplits = 16;
    const int slots = device_sms() * GEMM_CTAS;
    int splits = 1;
    const int kt = (K + BK - 1) / BK;
    if (ws && tiles > 0 && tiles < slots && kt >= 2 * kMinSplitTiles) {
        splits = std::min(std::min(slots / tiles, kt / kMinSplitTiles), kMaxSplits);
        const size_t slab = (size_t)M * N;
        while (splits > 1 && (size_t)splits * slab > ws_doubles) --splits;
    }
    double* part = splits > 1 ? ws : nullptr;
    const dim3 grid((unsigned)((M + B_ - 1) / B_) * (unsigned)((N + B_ - 1) / B_), splits);
    // GEMM_SHORT_ACC comes with GEMM_TRANS_B, GEMM_TRANS_A without it
    const auto kern = (mode & GEMM_TRANS_A)      ? k_gemm_f64<W, true, false, false>
                      : !(mode & GEMM_TRANS_B)   ? k_gemm_f64<W, false, false, false>
                      : (mode & GEMM_SHORT_ACC) ? k_gemm_f64<W, false, true, true>
                                                : k_gemm_f64<W, false, true, false>;
    kern<<<grid, GEMM_THREADS, GemmTile<W>::SMEM, st>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, amax, mode, part,
                                                        skip);
    count_launch();
    if (part) {
        const long total = (long)M * N;
        k_splitk_reduce<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(M, N, splits, part, alpha, beta, C, ldc,
                                                                          amax, mode, B_, skip);
        count_launch();
    }
}
}  // namespace

void gemm_f64_mode(int M, int N, int K, double alpha, const double* A, int lda, const double* B, int ldb,
                   double beta, double* C, int ldc, unsigned long long* amax, int mode, cudaStream_t st,
                   double* ws, size_t ws_doubles, const int* skip) {
    if (M <= 0 || N <= 0) return;
    if (active_tiles(M, N, GemmTile<32>::B, mode) < device_sms())
        launch_gemm<16>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, amax, mode, st, ws, ws_doubles, skip);
    else
        launch_gemm<32>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, amax, mode, st, ws, ws_doubles, skip);
}

void gemm_f64(int M, int N, int K, double alpha, const double* A, int lda, const double* B, int ldb,
              double beta, double* C, int ldc, unsigned long long* amax, cudaStream_t st) {
    gemm_f64_mode(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, amax, 0, st);
}

// ------------------------------------------------------------------------
// SPD inverse: recursive Cholesky A = L L^T that forms T = L^{-1} on the
// way, then A^{-1} = T^T T
// ------------------------------------------------------------------------
__global__ void __launch_bounds__(LEAF_THREADS) k_chol_leaf(const double* __restrict__ A, long lda, int k0,
                                                            int kb, double* T, long ldt, int* err) {
    extern __shared__ __align__(16) double lsm[];
    chol_leaf_tile(A, lda, k0, kb, T, ldt, err, lsm);
}

void prepare_dense_kernels() {
    gemm_attr<32>();
    gemm_attr<16>();
    static std::atomic<unsigned long long> attr{0};
    once_per_device(attr, [] {
        return cudaFuncSetAttribute(k_chol_leaf, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LEAF_SMEM) ==
               cudaSuccess;
    });
}

namespace {

// Where the recursion splits [r0, r1): the first half a multiple of 64.
int chol_split(int r0, int r1) {
    const int m = r0 + (((r1 - r0) / 2 + NB - 1) / NB) * NB;
    return m >= r1 ? r1 - NB : m;
}

// Factor A[r0:r1, r0:r1] (already updated by the earlier panels) and write
// T[r0:r1, r0:r1] = L^{-1}. With the split [r0, m) [m, r1):
//   L21 = A21 T11^T                 (into W; T11^T upper triangular)
//   A22 -= L21 L21^T                (lower tiles)
//   X   = L21 T11                   (into the A21 slot; T11 lower triangular)
//   recurse on A22 -> T22
//   T21 = -T22 X                    (T22 lower triangular)
// Every product is a GEMM whose k loop skips the zero triangle of its
// triangular operand, so the whole recursion costs n^3 / 3 + n^3 / 3 flops.
// Blocks that the tile tasks take (up to n = 3584) end the recursion: down to
// single leaves each 64 rows cost a leaf and five small dependent launches
// (n = 5401: 5.5 of 13.8 ms), as tasks one diagonal task of their chain.
int chol_rec(double* A, int lda, const SpdScratch& s, size_t wsd, int r0, int r1, int* err, cudaStream_t st) {
    const int n = r1 - r0;
    double* T = s.T;
    if (s.state && spd_tasks_apply(n)) {
        const long at = r0 + (long)r0 * lda;
        return chol_inverse_tasks(A + at, n, lda, T + at, nullptr, s.state, err, st, s.max_ctas);
    }
    if (n <= NB) {
        prepare_dense_kernels();
        k_chol_leaf<<<1, LEAF_THREADS, LEAF_SMEM, st>>>(A, lda, r0, n, T, lda, err);
        count_launch();
        return UNC_OK;
    }
    const int m = chol_split(r0, r1);
    const int h1 = m - r0, h2 = r1 - m;
    if (int r = chol_rec(A, lda, s, wsd, r0, m, err, st)) return r;
    double* A21 = A + m + (long)r0 * lda;
    const double* T11 = T + r0 + (long)r0 * lda;
    gemm_f64_mode(h2, h1, h1, 1.0, A21, lda, T11, lda, 0.0, s.W, lda, nullptr,
                  GEMM_TRANS_B | GEMM_KHI_N | GEMM_SHORT_ACC, st, s.ws, wsd);
    gemm_f64_mode(h2, h2, h1, -1.0, s.W, lda, s.W, lda, 1.0, A + m + (long)m * lda, lda, nullptr,
                  GEMM_TRANS_B | GEMM_LOWER | GEMM_SHORT_ACC, st, s.ws, wsd);
    gemm_f64_mode(h2, h1, h1, 1.0, s.W, lda, T11, lda, 0.0, A21, lda, nullptr, GEMM_KLO_N, st, s.ws, wsd);
    if (int r = chol_rec(A, lda, s, wsd, m, r1, err, st)) return r;
    gemm_f64_mode(h2, h1, h2, -1.0, T + m + (long)m * lda, lda, A21, lda, 0.0, T + m + (long)r0 * lda, lda,
                  nullptr, GEMM_KHI_M, st, s.ws, wsd);
    return UNC_OK;
}

int prepare_rec(int r0, int r1) {
    if (spd_tasks_apply(r1 - r0)) return spd_tasks_prepare(r1 - r0, false);
    const int m = chol_split(r0, r1);
    if (int r = prepare_rec(r0, m)) return r;
    return prepare_rec(m, r1);
}
}  // namespace

int spd_prepare(int n) { return spd_tasks_apply(n) ? spd_tasks_prepare(n, true) : prepare_rec(0, n); }

int chol_lower_inverse(double* A, int n, int lda, const SpdScratch& s, int* err, cudaStream_t st) {
    return chol_rec(A, lda, s, (size_t)n * lda, 0, n, err, st);
}

int spd_inverse(double* A, int n, int lda, double shift, double* e, const SpdScratch& s, double* Y, int* err,
                cudaStream_t st) {
    launch_shift_equilibrate(A, n, lda, shift, e, err, st);
    if (s.state && spd_tasks_apply(n)) {
        if (int r = chol_inverse_tasks(A, n, lda, s.T, s.W, s.state, err, st, s.max_ctas, s.poll_limit, s.skip_task,
                                       s.max_grid))
            return r;
        launch_unequilibrate_from(s.W, A, n, lda, e, Y, st);
        return UNC_OK;
    }
    if (int r = chol_lower_inverse(A, n, lda, s, err, st)) return r;
    // A^{-1} = T^T T: lower tiles, k >= the tile's first row (T lower triangular), written in both triangles
    gemm_f64_mode(n, n, n, 1.0, s.T, lda, s.T, lda, 0.0, A, lda, nullptr,
                  GEMM_LOWER | GEMM_KLO_M | GEMM_TRANS_A | GEMM_MIRROR, st);
    launch_unequilibrate(A, n, lda, e, Y, st);
    return UNC_OK;
}

// ------------------------------------------------------------------------
// elementwise helpers
// ------------------------------------------------------------------------
__device__ __forceinline__ void shift_diag_one(double* A, int i, long lda, double lambda, double* e, int* err) {
    double d = A[i + i * lda] + lambda;
    A[i + i * lda] = d;
    if (!(d > 0.0 && isfinite(d))) {
        atomicOr(err, ERRBIT_SINGULAR);
        e[i] = 1.0;
    } else {
        e[i] = 1.0 / sqrt(d);
    }
}

__global__ void k_shift_diag_scale(double* A, int n, long lda, double lambda, double* e, int* err) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    shift_diag_one(A, i, lda, lambda, e, err);
}

// Element-wise launches over an n x n matrix: blockIdx.y = first column, kScaleRows rows
// per block (no division per element).
constexpr int kScaleThreads = 256, kScaleRows = 4 * kScaleThreads;
dim3 scale_grid(int n) { return dim3((unsigned)((n + kScaleRows - 1) / kScaleRows), (unsigned)std::min(n, 65535)); }

// The rows r0 .. of column c: X(r, c) = S(r, c) e_r e_c (and Y the same), from row `first` on.
__device__ __forceinline__ void scale_column(const double* S, double* X, int n, long ld, int c, int r0, int first,
                                             const double* __restrict__ e, double* Y) {
    const double ec = e[c];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int r = r0 + (int)threadIdx.x + u * kScaleThreads;
        if (r < n && r >= first) {
            const double v = S[r + c * ld] * e[r] * ec;
            X[r + c * ld] = v;
            if (Y) Y[r + c * ld] = v;
        }
    }
}

// lower: the lower triangle only (all that a Cholesky factorisation reads)
__global__ void __launch_bounds__(kScaleThreads)
    k_scale_sym(const double* S, double* X, int n, long ld, const double* __restrict__ e, double* Y, int lower) {
    for (int c = blockIdx.y; c < n; c += gridDim.y)
        scale_column(S, X, n, ld, c, blockIdx.x * kScaleRows, lower ? c : 0, e, Y);
}

static void launch_scale(const double* S, double* X, int n, int lda, const double* e, double* Y, bool lower,
                         cudaStream_t st) {
    k_scale_sym<<<scale_grid(n), kScaleThreads, 0, st>>>(S, X, n, lda, e, Y, lower ? 1 : 0);
    count_launch();
}

void launch_shift_equilibrate(double* A, int n, int lda, double lambda, double* e, int* err,
                              cudaStream_t st) {
    k_shift_diag_scale<<<(n + 255) / 256, 256, 0, st>>>(A, n, lda, lambda, e, err);
    count_launch();
    launch_scale(A, A, n, lda, e, nullptr, true, st);
}

void launch_unequilibrate_from(const double* S, double* X, int n, int lda, const double* e, double* Y,
                               cudaStream_t st) {
    launch_scale(S, X, n, lda, e, Y, false, st);
}

void launch_unequilibrate(double* X, int n, int lda, const double* e, double* Y, cudaStream_t st) {
    launch_scale(X, X, n, lda, e, Y, false, st);
}

__global__ void k_te_decide(TeState* s, const unsigned long long* amax_bits, double k) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    if (s->done) return;
    double amax = __longlong_as_double((long long)*amax_bits);
    amax = fmax(amax, 2.2250738585072014e-308);  // absMax starts at DBL_MIN (ScaledDenseMatrix.cpp:208)
    if (!(amax <= 1.7976931348623157e308)) s->bad = 1;
    const double change = fabs(k * amax);
    if (change < 1e-5 || change > s->old_change) {  // compute.cpp:150-152
        s->done = 1;
        return;
    }
    s->old_change = change;
    if (s->iters < 20) s->change[s->iters] = change;
    s->iters += 1;
    s->coef = k;
}

__device__ __forceinline__ void te_init_one(TeState* s) {
    s->done = 0;
    s->bad = 0;
    s->iters = 0;
    s->old_change = 1.7976931348623157e308;  // DBL_MAX (compute.cpp:140)
    s->coef = 0.0;
    for (int i = 0; i < 20; ++i) s->change[i] = 0.0;
    for (int i = 0; i < 20; ++i) s->c[i] = 0.0;
    for (int i = 0; i < 8; ++i) s->skip[i] = 0;
}

__global__ void k_te_init(TeState* s, unsigned long long* dmax) {
    if (dmax && threadIdx.x < 24) dmax[threadIdx.x] = 0ULL;
    if (threadIdx.x == 0) te_init_one(s);
}

// ---- grouped forms over the dense stages of many matrices (a batch) ----
// Block b of an element-wise launch belongs to job m with blk[m] <= b < blk[m + 1].
__device__ __forceinline__ int job_of_block(const long* __restrict__ blk, int njobs, long b) {
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (blk[mid] <= b) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__global__ void k_shift_diag_scale_grouped(const DenseJob* __restrict__ jobs, int njobs, const long* __restrict__ blk) {
    const int m = job_of_block(blk, njobs, blockIdx.x);
    const DenseJob& j = jobs[m];
    const long i = (blockIdx.x - blk[m]) * (long)blockDim.x + threadIdx.x;
    if (i < j.n) shift_diag_one(j.Z, (int)i, j.ld, j.lambda, j.e, j.err);
}

// Element-wise over kScaleRows x kScaleCols pieces: block b - blk[m] of job m.
constexpr int kScaleCols = 8;
__host__ __device__ constexpr long scale_blocks(int n) {
    return (long)((n + kScaleRows - 1) / kScaleRows) * ((n + kScaleCols - 1) / kScaleCols);
}
__global__ void __launch_bounds__(kScaleThreads)
    k_scale_sym_grouped(const DenseJob* __restrict__ jobs, int njobs, const long* __restrict__ blk, int back) {
    const int m = job_of_block(blk, njobs, blockIdx.x);
    const DenseJob& j = jobs[m];
    const int rows = (j.n + kScaleRows - 1) / kScaleRows, b = (int)(blockIdx.x - blk[m]);
    for (int c = b / rows * kScaleCols; c < min(j.n, (b / rows + 1) * kScaleCols); ++c)
        scale_column(back ? j.add : j.Z, j.Z, j.n, j.ld, c, b % rows * kScaleRows, back ? 0 : c, j.e, nullptr);
}

__global__ void k_te_init_grouped(const DenseJob* __restrict__ jobs, int njobs) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < njobs) te_init_one(jobs[m].te);
}

void launch_shift_equilibrate_grouped(const DenseJob* d_jobs, int njobs, const long* d_blk_rows, long nblk_rows,
                                      const long* d_blk_elems, long nblk_elems, cudaStream_t st) {
    if (njobs <= 0) return;
    k_shift_diag_scale_grouped<<<(unsigned)nblk_rows, 256, 0, st>>>(d_jobs, njobs, d_blk_rows);
    k_scale_sym_grouped<<<(unsigned)nblk_elems, kScaleThreads, 0, st>>>(d_jobs, njobs, d_blk_elems, 0);
    count_launch(2);
}

void launch_unequilibrate_grouped(const DenseJob* d_jobs, int njobs, const long* d_blk_elems, long nblk_elems,
                                  cudaStream_t st) {
    if (njobs <= 0) return;
    k_scale_sym_grouped<<<(unsigned)nblk_elems, kScaleThreads, 0, st>>>(d_jobs, njobs, d_blk_elems, 1);
    count_launch();
}

long scale_blocks_grouped(int n) { return scale_blocks(n); }

void launch_te_init_grouped(const DenseJob* d_jobs, int njobs, cudaStream_t st) {
    if (njobs <= 0) return;
    k_te_init_grouped<<<(njobs + 127) / 128, 128, 0, st>>>(d_jobs, njobs);
    count_launch();
}

void launch_te_init(TeState* s, unsigned long long* dmax, cudaStream_t st) {
    k_te_init<<<1, 32, 0, st>>>(s, dmax);
    count_launch();
}

void launch_te_decide(TeState* s, const unsigned long long* amax, double k, cudaStream_t st) {
    k_te_decide<<<1, 32, 0, st>>>(s, amax, k);
    count_launch();
}

__global__ void k_axpy_te(double* Y, const double* __restrict__ X, const TeState* s, int n, long ld) {
    if (s->done) return;
    const double k = s->coef;
    long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
    long total = (long)n * n;
    if (idx >= total) return;
    int c = (int)(idx / n), r = (int)(idx - (long)c * n);
    long o = r + c * ld;
    Y[o] = Y[o] + k * X[o];
}

void launch_axpy_te(double* Y, const double* X, const TeState* s, int n, int ld, cudaStream_t st) {
    long total = (long)n * n;
    k_axpy_te<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(Y, X, s, n, ld);
    count_launch();
}

// Camera output: for camera c and j <= k in its block,
//   camUnc = (iZ(j,k) + iZ(k,j)/2) * d_j * d_k,  d = 1/s   (compute.cpp:176)
// plus the unscaled 9x9 covariance used by the point stage (compute.cpp:435):
//   sig(j,k) = iZ(j,k) * d_j * d_k.
__global__ void k_camera_output(const double* __restrict__ iZ, long ldz,
                                const double* __restrict__ s_cam, int num_cams, double* cam_unc,
                                double* sig) {
    int c = blockIdx.x;
    int e = threadIdx.x;  // 0..80
    if (c >= num_cams || e >= 81) return;
    int j = e / 9, k = e - j * 9;
    long r = 9L * c + j, q = 9L * c + k;
    // s_cam == nullptr: no column scaling (the SVD path, removeScaleJ4Z with d = NULL)
    double dj = s_cam ? 1.0 / s_cam[r] : 1.0, dk = s_cam ? 1.0 / s_cam[q] : 1.0;
    double a = iZ[r + q * ldz], b = iZ[q + r * ldz];
    if (sig) sig[81L * c + e] = a * dj * dk;
    if (k >= j) {
        int t = j * 9 - (j * (j - 1)) / 2 + (k - j);
        cam_unc[45L * c + t] = (a + b / 2) * dj * dk;
    }
}

void launch_camera_output(const double* iZ, int ldz, const double* s_cam, int num_cams,
                          double* cam_unc, double* sig, cudaStream_t st) {
    if (num_cams == 0) return;
    k_camera_output<<<num_cams, 96, 0, st>>>(iZ, ldz, s_cam, num_cams, cam_unc, sig);
    count_launch();
}

}  // namespace unc
