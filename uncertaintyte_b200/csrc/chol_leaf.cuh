// chol_leaf.cuh - the 64 x 64 Cholesky + inverse leaf shared by the recursive
// SPD inverse (dense.cu) and the tile-task inverse (dag.cu).
#pragma once
#include "internal.h"

namespace unc {

constexpr int NB = 64;  // leaf size

// Leaf: Cholesky of the kb x kb (kb <= 64) diagonal block of A at (k0, k0)
// and T_kk = L_kk^{-1}, written as a full kb x kb block of T (zeros above the
// diagonal). One CTA of 256 threads; the block (S) and its inverse (Ts) sit in
// shared memory, column-major with a stride of 68 doubles (fragment reads in
// both orientations and lane = row reads are conflict-free), padded to 64 x 64
// with an identity tail (the factor and inverse of blockdiag(A, I) are
// blockdiag(L, I) and blockdiag(L^-1, I), so every step has fixed shapes).
//
// The leaf is a chain of dependent operations, so everything but that chain
// runs beside it. Four 16-column panels q:
//  (A) warp 0 factors the 16 x 16 diagonal block in registers, two columns per
//      step: with pivot d, e below it and f the next diagonal entry,
//      1/L(p,p) = d^-1/2 and 1/L(p+1,p+1) = (d f - e^2)^-1/2 d^1/2, whose two
//      reciprocal square roots are one call, half of the warp's lanes taking the
//      one and half the other (two calls follow one another: n = 1351 432 us
//      instead of 421), and the next step's d, e, f are formed by every lane from
//      broadcast values (one shuffle latency per step). Lanes 0..15 hold the block's rows, lanes 16..31 the rows of the
//      identity, which the same instructions turn into D_q = L_qq^{-1}.
//  (B) the rows below: X = A_iq D_q^T on the FP64 tensor cores (DMMA);
//  (C) the next diagonal block takes its rank-16 update; the rest of the
//      trailing update and the blocks of T = L^{-1} (block forward
//      substitution: W_ij = sum_k L_ik T_kj in the T_ij slot, T_ij = -D_i W_ij)
//      are done by the other warps during the next panel's (A).
// Non-positive or non-finite pivots set ERRBIT_SINGULAR.
constexpr int LEAF_THREADS = 256;
constexpr int LEAF_LD = NB + 4;
constexpr int LEAF_PW = 16;
constexpr int LEAF_TILE = NB * LEAF_LD;                      // doubles of one 64 x 64 shared tile
constexpr size_t LEAF_SMEM = sizeof(double) * 2 * LEAF_TILE;  // S, Ts

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// Barrier `id` (1..15) over `threads` threads of the block.
__device__ __forceinline__ void named_barrier(int id, int threads) {
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

// c = A B over k = 16 for one 8 x 8 fragment of shared tiles (column-major,
// stride LEAF_LD): A(m, k) = a[k LD + m], B(k, n) = kBT ? b[k LD + n] :
// b[n LD + k]. Lane (g, t) gets C(g, 2t), C(g, 2t + 1).
template <bool kBT>
__device__ __forceinline__ void leaf_mma(const double* a, const double* b, int g, int t, double (&c)[2]) {
    double u[2] = {0.0, 0.0}, v[2] = {0.0, 0.0};  // two chains of two steps
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int k = 4 * h + t;
        dmma(u[0], u[1], a[k * LEAF_LD + g], kBT ? b[k * LEAF_LD + g] : b[g * LEAF_LD + k]);
        dmma(v[0], v[1], a[(8 + k) * LEAF_LD + g], kBT ? b[(8 + k) * LEAF_LD + g] : b[g * LEAF_LD + 8 + k]);
    }
    c[0] = u[0] + v[0];
    c[1] = u[1] + v[1];
}

// The 16 x 16 block (r, c) (in units of 16) of a shared tile.
__device__ __forceinline__ double* leaf_block(double* M, int r, int c) {
    return M + (c * LEAF_LD + r) * LEAF_PW;
}

// Fragment (fi, fj) of the block Cb -= Xi Xj^T.
__device__ __forceinline__ void leaf_update(double* Cb, const double* Xi, const double* Xj, int fi, int fj, int g,
                                            int t) {
    double c[2];
    leaf_mma<true>(Xi + 8 * fi, Xj + 8 * fj, g, t, c);
    double* z = Cb + (8 * fj + 2 * t) * LEAF_LD + 8 * fi + g;
    z[0] -= c[0];
    z[LEAF_LD] -= c[1];
}

// Rows 8 fi .. 8 fi + 7 of the block X <- X D^T, in place (one warp).
__device__ __forceinline__ void leaf_solve(double* X, const double* D, int fi, int g, int t) {
    double c[2][2];
#pragma unroll
    for (int fj = 0; fj < 2; ++fj) leaf_mma<true>(X + 8 * fi, D + 8 * fj, g, t, c[fj]);
    __syncwarp();
#pragma unroll
    for (int fj = 0; fj < 2; ++fj) {
        double* z = X + (8 * fj + 2 * t) * LEAF_LD + 8 * fi + g;
        z[0] = c[fj][0];
        z[LEAF_LD] = c[fj][1];
    }
}

// Fragment (fi, fj) of the block W (+)= L Tb.
__device__ __forceinline__ void leaf_gather(double* W, const double* L, const double* Tb, bool first, int fi, int fj,
                                            int g, int t) {
    double c[2];
    leaf_mma<false>(L + 8 * fi, Tb + 8 * fj * LEAF_LD, g, t, c);
    double* z = W + (8 * fj + 2 * t) * LEAF_LD + 8 * fi + g;
    z[0] = first ? c[0] : z[0] + c[0];
    z[LEAF_LD] = first ? c[1] : z[LEAF_LD] + c[1];
}

// Columns 8 fj .. 8 fj + 7 of the block W <- -D W, in place (one warp).
__device__ __forceinline__ void leaf_finish(double* W, const double* D, int fj, int g, int t) {
    double c[2][2];
#pragma unroll
    for (int fi = 0; fi < 2; ++fi) leaf_mma<false>(D + 8 * fi, W + 8 * fj * LEAF_LD, g, t, c[fi]);
    __syncwarp();
#pragma unroll
    for (int fi = 0; fi < 2; ++fi) {
        double* z = W + (8 * fj + 2 * t) * LEAF_LD + 8 * fi + g;
        z[0] = -c[fi][0];
        z[LEAF_LD] = -c[fi][1];
    }
}

// (A): one warp; the diagonal block Sb becomes L_qq, Db receives L_qq^{-1}.
__device__ __forceinline__ void leaf_panel(double* Sb, double* Db, int lane, int* err) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr double kTiny = 2.2250738585072014e-308, kHuge = 1.7976931348623157e308;  // normal pivots
    double a[LEAF_PW];
#pragma unroll
    for (int j = 0; j < LEAF_PW; ++j)
        a[j] = lane < LEAF_PW ? (j <= lane ? Sb[j * LEAF_LD + lane] : 0.0) : (j == lane - LEAF_PW ? 1.0 : 0.0);
    bool bad = false;
    double d = __shfl_sync(kAll, a[0], 0), e = __shfl_sync(kAll, a[0], 1), f = __shfl_sync(kAll, a[1], 1);
#pragma unroll
    for (int h = 0; h < LEAF_PW / 2; ++h) {
        const int p = 2 * h;
        // the next step's entries before this step's update
        double dn = 0.0, en = 0.0, fn = 0.0;
        if (p + 2 < LEAF_PW) {
            dn = __shfl_sync(kAll, a[p + 2], p + 2);
            en = __shfl_sync(kAll, a[p + 2], p + 3);
            fn = __shfl_sync(kAll, a[p + 3], p + 3);
        }
        const double det = fma(d, f, -(e * e)), r = rsqrt(lane < LEAF_PW ? d : det);
        const double other = __shfl_xor_sync(kAll, r, LEAF_PW);
        const double r0 = lane < LEAF_PW ? r : other, rd = lane < LEAF_PW ? other : r;
        bad |= !(d >= kTiny && det >= kTiny && d <= kHuge && det <= kHuge);
        const double r1 = rd * (d * r0);
        const double x0 = a[p] * r0;
        const double x1 = fma(-x0, e * r0, a[p + 1]) * r1;
        a[p] = x0;
        a[p + 1] = x1;
#pragma unroll
        for (int j = p + 2; j < LEAF_PW; ++j) {
            const double m0 = __shfl_sync(kAll, x0, j), m1 = __shfl_sync(kAll, x1, j);
            a[j] = fma(-x1, m1, fma(-x0, m0, a[j]));
            if (j == p + 2) {
                dn = fma(-m1, m1, fma(-m0, m0, dn));
                e = m0;  // rows p + 2 of the two columns, for the entry below the next pivot
                f = m1;
            }
            if (j == p + 3) {
                en = fma(-m1, f, fma(-m0, e, en));
                fn = fma(-m1, m1, fma(-m0, m0, fn));
            }
        }
        d = dn;
        e = en;
        f = fn;
    }
    if (lane == 0 && bad) atomicOr(err, ERRBIT_SINGULAR);
    double* out = lane < LEAF_PW ? Sb + lane : Db + (lane - LEAF_PW) * LEAF_LD;  // row of L, column of D
    const int step = lane < LEAF_PW ? LEAF_LD : 1;
#pragma unroll
    for (int j = 0; j < LEAF_PW; ++j)
        if (lane >= LEAF_PW || j <= lane) out[j * step] = a[j];
}

// Load phase: the kb x kb diagonal block of A at (k0, k0) into S (lower
// triangle, identity tail). A is read through L2 only (ld.global.cg), so that a
// persistent caller never sees a stale L1 line of a tile another CTA rewrote.
// The caller synchronises.
__device__ __forceinline__ void chol_leaf_load(const double* A, long lda, int k0, int kb, double* S) {
    const int tid = threadIdx.x;
    constexpr int kPer = NB * NB / LEAF_THREADS;
    const int i = tid & (NB - 1);
    double v[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int j = (tid >> 6) + u * (LEAF_THREADS / NB);
        v[u] = (i < kb && j < kb) ? (j <= i ? __ldcg(A + (k0 + i) + (long)(k0 + j) * lda) : 0.0) : (i == j ? 1.0 : 0.0);
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) S[((tid >> 6) + u * (LEAF_THREADS / NB)) * LEAF_LD + i] = v[u];
}

// Factorisation of the block in S (after chol_leaf_load and a barrier), T_kk
// in Ts (lower 16 x 16 blocks, the diagonal ones with zeros above the diagonal)
// and written to T at (k0, k0). One CTA of LEAF_THREADS threads. Warp 4 calls
// beside(q) during panel q, all threads last() after the panels: the caller's own work
// (no block barrier in it).
template <class F, class G>
__device__ __forceinline__ void chol_leaf_factor(int k0, int kb, double* T, long ldt, int* err, double* S, double* Ts,
                                                 F&& beside, G&& last) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    // the warps beside (A): 1, 2, 3, 5, 6, 7 (warp 4 shares warp 0's scheduler and FP64 pipe)
    const int worker = warp < 4 ? warp - 1 : warp - 2;
    constexpr int kWorkers = 6;
    auto S_ = [S](int r, int c) { return leaf_block(S, r, c); };
    auto T_ = [Ts](int r, int c) { return leaf_block(Ts, r, c); };
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
        if (warp == 0) {
            leaf_panel(S_(q, q), T_(q, q), lane, err);
        } else if (warp == 4) {
            beside(q);
        } else if (q > 0) {
            // beside panel q: the updates of panel p = q - 1 that panel q does not need
            const int p = q - 1;
            {
                int item = 0;
                // T_pj = -D_p W_pj, then (after the barrier) W_ij += L_ip T_pj
                for (int j = 0; j < p; ++j)
                    for (int fj = 0; fj < 2; ++fj)
                        if (item++ % kWorkers == worker) leaf_finish(T_(p, j), T_(p, p), fj, g, t);
                for (int i = q; i < 4; ++i)
                    for (int j = q; j <= i; ++j) {
                        if (i == q) continue;  // the diagonal block (q, q) was updated before the panel
                        for (int f = 0; f < 4; ++f)
                            if (item++ % kWorkers == worker)
                                leaf_update(S_(i, j), S_(i, p), S_(j, p), f & 1, f >> 1, g, t);
                    }
                for (int i = q; i < 4; ++i)
                    for (int f = 0; f < 4; ++f)
                        if (item++ % kWorkers == worker)
                            leaf_gather(T_(i, p), S_(i, p), T_(p, p), true, f & 1, f >> 1, g, t);
            }
            named_barrier(1, 32 * kWorkers);
            {
                int item = 0;
                for (int i = q; i < 4; ++i)
                    for (int j = 0; j < p; ++j)
                        for (int f = 0; f < 4; ++f)
                            if (item++ % kWorkers == worker)
                                leaf_gather(T_(i, j), S_(i, p), T_(p, j), false, f & 1, f >> 1, g, t);
            }
        }
        __syncthreads();
        if (q == 3) break;
        // (B): 8-row strips of the blocks below, the next block row first
        for (int s = warp; s < 2 * (3 - q); s += LEAF_THREADS / 32) leaf_solve(S_(q + 1 + s / 2, q), T_(q, q), s & 1, g, t);
        __syncthreads();
        // (C), the next diagonal block's lower fragments
        if (warp < 3) leaf_update(S_(q + 1, q + 1), S_(q + 1, q), S_(q + 1, q), warp > 0, warp > 1, g, t);
        __syncthreads();
    }
    last();
    for (int s = warp; s < 6; s += LEAF_THREADS / 32) leaf_finish(T_(3, s >> 1), T_(3, 3), s & 1, g, t);
    __syncthreads();
    const int i = tid & (NB - 1);
#pragma unroll
    for (int u = 0; u < NB * NB / LEAF_THREADS; ++u) {
        const int j = (tid >> 6) + u * (LEAF_THREADS / NB);
        if (i < kb && j < kb) T[(k0 + i) + (long)(k0 + j) * ldt] = i >= j ? Ts[j * LEAF_LD + i] : 0.0;
    }
}

// The whole leaf: load, barrier, factorisation (lsm: LEAF_SMEM bytes).
__device__ __forceinline__ void chol_leaf_tile(const double* A, long lda, int k0, int kb, double* T, long ldt,
                                               int* err, double* lsm) {
    chol_leaf_load(A, lda, k0, kb, lsm);
    __syncthreads();
    chol_leaf_factor(k0, kb, T, ldt, err, lsm, lsm + LEAF_TILE, [](int) {}, [] {});
}

}  // namespace unc
