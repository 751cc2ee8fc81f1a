// dag.cu - SPD inverse A^{-1} = L^{-T} L^{-1} as a graph of 64 x 64 tile tasks
// run by one persistent kernel (sm_100a), for the moderate sizes where the
// recursive form (dense.cu) is bound by its ~200 dependent launches.
//
// Tiles (i, j), j <= i, of the lower triangle; nt = ceil(n / 64). Tasks:
//   POTRF(k)      T(k,k) = chol(A(k,k))^{-1}                  (the 64 x 64 leaf)
//   TRSM(i,k)     L(i,k) = A(i,k) T(k,k)^T                    (in place in A)
//   UPDATE(i,j,k) A(i,j) -= L(i,k) L(j,k)^T                   (k < j <= i)
//   TACC(i,j,m)   W(i,j) += L(i,m) T(m,j)                     (j <= m < i, in the T(i,j) slot)
//   TFIN(i,j)     T(i,j) = -T(i,i) W(i,j)                     (block forward substitution)
//   PACC(i,j,k)   O(i,j) += T(k,i)^T T(k,j)                   (k >= i >= j; the last term also
//                                                             writes the transposed tile)
// UPDATE, TACC and PACC take 1 to 4 consecutive values of their last index in one
// task (its k field: first value + count << 16): a single one where the chain of
// diagonal tiles or of T's rows waits for it, groups of four elsewhere. A task
// streams its operands in slices of 32 k through three shared-memory stages and
// reads and writes its own tile once, so a group costs its products and not one
// load-compute-store round trip per 64 k.
// POTRF(k) also applies the last update of its tile (from panel k-1) before
// factoring and computes TRSM(k+1,k) after it, so the dependent chain from one
// diagonal tile to the next is one task. The host lists the tasks in a
// topological order that puts each diagonal factorisation right after the
// tasks it waits for (look-ahead).
// CTAs claim tasks from a global cursor in list order, wait (thread 0, with an
// iteration limit) on per-tile counters, run the task with all 256 threads
// and publish its counter. Every dependency of a claimed task was claimed
// earlier by a running CTA that waits only on still earlier tasks, so the
// schedule completes with any number of resident CTAs; updates of one tile
// are applied in a fixed order, so the result is bitwise repeatable. Tile data
// written by other CTAs is read through L2 only (ld.global.cg, cp.async.cg).
// One matrix alone: the CTA that claims POTRF(0) runs every POTRF(k) itself, one
// after the other (run_chain), and the other CTAs pass over those entries. The
// chain bounds the whole inverse at these sizes; kept in one CTA, L(k+1,k) is
// in shared memory when POTRF(k+1) needs it and the next tiles are fetched
// beside the leaf, and the SM's second CTA leaves it the FP64 pipe (it retires
// once a CTA elsewhere takes tasks). The other CTAs' tasks still depend only on
// earlier entries and on the chain. Where none of them is resident to take the
// entries before POTRF(k), the chain's CTA takes those itself while it waits
// (chain_wait), in list order, so that it completes alone as well.
//
// Counters (ints, zeroed before the launch): cursor, abort flag, 1 + the SM of the
// chain, CTAs on other SMs, then per
// lower tile: ver (updates applied to A), lrdy (L final / T(k,k) ready),
// tacc (W accumulations), trdy (T final), pacc (O accumulations).
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "chol_leaf.cuh"
#include "internal.h"

namespace unc {
namespace {

constexpr int TB = NB;                   // tile size (the leaf size)
constexpr int DAG_THREADS = LEAF_THREADS;
constexpr int TLD = LEAF_LD;             // shared tile stride: fragment reads conflict-free in both orientations
// Two CTAs of 256 threads per SM, so that one waits, loads or stores while the
// other computes. Shared memory of a CTA: two operand tiles and the leaf's block
// (whose inverse takes the second operand tile), or the stages of a stream.
constexpr int DAG_CTAS = 2;
constexpr int SLICE = 32, STREAM_STAGES = 3;      // k of a slice
constexpr int SLD = SLICE + 4;                    // stride of a slice of rows (k contiguous)
constexpr int SLOT = TB * SLD > SLICE * TLD ? TB * SLD : SLICE * TLD;  // doubles of one operand's slice
constexpr size_t DAG_SMEM = sizeof(double) * (2 * STREAM_STAGES * SLOT > 3 * LEAF_TILE ? 2 * STREAM_STAGES * SLOT : 3 * LEAF_TILE);
constexpr int MAX_GROUP = 4;                      // consecutive k of a group, at most
constexpr long kDagSpin = 1L << 22;      // polls of one dependency before the kernel gives up
constexpr int kMaxTilesN = 56;           // tasks are used up to n = 56 * 64

enum : int { K_POTRF = 0, K_TRSM = 1, K_UPDATE = 2, K_TACC = 3, K_TFIN = 4, K_PACC = 5 };

__device__ __forceinline__ int tri(int i, int j) { return i * (i + 1) / 2 + j; }

__device__ __forceinline__ int ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// One thread: wait until *flag >= v (or the abort flag is raised / the limit of
// `spin` polls runs out)
__device__ bool wait_ge(const int* flag, int v, const int* abort, long spin) {
    for (long it = 0; it < spin; ++it) {
        if (ld_acquire(flag) >= v) return true;
        if (ld_acquire(abort)) return false;
        __nanosleep(32);
    }
    return false;
}

// One warp: the same for one flag per lane (nullptr: none), polled together. The
// lanes leave together: one lane reads the abort flag and the warp votes on what it
// read (with a read per lane, some could see the flag and leave while the others
// wait for them at the next vote).
__device__ bool wait_all(const int* flag, int v, const int* abort, long spin) {
    const int lane = threadIdx.x & 31;
    for (long it = 0; it < spin; ++it) {
        const bool ok = !flag || ld_acquire(flag) >= v;
        if (__all_sync(0xffffffffu, ok)) return true;
        if (__any_sync(0xffffffffu, lane == 0 && ld_acquire(abort) != 0)) return false;
        __nanosleep(32);
    }
    return false;
}

// Tile X (column-major, leading dimension ld; rows < vr and columns < vc
// valid, the rest zero) into shared memory as sm[c * TLD + r], asynchronously
// and past L1, by `threads` threads; tile_wait() before the barrier that
// publishes it. cols: columns of the tile that are copied.
__device__ __forceinline__ void load_tile(double* sm, const double* X, long ld, int vr, int vc, int tid,
                                          int threads = DAG_THREADS, int cols = TB) {
    for (int q = tid; q < cols * (TB / 2); q += threads) {
        const int c = q >> 5, r2 = (q & 31) * 2;
        const int left = c < vc ? vr - r2 : 0;
        const int bytes = left >= 2 ? 16 : (left == 1 ? 8 : 0);
        const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(sm + c * TLD + r2));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst),
                     "l"(bytes ? X + r2 + (long)c * ld : X), "r"(bytes)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void tile_wait() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// A tile of a matrix: its first element and its valid rows and columns.
struct TileRef {
    const double* p;
    int rows, cols;
};

// acc += A op(B) over k in [kb, ke) (multiples of 4) for this warp's 32 x 16
// block (rows wm.., columns wn..), op(B)(k, n) = B(n, k), whole tiles as left by
// load_tile.
using Acc = double[4][2][2];
__device__ __forceinline__ void tile_mma(const double* As, const double* Bs, int wm, int wn, int g, int t, int kb,
                                         int ke, Acc& acc) {
    for (int kk = kb; kk < ke; kk += 4) {
        double a[4], b[2];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = As[(kk + t) * TLD + wm + 8 * i + g];
#pragma unroll
        for (int j = 0; j < 2; ++j) b[j] = Bs[(kk + t) * TLD + wn + 8 * j + g];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
}

// One operand of a stream: tile(kt) is its tile at k tile kt, of rows x cols
// valid elements. kRows: k runs along the tile's rows, else along its columns.
template <bool kRows>
__device__ __forceinline__ void load_slice(double* sm, const double* X, long ld, int vr, int vc, int half, int tid) {
#pragma unroll
    for (int u = 0; u < TB * SLICE / 2 / DAG_THREADS; ++u) {
        const int q = tid + u * DAG_THREADS;
        const int c = kRows ? q / (SLICE / 2) : q / (TB / 2) + half * SLICE;
        const int r2 = kRows ? (q % (SLICE / 2)) * 2 + half * SLICE : (q % (TB / 2)) * 2;
        const int left = c < vc ? vr - r2 : 0;
        const int bytes = left >= 2 ? 16 : (left == 1 ? 8 : 0);
        double* d = kRows ? sm + c * SLD + (r2 - half * SLICE) : sm + (c - half * SLICE) * TLD + r2;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                         static_cast<unsigned>(__cvta_generic_to_shared(d))),
                     "l"(bytes ? X + r2 + (long)c * ld : X), "r"(bytes)
                     : "memory");
    }
}

// acc += sum over k tiles k0 .. k0 + count - 1 of op(A) op(B): fa(kt), fb(kt)
// give the operands' tiles (pointer, valid rows, valid columns). op(A)(m, k) =
// kRowsA ? A(k, m) : A(m, k), op(B)(k, n) = kRowsB ? B(k, n) : B(n, k). klim:
// this warp's products stop at that k of a tile (a triangular operand).
template <bool kRowsA, bool kRowsB, class FA, class FB>
__device__ __forceinline__ void stream_mma(double* sm, long ld, int k0, int count, FA&& fa, FB&& fb, int wm, int wn,
                                           int g, int t, int klim, int tid, Acc& acc) {
    const int n = 2 * count;
    auto issue = [&](int it) {
        if (it < n) {
            double* st = sm + (it % STREAM_STAGES) * 2 * SLOT;
            const TileRef a = fa(k0 + it / 2), b = fb(k0 + it / 2);
            load_slice<kRowsA>(st, a.p, ld, a.rows, a.cols, it & 1, tid);
            load_slice<kRowsB>(st + SLOT, b.p, ld, b.rows, b.cols, it & 1, tid);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    issue(0);
    issue(1);
    for (int it = 0; it < n; ++it) {
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        issue(it + 2);
        const double* As = sm + (it % STREAM_STAGES) * 2 * SLOT;
        const double* Bs = As + SLOT;
        const int ke = min(SLICE, klim - (it & 1) * SLICE);
#pragma unroll 4
        for (int kk = 0; kk < ke; kk += 4) {
            double a[4], b[2];
            const int k = kk + t;
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = kRowsA ? As[(wm + 8 * i + g) * SLD + k] : As[k * TLD + wm + 8 * i + g];
#pragma unroll
            for (int j = 0; j < 2; ++j) b[j] = kRowsB ? Bs[(wn + 8 * j + g) * SLD + k] : Bs[k * TLD + wn + 8 * j + g];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
        }
    }
}

// f(row, column, element of x) over this thread's elements of the warp's block
// that lie in the vr x vc valid part of the tile.
template <class F>
__device__ __forceinline__ void tile_elements(int vr, int vc, int wm, int wn, int g, int t, Acc& x, F&& f) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = wm + 8 * i + g, c = wn + 8 * j + 2 * t + h;
                if (r < vr && c < vc) f(r, c, x[i][j][h]);
            }
}

// prev = X where valid: issued before the products, so that its latency is
// covered by the operand loads and the products.
__device__ __forceinline__ void load_prev(const double* X, long ld, int vr, int vc, int wm, int wn, int g, int t,
                                          Acc& prev) {
    tile_elements(vr, vc, wm, wn, g, t, prev, [&](int r, int c, double& v) { v = __ldcg(X + r + (long)c * ld); });
}

// X(r, c) = alpha acc + prev for r < vr, c < vc; with Xm, also Xm(c, r) = the
// same value (the transposed tile).
__device__ __forceinline__ void store_tile(double* X, long ld, int vr, int vc, Acc& acc, double alpha, const Acc& prev,
                                           double* Xm, int wm, int wn, int g, int t) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) acc[i][j][h] = fma(alpha, acc[i][j][h], prev[i][j][h]);
    tile_elements(vr, vc, wm, wn, g, t, acc, [&](int r, int c, double& v) {
        X[r + (long)c * ld] = v;
        if (Xm) Xm[c + (long)r * ld] = v;
    });
}

// The n x n matrix of a task: tiles of A, T, O and the counters (laid out as
// described at the top).
struct TaskMatrix {
    double *A, *T, *O;
    int n;
    long ld;
    int *ver, *lrdy, *tacc, *trdy, *pacc;
    int* err;
    int* abort;
    long spin;

    __device__ __forceinline__ TaskMatrix(double* A_, double* T_, double* O_, int n_, long ld_, int* state, int ntri,
                                          int* err_, int* abort_, long spin_)
        : A(A_), T(T_), O(O_), n(n_), ld(ld_), ver(state + 4), lrdy(ver + ntri), tacc(lrdy + ntri), trdy(tacc + ntri),
          pacc(trdy + ntri), err(err_), abort(abort_), spin(spin_) {}
    __device__ __forceinline__ int ext(int b) const { return min(TB, n - TB * b); }
    __device__ __forceinline__ int tiles() const { return (n + TB - 1) / TB; }
    __device__ __forceinline__ double* tile(double* M, int i, int j) const { return M + (long)TB * i + (long)TB * j * ld; }
    // thread 0 only
    __device__ __forceinline__ bool wait(const int* flag, int v) const { return wait_ge(flag, v, abort, spin); }
    __device__ __forceinline__ bool give_up() const {
        atomicOr(err, ERRBIT_TIMEOUT);
        atomicExch(abort, 1);
        return false;
    }
};

// The lower 8 x 8 blocks of a 64 x 64 tile dealt to eight warps, four or five each and
// nine or ten to the two warps of a scheduler (its FP64 pipe takes one DMMA per 16
// cycles; n = 1351: 364 -> 350 us): nibbles 0 and 1 the block rows of slots 0-2 and
// 3-4, nibbles 2-6 the block columns of the slots, nibble 7 whether slot 4 is used.
// Warp 6 repeats its slot 1 as slot 2. Two warps of a scheduler with 32 x 16 blocks took 16.
__constant__ const unsigned kDiagBlocks[8] = {0x14321077u, 0x14321066u, 0x14321055u, 0x14321044u,
                                              0x03321033u, 0x00021002u, 0x16511061u, 0x05576557u};

// The chain's place (shared): where it goes on after the entry `taken`, which its CTA
// runs meanwhile.
struct Chain {
    int step;      // 2 k, or 2 k + 1 when POTRF(k) has its T(k,k) and waits for A(k+1,k); -1: not this CTA's
    int taken;     // the entry to run
    int patience;  // polls of a wait before the CTA takes entries itself
};
enum : int { CHAIN_GAVE_UP = 0, CHAIN_ON = 1, CHAIN_TAKEN = 2 };
constexpr int kChainPatience = 512;

// The chain's wait for *counter >= v before or in POTRF(k). Once `patience` polls have
// passed without it and the entries before POTRF(k) are not all claimed, it claims
// the next of them for its own CTA (CHAIN_TAKEN). Such an entry depends on entries
// before itself only: claimed by CTAs that run, run here already, or diagonal tasks
// that are done. Never at or past POTRF(k) (place, see append_places): those may wait
// for it. The first time takes longer than any wait beside other CTAs; from then on
// entries are taken without delay. flag: a shared int.
__device__ int chain_wait(const TaskMatrix& m, Chain* chain, int* cursor, const int4* place, const int* counter, int v,
                          int* flag) {
    if (threadIdx.x == 0) {
        int r = CHAIN_GAVE_UP;
        for (long it = 0; it < m.spin && r == CHAIN_GAVE_UP; ++it) {
            if (ld_acquire(counter) >= v) {
                r = CHAIN_ON;
            } else if (ld_acquire(m.abort)) {
                break;
            } else if (it >= chain->patience) {
                const int next = ld_acquire(cursor);
                if (next < place->x && atomicCAS(cursor, next, next + 1) == next) {
                    chain->taken = next;
                    chain->patience = 0;
                    r = CHAIN_TAKEN;
                }
            }
            if (r == CHAIN_GAVE_UP) __nanosleep(32);
        }
        if (r == CHAIN_GAVE_UP) m.give_up();
        flag[0] = r;
    }
    __syncthreads();
    return flag[0];
}

// POTRF(k): A(k,k) -= L(k,k-1) L(k,k-1)^T, the leaf, T(k,k) published, then
// L(k+1,k) = A(k+1,k) T(k,k)^T with T(k,k) still in shared memory (Bs), published.
// A(k+1,k) is fetched beside the leaf once its updates are in. chained: called in
// order by one CTA: L(k,k-1) is left in As by the call before (unless gone: other
// tasks ran since), which also fetched A(k,k) into S when diag_in; at a wait the call
// may return CHAIN_TAKEN, to be repeated with gone (and chain->step odd: from T(k,k)
// on) after the entry taken. Otherwise the caller has waited for both. flag: three
// shared ints.
template <bool chained>
__device__ __forceinline__ int potrf(const TaskMatrix& m, int k, Chain* chain, int* cursor, const int4* place, bool gone,
                                     bool& diag_in, double* sm, int* flag) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    // column blocks 0, 16, 48, 32: the product with a lower triangle takes warps w and
    // w + 4, which share a scheduler, the same time in sum
    const int wm = (warp & 1) * 32, wn = ((warp >> 1) ^ (warp >> 2)) * 16;
    double *As = sm, *Bs = sm + LEAF_TILE, *S = sm + 2 * LEAF_TILE;
    const bool below = k + 1 < m.tiles();
    const bool from_panel = chained && (chain->step & 1);  // T(k,k) is there
    if (!from_panel) {
        if (chained && k > 0 && !diag_in) {
            const int r = chain_wait(m, chain, cursor, place + k, m.ver + tri(k, k), k - 1, flag);
            if (r != CHAIN_ON) return r;
        }
        if (!diag_in) chol_leaf_load(m.A, m.ld, TB * k, m.ext(k), S);
        if (k > 0 && (!chained || gone)) load_tile(As, m.tile(m.A, k, k - 1), m.ld, m.ext(k), m.ext(k - 1), tid);
        tile_wait();
        __syncthreads();
        if (k > 0) {
            // S -= As As^T, lower 8 x 8 blocks only, four or five per warp (kDiagBlocks)
            const unsigned tab = kDiagBlocks[warp];
            const int rows[2] = {(int)(tab & 7u) * 8, (int)(tab >> 4 & 7u) * 8};
            const bool five = (tab >> 28) != 0u;
            int cols[5];
            double c[5][2], d[5][2];
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                cols[q] = (int)(tab >> (8 + 4 * q) & 7u) * 8;
                c[q][0] = c[q][1] = 0.0;
#pragma unroll
                for (int h = 0; h < 2; ++h) d[q][h] = S[(cols[q] + 2 * t4 + h) * TLD + rows[q / 3] + g];
            }
#pragma unroll 4
            for (int kk = 0; kk < TB; kk += 4) {
                const double* at = As + (kk + t4) * TLD + g;
                const double a[2] = {at[rows[0]], at[rows[1]]};
#pragma unroll
                for (int q = 0; q < 4; ++q) dmma(c[q][0], c[q][1], a[q / 3], at[cols[q]]);
                if (five) dmma(c[4][0], c[4][1], a[1], at[cols[4]]);
            }
#pragma unroll
            for (int q = 0; q < 5; ++q)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int col = cols[q] + 2 * t4 + h, row = rows[q / 3] + g;
                    if (col <= row && (q < 4 || five) && !(q == 2 && cols[2] == cols[1]))
                        S[col * TLD + row] = d[q][h] - c[q][h];
                }
        }
        if (tid == 0) flag[0] = 0;
        __syncthreads();
        // A(k+1,k) into As before the leaf's last products when warp 4 has seen its updates
        // (one warp's loads of a tile take longer than a panel: 1.8 us more per step)
        chol_leaf_factor(
            TB * k, m.ext(k), m.T, m.ld, m.err, S, Bs,
            [&](int q) {
                if (!below || q < 2) return;
                for (int poll = q; poll < 5; poll += 2)  // the third panel: twice
                    if (lane == 0 && !flag[0] && ld_acquire(m.ver + tri(k + 1, k)) >= k) flag[0] = 1;
            },
            [&] {
                if (flag[0]) load_tile(As, m.tile(m.A, k + 1, k), m.ld, m.ext(k + 1), m.ext(k), tid);
            });
        tile_wait();
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            atomicExch(m.lrdy + tri(k, k), 1);
            atomicExch(m.trdy + tri(k, k), 1);
        }
    }
    if (!below) return CHAIN_ON;
    if (from_panel || !flag[0]) {
        if (chained) {
            const int r = chain_wait(m, chain, cursor, place + k, m.ver + tri(k + 1, k), k, flag + 1);
            if (r != CHAIN_ON) {
                if (tid == 0) chain->step = 2 * k + 1;
                return r;
            }
            if (from_panel) load_tile(Bs, m.tile(m.T, k, k), m.ld, m.ext(k), m.ext(k), tid);
        } else {
            if (tid == 0) flag[1] = m.wait(m.ver + tri(k + 1, k), k) || m.give_up();
            __syncthreads();
            if (!flag[1]) return CHAIN_GAVE_UP;
        }
        load_tile(As, m.tile(m.A, k + 1, k), m.ld, m.ext(k + 1), m.ext(k), tid);
        tile_wait();
    }
    // the next diagonal tile, when its updates but the last are in (a partial
    // one takes its identity tail from chol_leaf_load)
    if (tid == 32) flag[2] = chained && m.ext(k + 1) == TB && ld_acquire(m.ver + tri(k + 1, k + 1)) >= k;
    __syncthreads();
    diag_in = flag[2];
    if (diag_in) load_tile(S, m.tile(m.A, k + 1, k + 1), m.ld, TB, TB, tid);
    Acc acc = {};
    tile_mma(As, Bs, wm, wn, g, t4, 0, wn + 16, acc);
    if (chained) {
        __syncthreads();  // As is read no more
        tile_elements(TB, TB, wm, wn, g, t4, acc, [&](int r, int c, double& v) { As[c * TLD + r] = v; });
    }
    double* L = m.tile(m.A, k + 1, k);
    tile_elements(m.ext(k + 1), m.ext(k), wm, wn, g, t4, acc, [&](int r, int c, double& v) { L[r + (long)c * m.ld] = v; });
    if (chained && tid == 0) chain->step = 2 * k + 2;
    __syncthreads();
    if (tid == 32 * 5) {  // warp 5: its share of the next update is short
        __threadfence();
        atomicExch(m.lrdy + tri(k + 1, k), 1);
    }
    return CHAIN_ON;
}

// Every POTRF(k) of one matrix from chain->step on, in order, by the calling CTA;
// place: of POTRF(0 ..) in the list.
__device__ __forceinline__ int run_chain(const TaskMatrix& m, Chain* chain, int* cursor, const int4* place, double* sm,
                                         int* flag) {
    bool diag_in = false, gone = true;  // k = 0 needs no tile of before
    for (int k = chain->step >> 1; k < m.tiles(); ++k, gone = false) {
        const int r = potrf<true>(m, k, chain, cursor, place, gone, diag_in, sm, flag);
        if (r != CHAIN_ON) return r;
    }
    return CHAIN_ON;
}

// One tile task (type, i, j, k with its count), run by all DAG_THREADS threads of
// the block; warp 0 waits for its dependencies first. Returns false when a wait
// gave up (ERRBIT_TIMEOUT and the abort flag are set): the caller stops taking
// tasks. kDiagonal: POTRF may be among them.
template <bool kDiagonal>
__device__ __forceinline__ bool run_task(const TaskMatrix& m, int type, int i, int j, int kc, double* sm, int* flag) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t4 = lane & 3;
    const int wm = (warp & 1) * 32, wn = (warp >> 1) * 16;
    const int k = kc & 0xffff, count = kc >> 16;
    const long ld = m.ld;
    if (warp == 0) {
        // lane 0: the tile's own counter; lanes 1 .. count and count + 1 .. 2 count: the operands of each k
        const int *own = nullptr, *first = nullptr, *second = nullptr;
        int v = 0;
        const int q = lane > count ? lane - count - 1 : lane - 1;
        switch (type) {
            case K_POTRF:  // its last update (from panel k-1) is applied inside the task
                if (k > 0) {
                    own = m.ver + tri(k, k);
                    v = k - 1;
                    first = m.lrdy + tri(k, k - 1);
                }
                break;
            case K_TRSM: own = m.ver + tri(i, k), v = k, first = m.lrdy + tri(k, k); break;
            case K_UPDATE:
                own = m.ver + tri(i, j), v = k, first = m.lrdy + tri(i, k + q), second = m.lrdy + tri(j, k + q);
                break;
            case K_TACC:
                own = m.tacc + tri(i, j), v = k - j, first = m.lrdy + tri(i, k + q), second = m.trdy + tri(k + q, j);
                break;
            case K_TFIN: own = m.tacc + tri(i, j), v = i - j, first = m.trdy + tri(i, i); break;
            default:  // K_PACC
                own = m.pacc + tri(i, j), v = k - i, first = m.trdy + tri(k + q, i), second = m.trdy + tri(k + q, j);
                break;
        }
        const int* f = lane == 0 ? own : (lane <= count ? first : (lane <= 2 * count ? second : nullptr));
        const bool ok = wait_all(f, lane == 0 ? v : 1, m.abort, m.spin);
        if (lane == 0) flag[0] = ok || m.give_up();
    }
    __syncthreads();
    if (!flag[0]) return false;
    if (kDiagonal && type == K_POTRF) {
        bool diag_in = false;
        return potrf<false>(m, k, nullptr, nullptr, nullptr, false, diag_in, sm, flag) != CHAIN_GAVE_UP;
    }
    auto ref = [&](double* M, int r, int c) { return TileRef{m.tile(M, r, c), m.ext(r), m.ext(c)}; };
    Acc acc = {}, prev = {};
    switch (type) {
        case K_TRSM:  // L(i,k) = A(i,k) T(k,k)^T; T(k,k) lower: terms k' <= n only
            stream_mma<false, false>(sm, ld, k, 1, [&](int) { return ref(m.A, i, k); },
                                     [&](int) { return ref(m.T, k, k); }, wm, wn, g, t4, wn + 16, tid, acc);
            store_tile(m.tile(m.A, i, k), ld, m.ext(i), m.ext(k), acc, 1.0, prev, nullptr, wm, wn, g, t4);
            break;
        case K_UPDATE:  // A(i,j) -= L(i,k) L(j,k)^T
            load_prev(m.tile(m.A, i, j), ld, m.ext(i), m.ext(j), wm, wn, g, t4, prev);
            stream_mma<false, false>(sm, ld, k, count, [&](int q) { return ref(m.A, i, q); },
                                     [&](int q) { return ref(m.A, j, q); }, wm, wn, g, t4, TB, tid, acc);
            store_tile(m.tile(m.A, i, j), ld, m.ext(i), m.ext(j), acc, -1.0, prev, nullptr, wm, wn, g, t4);
            break;
        case K_TACC:  // W(i,j) += L(i,k) T(k,j)
            if (k > j) load_prev(m.tile(m.T, i, j), ld, m.ext(i), m.ext(j), wm, wn, g, t4, prev);
            stream_mma<false, true>(sm, ld, k, count, [&](int q) { return ref(m.A, i, q); },
                                    [&](int q) { return ref(m.T, q, j); }, wm, wn, g, t4, TB, tid, acc);
            store_tile(m.tile(m.T, i, j), ld, m.ext(i), m.ext(j), acc, 1.0, prev, nullptr, wm, wn, g, t4);
            break;
        case K_TFIN:  // T(i,j) = -T(i,i) W(i,j); T(i,i) lower: terms k' <= m only
            stream_mma<false, true>(sm, ld, i, 1, [&](int) { return ref(m.T, i, i); },
                                    [&](int) { return ref(m.T, i, j); }, wm, wn, g, t4, wm + 32, tid, acc);
            store_tile(m.tile(m.T, i, j), ld, m.ext(i), m.ext(j), acc, -1.0, prev, nullptr, wm, wn, g, t4);
            break;
        default: {  // K_PACC: O(i,j) += T(k,i)^T T(k,j)
            if (k > i) load_prev(m.tile(m.O, i, j), ld, m.ext(i), m.ext(j), wm, wn, g, t4, prev);
            stream_mma<true, true>(sm, ld, k, count, [&](int q) { return ref(m.T, q, i); },
                                   [&](int q) { return ref(m.T, q, j); }, wm, wn, g, t4, TB, tid, acc);
            const bool last = k + count == m.tiles();
            store_tile(m.tile(m.O, i, j), ld, m.ext(i), m.ext(j), acc, 1.0, prev,
                       (last && i > j) ? m.tile(m.O, j, i) : nullptr, wm, wn, g, t4);
            break;
        }
    }
    // release: the barrier orders every thread's tile writes before thread 0's
    // gpu-scope fence, which orders them before the counter
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        switch (type) {
            case K_TRSM: atomicExch(m.lrdy + tri(i, k), 1); break;
            case K_UPDATE: atomicAdd(m.ver + tri(i, j), count); break;
            case K_TACC: atomicAdd(m.tacc + tri(i, j), count); break;
            case K_TFIN: atomicExch(m.trdy + tri(i, j), 1); break;
            default: atomicAdd(m.pacc + tri(i, j), count); break;
        }
    }
    return true;
}

__device__ __forceinline__ int sm_id() {
    unsigned id;
    asm volatile("mov.u32 %0, %%smid;\n" : "=r"(id));
    return (int)id;
}

__global__ void __launch_bounds__(DAG_THREADS, DAG_CTAS)
    k_spd_inverse_tasks(double* A, double* T, double* O, int n, long ld, const int4* __restrict__ tasks, int ntasks,
                        int* state, int ntri, int* err, long spin) {
    extern __shared__ __align__(16) double sm[];
    __shared__ int s_task, flag[3];
    __shared__ Chain chain;
    int* const cursor = state;
    int* const chain_sm = state + 2;  // 1 + the SM that runs the chain
    int* const others = state + 3;    // CTAs that take tasks on other SMs until the list is done
    const TaskMatrix m(A, T, O, n, ld, state, ntri, err, state + 1, spin);
    bool counted = false, begin = false, ran_chain = false;  // thread 0
    if (threadIdx.x == 0) chain = Chain{-1, 0, (int)min((long)kChainPatience, spin / 2)};
    while (true) {
        if (threadIdx.x == 0) {
            if (begin) chain.step = 0;
            begin = false;
            if (chain.step < 0) {
                const int at = ld_acquire(chain_sm), here = sm_id() + 1;
                if (at != 0 && at != here && !counted) {
                    atomicAdd(others, 1);
                    counted = true;
                }
                // beside the chain, unless nobody else is there to do the tasks
                const bool retire = at == here && !ran_chain && ld_acquire(others) > 0;
                s_task = retire ? ntasks : atomicAdd(cursor, 1);
            }
        }
        __syncthreads();
        int4 tk;
        if (chain.step < 0) {
            if (s_task >= ntasks) break;
            tk = tasks[s_task];
            if (threadIdx.x == 0 && tk.x == K_POTRF && tk.y == 0) {
                begin = ran_chain = true;  // the chain, from the next round on
                atomicExch(chain_sm, sm_id() + 1);
            }
        } else {
            const int r = run_chain(m, &chain, cursor, tasks + ntasks, sm, flag);
            if (r == CHAIN_GAVE_UP) break;
            __syncthreads();
            tk = tasks[chain.taken];
            if (r == CHAIN_ON) {  // all done: among the others from now on
                tk.x = K_POTRF;
                if (threadIdx.x == 0) chain.step = -1;
            }
        }
        if (tk.x != K_POTRF && !run_task<false>(m, tk.x, tk.y, tk.z, tk.w, sm, flag)) break;
        __syncthreads();  // s_task, flag and the chain's place are rewritten
    }
}

// The same schedule over the tile tasks of many matrices (a batch of
// reconstructions) in one persistent launch: task.x = type + 8 * matrix, the
// matrices' descriptors in `mats`, their counters at mats[m].state, one cursor
// and one abort flag (ctl[0], ctl[1]) for the whole list. The list interleaves
// the matrices' own topological orders, so every dependency of a task is still
// earlier in the list and the launch completes with any number of resident
// CTAs; each task does exactly the arithmetic of the single-matrix kernel, so
// the results are bitwise those of one launch per matrix.
__global__ void __launch_bounds__(DAG_THREADS, DAG_CTAS)
    k_spd_inverse_tasks_grouped(const SpdTaskMatrix* __restrict__ mats, const int4* __restrict__ tasks, int ntasks,
                                int* ctl, long spin) {
    extern __shared__ __align__(16) double sm[];
    __shared__ int s_task, flag[3];
    while (true) {
        if (threadIdx.x == 0) s_task = atomicAdd(ctl, 1);
        __syncthreads();
        const int task = s_task;
        if (task >= ntasks) break;
        const int4 tk = tasks[task];
        const SpdTaskMatrix& d = mats[tk.x >> 3];
        const TaskMatrix m(d.A, d.T, d.O, d.n, d.ld, d.state, d.ntri, d.err, ctl + 1, spin);
        if (!run_task<true>(m, tk.x & 7, tk.y, tk.z, tk.w, sm, flag)) break;
        __syncthreads();
    }
}

// Consecutive terms of one tile that a task takes, by the number of tiles: the
// work of a step grows with nt^2, the chain's time for it does not. While the
// CTAs keep up with single terms a group only delays its tile; beyond that the
// longer groups save the CTAs a load and a store of the tile per term. Single,
// pairs, threes and fours, with the product (us): n = 1800 505, 525, 539, 572;
// 2300 816, 700, 725, 794; 2432 951, 808, 787, 845; 2752 1355, 1130, 1076, 1056.
// Without the product a step has about two thirds of the work: n = 1984 497, 510,
// 534, 550; 2400 714, 649, 667, 728; 2701 969, 841, 834, 863; 3584 1994, 1645,
// 1566, 1538.
int group_size(int nt, bool product) {
    const int load = product ? nt : nt - 4;
    return load <= 30 ? 1 : load <= 37 ? 2 : load <= 41 ? 3 : MAX_GROUP;
}

// The task list of nt x nt tiles in the order described above; without the
// product, T = L^{-1} only (no PACC). At step s panel s, T's row s - 1 and the
// product terms of T's row s - 1 become available (T's row s is final at the end
// of step s: its product terms come a step later, where they do not wait for it;
// n = 1800: 562 -> 504 us). A tile that is not needed in the next two steps takes
// its terms in groups, whose ends fall on another step for each of the group's
// size of neighbouring tiles, so that every step has its share of them and none
// floods the CTAs that the chain waits for; one that is needed in the step after
// next takes the rest of its group, so that only a single term is left when the
// next step waits for it. The last two product terms are single ones (a short
// tail).
std::vector<int4> build_tasks(int nt, bool product = true) {
    std::vector<int4> v;
    auto add = [&v](int ty, int i, int j, int first, int last) {
        v.push_back(make_int4(ty, i, j, first | (last - first + 1) << 16));
    };
    const int size = group_size(nt, product);
    // tile (i, j): terms first_of(i, j, s) .. s are one group at step s when ends(i, j, s)
    auto ends = [size](int i, int j, int s) { return (s + i + j) % size == size - 1; };
    auto first_of = [size](int i, int j, int s) { return std::max(0, s - (s + i + j) % size); };
    // POTRF(k) also applies UPDATE(k,k,k-1) first and computes TRSM(k+1,k) last
    add(K_POTRF, 0, 0, 0, 0);
    for (int i = 2; i < nt; ++i) add(K_TRSM, i, 0, 0, 0);
    for (int s = 0; s < nt; ++s) {
        if (s + 1 < nt) {
            if (s + 2 < nt) add(K_UPDATE, s + 2, s + 1, s, s);  // the input of the fused TRSM(s+2,s+1)
            add(K_POTRF, s + 1, s + 1, s + 1, s + 1);
            if (s + 2 < nt) add(K_UPDATE, s + 2, s + 2, first_of(s + 2, s + 2, s), s);  // the next diagonal tile
            for (int i = s + 3; i < nt; ++i) {
                add(K_UPDATE, i, s + 1, s, s);
                add(K_TRSM, i, s + 1, s + 1, s + 1);
            }
            for (int j = s + 2; j < nt; ++j)
                for (int i = j + (j == s + 2); i < nt; ++i)
                    if (j == s + 2 || ends(i, j, s)) add(K_UPDATE, i, j, first_of(i, j, s), s);
        }
        if (s >= 1) {
            const int p = s - 1;  // T's row p is final
            for (int c = 0; c < s; ++c) add(K_TACC, s, c, p, p);
            for (int r = s + 1; r < nt; ++r)
                for (int c = 0; c < s; ++c)
                    if (r == s + 1 || ends(r, c, p)) add(K_TACC, r, c, std::max(c, first_of(r, c, p)), p);
        }
        for (int c = 0; c < s; ++c) add(K_TFIN, s, c, 0, 0);
        for (int k = s - 1; product && k <= (s == nt - 1 ? s : s - 1); ++k)
            for (int r = 0; r <= k; ++r)
                for (int c = 0; c <= r; ++c) {
                    const bool last = k == nt - 1;
                    if (last || k == nt - 2 || ends(r, c, k))
                        add(K_PACC, r, c, last ? k : std::max(r, first_of(r, c, k)), k);
                }
    }
    return v;
}

// The same with every group as its single terms, one after the other.
std::vector<int4> single_tasks(const std::vector<int4>& v) {
    std::vector<int4> out;
    for (const int4& t : v)
        for (int q = 0; q < t.w >> 16; ++q) out.push_back(make_int4(t.x, t.y, t.z, ((t.w & 0xffff) + q) | 1 << 16));
    return out;
}

// After the list the places of POTRF(0 .. nt - 1) in it, for the chain (0 where one is left out).
void append_places(std::vector<int4>& v, int nt) {
    std::vector<int> place(nt, 0);
    for (size_t q = 0; q < v.size(); ++q)
        if (v[q].x == K_POTRF) place[v[q].y] = (int)q;
    for (int p : place) v.push_back(make_int4(p, 0, 0, 0));
}

struct TaskLists {
    std::mutex mu;
    std::map<std::tuple<int, int, bool>, std::pair<int4*, int>> lists;  // (device, nt, product) -> device copy, tasks
    std::map<int, cudaStream_t> upload;                          // device -> upload stream
};
TaskLists& task_lists() {
    static TaskLists* t = new TaskLists;  // lives until exit, like the device buffers it holds
    return *t;
}

}  // namespace

bool spd_tasks_apply(int n) { return n > 0 && (n + TB - 1) / TB <= kMaxTilesN; }

size_t spd_task_state_ints(int n) {
    const size_t nt = (size_t)(n + TB - 1) / TB;
    return 4 + 5 * nt * (nt + 1) / 2;
}

int spd_tasks_prepare(int n, bool product) {
    if (!spd_tasks_apply(n)) return UNC_ERR_INVALID_ARG;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return UNC_ERR_CUDA;
    const int nt = (n + TB - 1) / TB;
    TaskLists& tl = task_lists();
    std::lock_guard<std::mutex> lock(tl.mu);
    if (tl.lists.count({dev, nt, product})) return UNC_OK;
    std::vector<int4> h = build_tasks(nt, product);
    const int ntasks = (int)h.size();
    append_places(h, nt);
    // upload on a private non-blocking stream: a copy on the legacy default
    // stream would wait for every other stream's work (a serving process runs
    // several requests at once)
    auto it = tl.upload.find(dev);
    if (it == tl.upload.end()) {
        cudaStream_t us = nullptr;
        if (cudaStreamCreateWithFlags(&us, cudaStreamNonBlocking) != cudaSuccess) return UNC_ERR_CUDA;
        it = tl.upload.emplace(dev, us).first;
    }
    cudaStream_t us = it->second;
    int4* d = nullptr;
    if (cudaMallocAsync(reinterpret_cast<void**>(&d), sizeof(int4) * h.size(), us) != cudaSuccess)
        return UNC_ERR_OUT_OF_MEMORY;
    if (cudaMemcpyAsync(d, h.data(), sizeof(int4) * h.size(), cudaMemcpyHostToDevice, us) != cudaSuccess ||
        cudaStreamSynchronize(us) != cudaSuccess) {
        cudaFreeAsync(d, us);
        return UNC_ERR_CUDA;
    }
    static std::atomic<unsigned long long> attr{0};
    once_per_device(attr, [] {
        return cudaFuncSetAttribute(k_spd_inverse_tasks, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)DAG_SMEM) == cudaSuccess;
    });
    tl.lists[{dev, nt, product}] = {d, ntasks};
    return UNC_OK;
}

int chol_inverse_tasks(double* A, int n, int lda, double* T, double* O, int* state, int* err, cudaStream_t st,
                       int max_ctas, long long poll_limit, int skip_task, int max_grid) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return UNC_ERR_CUDA;
    const int nt = (n + TB - 1) / TB;
    std::pair<int4*, int> list{nullptr, 0};
    {
        TaskLists& tl = task_lists();
        std::lock_guard<std::mutex> lock(tl.mu);
        auto it = tl.lists.find({dev, nt, O != nullptr});
        if (it == tl.lists.end()) return UNC_ERR_INVALID_ARG;  // spd_tasks_prepare first (outside any capture)
        list = it->second;
    }
    const int ntri = nt * (nt + 1) / 2;
    if (cudaMemsetAsync(state, 0, sizeof(int) * spd_task_state_ints(n), st) != cudaSuccess) return UNC_ERR_CUDA;
    const long spin = poll_limit > 0 ? (long)std::min<long long>(poll_limit, kDagSpin) : kDagSpin;
    int4* own = nullptr;  // a schedule with one task left out (tests of the bounded waits)
    if (skip_task >= 0 && skip_task < unc_spd_task_list(n, nullptr, 0)) {
        std::vector<int4> h = single_tasks(build_tasks(nt, O != nullptr));
        h.erase(h.begin() + skip_task);
        const int left = (int)h.size();
        append_places(h, nt);
        if (cudaMallocAsync(reinterpret_cast<void**>(&own), sizeof(int4) * h.size(), st) != cudaSuccess)
            return UNC_ERR_OUT_OF_MEMORY;
        if (cudaMemcpyAsync(own, h.data(), sizeof(int4) * h.size(), cudaMemcpyHostToDevice, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess) {
            cudaFreeAsync(own, st);
            return UNC_ERR_CUDA;
        }
        list = {own, left};
    }
    int grid = std::max(1, std::min(DAG_CTAS * std::min(device_sms(), max_ctas), list.second));
    if (max_grid > 0) grid = std::min(grid, max_grid);
    k_spd_inverse_tasks<<<grid, DAG_THREADS, DAG_SMEM, st>>>(A, T, O, n, lda, list.first, list.second, state, ntri,
                                                             err, spin);
    count_launch();
    if (own && cudaFreeAsync(own, st) != cudaSuccess) return UNC_ERR_CUDA;
    return UNC_OK;
}

std::vector<int4> spd_tasks_grouped_list(const std::vector<int>& ns) {
    struct Item {
        double key;
        int m, q;
        int4 t;
    };
    std::vector<Item> items;
    for (int m = 0; m < (int)ns.size(); ++m) {
        const std::vector<int4> v = build_tasks((ns[m] + TB - 1) / TB);
        for (int q = 0; q < (int)v.size(); ++q) {
            int4 t = v[q];
            t.x += 8 * m;
            items.push_back({(q + 1.0) / (double)v.size(), m, q, t});
        }
    }
    // stable in (key, matrix, position): a matrix's own order is kept
    std::sort(items.begin(), items.end(), [](const Item& a, const Item& b) {
        if (a.key != b.key) return a.key < b.key;
        if (a.m != b.m) return a.m < b.m;
        return a.q < b.q;
    });
    std::vector<int4> out(items.size());
    for (size_t i = 0; i < items.size(); ++i) out[i] = items[i].t;
    return out;
}

void prepare_task_kernels() {
    static std::atomic<unsigned long long> attr{0};
    once_per_device(attr, [] {
        return cudaFuncSetAttribute(k_spd_inverse_tasks, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)DAG_SMEM) == cudaSuccess &&
               cudaFuncSetAttribute(k_spd_inverse_tasks_grouped, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)DAG_SMEM) == cudaSuccess;
    });
}

int chol_inverse_tasks_grouped(const SpdTaskMatrix* d_mats, const int4* d_tasks, int ntasks, int* ctl,
                               cudaStream_t st, int max_ctas, long long poll_limit) {
    if (ntasks <= 0) return UNC_OK;
    prepare_task_kernels();
    const long spin = poll_limit > 0 ? (long)std::min<long long>(poll_limit, kDagSpin) : kDagSpin;
    const int grid = std::max(1, std::min(DAG_CTAS * std::min(device_sms(), max_ctas), ntasks));
    k_spd_inverse_tasks_grouped<<<grid, DAG_THREADS, DAG_SMEM, st>>>(d_mats, d_tasks, ntasks, ctl, spin);
    count_launch();
    return UNC_OK;
}

}  // namespace unc

// The task order of the tile-task inverse for an n x n matrix, for tools that
// check or draw the schedule: returns the number of tasks; with out != NULL and
// capacity >= that number, out receives 4 ints per task (kind 0..5 = POTRF,
// TRSM, UPDATE, TACC, TFIN, PACC; then i, j, k as in the kernel). Host only.
extern "C" int unc_spd_task_list(int n, int* out, int capacity) {
    unc::g_last_error.clear();
    if (!unc::spd_tasks_apply(n)) {
        unc::g_last_error = "unc_spd_task_list: n must be in 1..3584";
        return UNC_ERR_INVALID_ARG;
    }
    const std::vector<int4> v = unc::single_tasks(unc::build_tasks((n + unc::NB - 1) / unc::NB));
    if (out && capacity >= (int)v.size())
        for (size_t q = 0; q < v.size(); ++q) {
            out[4 * q] = v[q].x;
            out[4 * q + 1] = v[q].y;
            out[4 * q + 2] = v[q].z;
            out[4 * q + 3] = v[q].w & 0xffff;
        }
    return (int)v.size();
}
