// internal.h - shared declarations of the uncertaintyTE B200 kernels.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/uncte.h"

namespace unc {

// Device-side error bits (accumulated with atomicOr into a device int).
enum : int {
    ERRBIT_LAYOUT = 1,      // observation rows not 12 entries / columns out of range
    ERRBIT_SINGULAR = 2,    // non-positive or non-finite pivot
    ERRBIT_NONFINITE = 4,   // NaN / Inf produced
    ERRBIT_SCHUR_CAP = 32,  // a point has more observations than the Schur stage takes (kSchurMaxList)
    ERRBIT_TIMEOUT = 16,    // a bounded device wait ran out (tensor-core pipeline)
};

constexpr int kCamParams = 9;
constexpr int kObsVals = 24;  // one observation = 2 rows x (9 camera + 3 point) values

// Round a leading dimension up so every column starts 64-byte aligned.
inline int ld_of(int n) { return (n + 7) & ~7; }

extern thread_local std::string g_last_error;

// Streaming multiprocessors of the current device (queried once per device;
// 148 on a B200, fewer on a partitioned GPU).
int device_sms();

// Runs f() (returning true on success) until it succeeds once per device
// (ordinal < 64) for one call site, from any thread: per-function CUDA
// attributes are per device, and several host threads (one per context) may
// launch the same kernels concurrently. prepare_kernels() runs every such site
// when a context is created, outside any stream capture.
template <class F>
void once_per_device(std::atomic<unsigned long long>& done, F&& f) {
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ULL << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return;
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    if (done.load(std::memory_order_relaxed) & bit) return;
    if (f()) done.fetch_or(bit, std::memory_order_release);
}
// Device scratch of one call, allocated in stream order from the library's own
// memory pool of the current device and freed in stream order when it goes out
// of scope. Between calls the pool keeps at most kScratchKept bytes, so that a
// repeated call neither maps nor unmaps memory (cudaMalloc, cudaFree and their
// implicit synchronisation cost 0.4 to 4 ms beside kernels of 0.5 to 15 ms);
// more than that goes back at the next synchronisation, everything when
// scratch_trim is called (a context or batch is released or destroyed).
// Thread-safe; streams may differ from call to call.
constexpr unsigned long long kScratchKept = 1ULL << 30;
struct Scratch {
    void* p = nullptr;
    cudaStream_t st = nullptr;
    cudaError_t alloc(size_t bytes, cudaStream_t stream);
    ~Scratch();
};
void scratch_trim();  // of the current device

// Per-device set-up of the kernels' shared-memory attributes (current device).
void prepare_assembly_kernels();
void prepare_dense_kernels();
void prepare_mixed_kernels();

// Bump allocator over one device allocation; every piece 256-byte aligned.
// With base == nullptr it only measures the total size.
struct Carver {
    char* base;
    size_t off = 0;
    template <class T>
    T* take(size_t n) {
        off = (off + 255) & ~size_t(255);
        T* p = reinterpret_cast<T*>(base ? base + off : nullptr);
        off += n * sizeof(T);
        return p;
    }
};
extern long long g_launches;
extern thread_local long long g_thread_launches;
inline void count_launch(int n = 1) {
    __atomic_add_fetch(&g_launches, n, __ATOMIC_RELAXED);
    g_thread_launches += n;
}

// ---------------- assembly.cu ----------------
struct SceneDev {
    int num_cams, num_points, num_obs;  // num_obs = num_rows / 2
    long nnz;                           // entries of cols / values
    int fix[3];
    int has_fix;
    const int* rows;      // CRS rowptr
    const int* cols;      // CRS column ids
    const double* J;      // observation blocks, 24 doubles each: [row0: c0..c8 p0..p2 | row1: ...]
    int* obs_cam;         // per observation camera id (-1 = dropped)
    int* obs_pt;          // per observation point id (-1 = dropped: fixed point or no point)
    int* cam_ptr;         // num_cams + 1
    int* cam_obs;         // observation ids grouped by camera (ascending within a camera): the camera order
    int* pt_ptr;          // num_points + 1
    int2* pt_list;        // per point its observations: (position in the camera order, camera), ascending
    int2* pt_tmp;         // scratch: the lists in arrival order
    int2* pos_list;       // per position: the start of its point's list, its rank in it
    int* index_tmp;       // scratch: index_scratch_ints(num_cams, num_points)
    double* s_cam;        // 9*num_cams column norms of J (camera columns)
    double* is_cam;       // 9*num_cams their inverses (1 for a zero norm)
    double* Vraw;         // 6*num_points upper triangle of the unscaled point block J_p^T J_p
    double* Mp;           // 6*num_points M_p, M_p M_p^T = V_p^{-1} (k_point_blocks), or nullptr
    double* Q;            // 27*num_obs by position: Q_o = W_o M_p, 9x3 row-major (W_o = J_c^T J_p); after the
                          // Schur stage 6 per position: the observation's share of its point's covariance
    double* cam_part;     // 90 * camera_tile_slots(): per-tile partial sums of the camera blocks and self terms
    double* Ucam;         // 81*num_cams scaled camera blocks U (9 x 9, column-major)
    int* err;             // device error bits
};

void launch_validate_obs(const SceneDev& s, cudaStream_t st);
// Camera observations are processed in tiles of 256; slots = C + num_obs/256 + 1.
size_t camera_tile_slots(int num_cams, int num_obs);
void launch_build_index(SceneDev& s, cudaStream_t st);
// After it, where points of more than kSchurMaxList observations are taken (not in a solve): their lists.
void launch_long_lists(const SceneDev& s, cudaStream_t st);
size_t index_scratch_ints(int num_cams, int num_points);
// Point blocks and, unless s.Mp is nullptr, their inverse factors.
void launch_point_blocks(const SceneDev& s, cudaStream_t st);
// U blocks (scaled) into s.Ucam, column norms into s.s_cam / s.is_cam, the Q
// records (after the point blocks).
void launch_camera_blocks(const SceneDev& s, cudaStream_t st);
// The Schur complement Z = U - W V^-1 W^T (schur.cu) over a zeroed Z: the
// diagonal blocks from s.Ucam, every co-visible camera-pair block written in
// both triangles, bitwise symmetric. UNC_ERR_TOO_LARGE above kSchurMaxCams;
// nothing is written when ERRBIT_SCHUR_CAP is set.
constexpr int kSchurMaxList = 12288;  // observations of one point
constexpr int kSchurMaxCams = 5120;  // above the dense path's limit (9 C <= 46000)
int launch_schur_columns(const SceneDev& s, double* Z, int ldz, cudaStream_t st);
size_t schur_columns_smem(int num_cams);
void prepare_schur_columns();  // kernel attributes (before any stream capture)
// Generic 9/12-entry-row repack for the J^T J export (camera-only rows allowed).
void launch_repack_generic(int num_obs, int num_cams, int num_points, const int* rows, const int* cols,
                           const double* vals, double* J, int* obs_cam, int* obs_pt, int* err,
                           cudaStream_t st);
void launch_unscaled_blocks(const SceneDev& s, double* U, double* W, cudaStream_t st);

// ---------------- dense.cu ----------------
// C = alpha*A*B + beta*C, column-major, FP64 on DMMA. If amax != nullptr the
// epilogue folds max|C| into *amax (bit pattern of a non-negative double).
void gemm_f64(int M, int N, int K, double alpha, const double* A, int lda, const double* B,
              int ldb, double beta, double* C, int ldc, unsigned long long* amax, cudaStream_t st);
// Mode bits of gemm_f64_mode. The k-range bits restrict the k loop of the output
// tile at (m0, n0) when an operand is triangular (terms outside the range are
// zero): KLO_M k >= m0, KLO_N k >= n0, KHI_M k < m0 + B, KHI_N k < n0 + B, B the
// side of the tile (64, or 32 where 64 x 64 tiles are fewer than the SMs).
enum : int {
    GEMM_LOWER = 1,    // tiles strictly above the diagonal are skipped
    GEMM_TRANS_B = 2,  // B(k, n) is read from B[n + k * ldb]
    GEMM_KLO_M = 4,
    GEMM_KLO_N = 8,
    GEMM_KHI_M = 16,
    GEMM_KHI_N = 32,
    GEMM_MIRROR = 64,  // symmetric C: write the lower triangle at (i, j) and (j, i), nothing above it directly
    GEMM_SHORT_ACC = 128,  // partial sums over k = 32 from zero, added to the running sums (the products
                           // that feed Cholesky pivots: see k_gemm_f64); with GEMM_TRANS_B only
    GEMM_TRANS_A = 256,    // A(m, k) is read from A[k + m * lda]; without GEMM_TRANS_B only
};
// ws (ws_doubles): optional scratch that enables split-K for outputs with
// fewer tiles than SMs (partials summed in a fixed order by a second kernel).
// skip: optional device flag; when it is non-zero the kernels return at once
// (the Taylor loop launches all its iterations and stops on the device).
void gemm_f64_mode(int M, int N, int K, double alpha, const double* A, int lda, const double* B, int ldb,
                   double beta, double* C, int ldc, unsigned long long* amax, int mode, cudaStream_t st,
                   double* ws = nullptr, size_t ws_doubles = 0, const int* skip = nullptr);
// Scratch of an SPD inverse of order n: T (receives L^{-1}; its tiles above the
// diagonal are neither read nor written) and W, n x lda each; ws: n x lda doubles of split-K
// partial sums, or unused by the tile tasks; state: spd_task_state_ints(n) ints
// of the tile tasks (dag.cu), nullptr to run without them (nothing uploaded).
struct SpdScratch {
    double *T, *W, *ws;
    int* state;
    int max_ctas = 148;        // SMs that the tile tasks may cover
    long long poll_limit = 0;  // as chol_inverse_tasks
    int skip_task = -1;
    int max_grid = 0;
};
// Uploads the task lists that an inverse of order n uses (once per device and
// size; outside any stream capture).
int spd_prepare(int n);
// In-place inverse of A + shift I (SPD, n x n, lda, both triangles), Jacobi
// equilibrated (e: n doubles): tile tasks up to n = 3584, above by recursion on
// halves. Y (optional): a copy of the result. Sets ERRBIT_SINGULAR in err.
int spd_inverse(double* A, int n, int lda, double shift, double* e, const SpdScratch& s, double* Y, int* err,
                cudaStream_t st);
// The recursion alone: T = L^{-1} (lower triangle), A overwritten.
int chol_lower_inverse(double* A, int n, int lda, const SpdScratch& s, int* err, cudaStream_t st);
// A <- A + lambda*I and symmetric Jacobi equilibration: A_s = E A E, E = diag(A_ii)^-1/2.
void launch_shift_equilibrate(double* A, int n, int lda, double lambda, double* e, int* err,
                              cudaStream_t st);
// X <- E X E (undo equilibration), also copies into Y if Y != nullptr.
void launch_unequilibrate(double* X, int n, int lda, const double* e, double* Y, cudaStream_t st);
// X = diag(e) S diag(e) from a separate source S, Y (optional) = X.
void launch_unequilibrate_from(const double* S, double* X, int n, int lda, const double* e, double* Y,
                               cudaStream_t st);

// ---------------- dag.cu ----------------
// SPD inverse as 64 x 64 tile tasks in one persistent kernel, for n <= 3584:
// A (lower triangle) is overwritten by L, T receives L^{-1} (lower tiles) and
// O = A^{-1} (both triangles). state: spd_task_state_ints(n) ints.
// spd_tasks_prepare uploads the task list of this size once per device (call it
// outside stream capture). O == nullptr (prepared with product = false): T only.
bool spd_tasks_apply(int n);
size_t spd_task_state_ints(int n);
int spd_tasks_prepare(int n, bool product = true);
// max_ctas bounds the SMs that the persistent grid covers (two CTAs each);
// the task order and every tile's update order do not depend on it, so neither
// do the results.
// poll_limit (> 0): polls of one dependency before a wait gives up (default
// and maximum 2^22); skip_task >= 0 leaves that task out of the schedule, which
// can then not complete: only for tests of the bounded waits; max_grid > 0 bounds
// the CTAs of the launch.
int chol_inverse_tasks(double* A, int n, int lda, double* T, double* O, int* state, int* err, cudaStream_t st,
                       int max_ctas = 148, long long poll_limit = 0, int skip_task = -1, int max_grid = 0);
// One matrix of a grouped tile-task inverse: A (lower triangle) becomes L, T
// receives L^{-1}, O = A^{-1}; state: spd_task_state_ints(n) zeroed ints; err:
// the matrix's error word.
struct SpdTaskMatrix {
    double *A, *T, *O;
    long ld;
    int n, ntri;
    int* state;
    int* err;
};
// The interleaved task list of matrices of sizes ns (each <= 3584): every
// matrix's own order kept, merged by fractional position so that all matrices
// progress together; task.x = type + 8 * matrix index.
std::vector<int4> spd_tasks_grouped_list(const std::vector<int>& ns);
// Shared-memory attributes of the tile-task kernels (current device; call it
// outside any stream capture).
void prepare_task_kernels();
// One persistent launch over the list (d_mats / d_tasks in device memory; ctl:
// 2 ints, zeroed by the caller in stream order, as is every matrix's state).
int chol_inverse_tasks_grouped(const SpdTaskMatrix* d_mats, const int4* d_tasks, int ntasks, int* ctl,
                               cudaStream_t st, int max_ctas, long long poll_limit = 0);
// per context: the largest grid of the tile-task inverse (148 unless set)
void context_set_task_ctas(unc_context* c, int max_ctas);
// Device-side control of the Taylor loop (compute.cpp:141-160): the stop rule
// runs on the device so that the host never waits inside the loop.
struct TeState {
    int done;               // the loop has stopped: later iteration kernels return at once
    int bad;                // a power was not finite
    int iters;              // iterations performed
    double old_change;      // previous |k * max|add||
    double coef;            // k of the current iteration (read by the axpy)
    double change[20];      // cycle_change record
    // blocked-power evaluation (powers.cu): the series' coefficients c[0] = 1,
    // c[i] = k_i for the performed iterations, 0 after; skip[0]: X^16 is not
    // needed, skip[q] (q = 1..4): the terms c[4q .. 4q + 3] are all zero
    double c[20];
    int skip[8];
};
// One thread: change = |k * max(amax, DBL_MIN)|; stop when change < 1e-5 or
// change > old_change, else record it and publish k for the axpy.
void launch_te_decide(TeState* s, const unsigned long long* amax, double k, cudaStream_t st);
// Reset the state (not done, no iteration, old change = DBL_MAX) and the 24
// words of dmax (optional).
void launch_te_init(TeState* s, unsigned long long* dmax, cudaStream_t st);
// ---------------- powers.cu ----------------
// The Taylor series iZ = X + sum_{i=1..m} k_i X^(i+1) (compute.cpp:141-160)
// evaluated from the powers X^2, X^3, X^4, X^8, X^12 (X^16 when m >= 15) on the
// camera blocks of iZ: the stop rule's max|X^j| is the largest diagonal entry of
// the SPD power X^j, the dot product of columns of two lower powers, and the
// camera blocks of X^(4q + r + 1) are products of nine columns of X^(4q) and
// X^(r+1). 5 products for m <= 15 instead of m + 1.
constexpr int kPowerPairs = 45;  // lower triangle of a 9 x 9 block
struct PowerSet {
    double* M[7];  // X, X^2, X^3, X^4, X^8, X^12, X^16
    double* blk;   // [camera][4 (q - 1) + r][45]: camera blocks of X^(4q) X^(r+1), q = 1..4, r = 0..3
    int n;
    long ld;       // even, the matrices 16-byte aligned
    unsigned long long* dmax;  // 21 words: max diag of X^j, j = 0..20 (bits of a non-negative double)
    TeState* te;
};
// Slices of the int8-sliced products of the blocked-power evaluation (mixed
// modes with S slices). Product q: 0..5 = X^2, X^3, X^4, X^8, X^12, X^16. Z is
// positive semi-definite, so the eigenvalues of X = (Z + lambda I)^-1 are at
// most 1/lambda and the series term lambda^i / (i-1)! X^(i+1) = X (lambda X)^i /
// (i-1)! has norm at most ||X|| / (i-1)! (32-bit factorial): the terms past
// X^8, which alone come from X^8, X^12 and X^16, add at most 2.3e-4 ||X||, so
// those three take one slice (7 bits) fewer; for the stop rule's diagonal maxima
// that is a relative error of ~2^-28. The digits are rounded greedily, so the
// first k slices of an operand are its k-slice form: the same slice buffers
// serve every count.
inline int power_product_slices(int q, int S) { return q >= 3 && S > 2 ? S - 1 : S; }
// k[i - 1] = lambda^i / factorial(i - 1), i = 1..19 (host values)
struct TaylorCoefs {
    double k[19];
};
// The camera blocks and diagonal maxima from X .. X^12 (past_15: those with
// X^16), unless *skip; grouped: over the cameras of every set (d_blk_cols: the
// sets' column offsets).
void prepare_power_kernels();  // kernel attributes (before any stream capture)
void launch_power_blocks(const PowerSet& ps, bool past_15, const int* skip, cudaStream_t st);
void launch_power_blocks_grouped(const PowerSet* d_sets, int nsets, const long* d_blk_cols, long nblk_cols, bool past_15,
                                 cudaStream_t st);
// The stop rule over iterations [ilo, ihi] from the diagonal maxima (a
// non-finite one marks the state bad); the coefficients c[i] of the performed
// iterations; after ilo..15 the X^16 skip word, after ..19 the block skip words.
void launch_power_decide(TeState* te, const unsigned long long* dmax, const TaylorCoefs& k, int ilo, int ihi,
                         cudaStream_t st);
// d_k: 19 coefficients per set (set-major)
void launch_power_decide_grouped(const PowerSet* d_sets, int nsets, const double* d_k, int ilo, int ihi,
                                 cudaStream_t st);
// The camera output and the unscaled 9x9 camera covariance blocks (as
// launch_camera_output) of the series' sum.
void launch_power_output(const PowerSet& ps, const double* s_cam, double* cam_unc, double* sig, cudaStream_t st);

// Grouped dense-stage kernels over many matrices (a batch). Element-wise
// launches: block b belongs to job m with blk[m] <= b < blk[m + 1] (blk: njobs
// + 1 longs; 256 threads per block over the job's rows, or
// scale_blocks_grouped(n) blocks over its elements).
struct DenseJob {
    double *Z, *add, *e;  // Z (in: Schur complement, out: X), add (O = inverse)
    long ld;
    int n;
    double lambda;
    int* err;
    TeState* te;
};
// Z += lambda I and the symmetric equilibration of every job (as launch_shift_equilibrate).
void launch_shift_equilibrate_grouped(const DenseJob* d_jobs, int njobs, const long* d_blk_rows, long nblk_rows,
                                      const long* d_blk_elems, long nblk_elems, cudaStream_t st);
// Z = E add E for every job (as launch_unequilibrate_from(add, Z, ...)).
void launch_unequilibrate_grouped(const DenseJob* d_jobs, int njobs, const long* d_blk_elems, long nblk_elems,
                                  cudaStream_t st);
long scale_blocks_grouped(int n);
void launch_te_init_grouped(const DenseJob* d_jobs, int njobs, cudaStream_t st);
void launch_axpy_te(double* Y, const double* X, const TeState* s, int n, int ld, cudaStream_t st);
// Camera output (a+b/2 quirk) and the unscaled 9x9 camera covariance blocks.
void launch_camera_output(const double* iZ, int ldz, const double* s_cam, int num_cams,
                          double* cam_unc, double* sig, cudaStream_t st);

// ---------------- mixed.cu ----------------
// A symmetric FP64 operand sliced into `slices` int8 planes for the tcgen05
// (kind::i8) products, with its TMA descriptor and per-row exponents.
struct MixedOperand {
    CUtensorMap map;
    int8_t* buf;   // slices x rows x kp bytes, zeros past column n
    int* exps;     // n row exponents
    int n, slices, rows, kp;
};
int mixed_tile_n(int slices, int n);
// int8 multiply-adds x 2 that one lower-triangle product of n x n operands
// issues with `slices` slices (tile padding included).
double mixed_issued_ops(int n, int slices);
size_t mixed_slice_bytes(int n, int slices);
// Prepare the operand over buf/exps (as_b: box rows of the B operand). False
// when the driver's tensor-map encoder is unavailable.
bool mixed_plan(MixedOperand& op, int8_t* buf, int* exps, int n, int slices, bool as_b);
struct TeState;
// Operand planning with an explicit output tile width nt (the B boxes' rows):
// rows padded for both the 128-row A boxes and nt; the slice bytes for it.
bool mixed_plan_nt(MixedOperand& op, int8_t* buf, int* exps, int n, int slices, bool as_b, int nt);
size_t mixed_slice_bytes_nt(int n, int slices, int nt);
// The same sliced operand used with its first `slices` slices only (the digits
// are greedy, so they are the operand's representation with fewer slices):
// same buffer and plane stride; as_b: a B map with that slice count's tile
// width. *ok: false when the tensor map could not be encoded.
MixedOperand mixed_fewer_slices(const MixedOperand& op, int slices, bool as_b, bool* ok);
// Grouped forms for a batch of matrices (arguments in device memory).
struct MixedSliceJob {  // k_slice_rows of one matrix
    const double* A;
    long lda;
    int n;
    int8_t* out;
    int rows_pad, kp;
    int* exps;
};
struct MixedGemmJob {  // one lower-triangle symmetric product C = P X (mirrored)
    const CUtensorMap* tA;  // 64-byte aligned maps in device memory
    const CUtensorMap* tB;
    int n, kp, rowsA, rowsB;
    const int* eA;
    const int* eB;
    double* C;
    long ldc;
    unsigned long long* amax;
    int* err;
    const int* skip;
};
// block b of the launch slices row b - row_start[m] of job m (row_start: njobs + 1 ints)
void mixed_slice_grouped(int slices, const MixedSliceJob* d_jobs, int njobs, const int* d_row_start, int total_rows,
                         cudaStream_t st);
// the lower-triangle 128 x nt tiles of an n x n product, as (job, m0, n0, 0)
void mixed_lower_tiles(int job, int n, int nt, std::vector<int4>& out);
// tile width of a grouped product over scenes of sizes ns: 128 for up to 4
// slices; for 5, 64 or 96 by the single-scene cost model over all the tiles
int mixed_group_tile_n(int slices, const std::vector<int>& ns);
// A = T^T T (lower tiles, mirrored) for lower-triangular n x n T from
// kGramSlices int8 slices of T's columns; buf holds mixed_gram_bytes(n) bytes,
// exps n + 64 ints. false: tensor-map encoding failed.
constexpr int kGramSlices = 7;
size_t mixed_gram_bytes(int n);
bool mixed_gram_lower_tri(const double* T, int n, int ld, int8_t* buf, int* exps, double* A, int lda, int* err,
                          cudaStream_t st);
void mixed_gemm_grouped(int slices, int nt, const MixedGemmJob* d_jobs, const int4* d_tiles, int ntiles,
                        cudaStream_t st);
// Y, te (optional): Y += te->coef * A while A is sliced, unless te->done.
// lower: A is lower triangular (the elements above its diagonal are not read).
void mixed_slice(const double* A, int lda, MixedOperand& op, cudaStream_t st, const int* skip = nullptr,
                 double* Y = nullptr, const TeState* te = nullptr, bool lower = false);
// C = P * X from the slices of P (a) and X (b); lower_only: tiles on/below the
// diagonal; mirror: the result's lower triangle is also written transposed
// into the upper one (a symmetric product needs no separate mirror pass).
void mixed_gemm(const MixedOperand& a, const MixedOperand& b, double* C, int ldc, unsigned long long* amax,
                bool lower_only, int* err, cudaStream_t st, const int* skip = nullptr, bool mirror = false);

// ---------------- svd.cu ----------------
// Scratch of the PSD pseudo-inverse (n x ld matrices and p x n blocks).
struct PinvBuffers {
    double *G, *T, *W, *Tt;        // shifted inverse, Cholesky-inverse scratch
    double *X, *Y, *MX;            // n x 32 subspace blocks
    double *H, *Wr, *S;            // 32 x 32
    double *theta, *res, *e;
    int* state;                    // counters of the tile tasks
    int* err;
    unsigned long long* dmax;
};
struct PinvInfo {
    int iterations, removed;
    double shift, residual, lambda_removed_max, lambda_kept_min;
};
size_t pinv_carve(char* base, int n, int ld, PinvBuffers& b);
// In place: M (n x ld, symmetric PSD) <- its pseudo-inverse without the
// remove_n smallest |eigenvalues| (remove_n >= 0) or without those with
// |eigenvalue| <= eps (remove_n == -1). Synchronises the stream.
int pinv_psd(double* M, int n, int ld, int remove_n, double eps, const PinvBuffers& b, cudaStream_t sm,
             PinvInfo* info);
// SVD_QR_ITERATION / SVD_DEVIDE_AND_CONQUER of computeCovariances; ev: 6 events.
size_t svd_workspace_bytes(int C, int P, int nobs, bool host_io, long long nnz, int nrows);
int svd_pipeline(char* ws, const unc_options* o, int num_rows, long long nnz, const int* rows, const int* cols,
                 const double* vals, double* cam_unc, double* pt_unc, bool host_io, unc_statistic* st,
                 cudaEvent_t* ev, cudaStream_t sm);

// ---------------- jacobian.cu ----------------
// Analytic reprojection Jacobian of a scene in the reference CRS layout
// (rows: 2 * num_obs + 1, cols / vals: 24 per observation).
int launch_scene_jacobian(int num_cams, int num_points, int num_obs, const double* cams, const double* pts,
                          const int* obs_cam, const int* obs_pt, int* rows, int* cols, double* vals, int* err,
                          cudaStream_t st);

// ---------------- points.cu ----------------
void launch_point_cov(const SceneDev& s, const double* sig, double* pt_unc, cudaStream_t st);
void prepare_point_kernels();  // kernel attributes (before any stream capture)

}  // namespace unc
