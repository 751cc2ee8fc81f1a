// accessors.cu - batched eigen-decompositions of the covariance blocks behind
// the Uncertainty accessors (uncertainty.cpp:74-183: eigenvalues of every
// camera and point block, sorted descending, and eigenvectors of the point
// blocks and of the camera-centre 3 x 3 sub-blocks). The reference runs one
// Eigen::EigenSolver per block on the host; here one to nine lanes own one block (k_block_eigen).
//
// Input: packed upper triangles (row-major, i <= j) of src x src blocks
// (45 values for src = 9, 6 for src = 3); the sub-block [off, off + dim) of each
// is decomposed. Output: dim eigenvalues per block in descending order and the
// matching unit eigenvectors, column c of block b at vectors[b*dim*dim + c*dim].
// Method: cyclic Jacobi rotations (Golub & Van Loan, symmetric Schur 2 x 2),
// off-diagonal entries below 1e-17 sqrt(|a_pp a_qq|) left alone; eigenvector
// signs are arbitrary (as with the reference's EigenSolver).
#include "../../include/uncte.h"
#include "internal.h"
#include "rotation.cuh"

namespace unc {
namespace {

constexpr int kMaxDim = 9;

// One D x D block on L lanes, everything in registers: every lane of a block
// carries the whole upper triangle and applies every rotation to it, so the
// rotations need no shared memory, shuffle or barrier; the rows of V are dealt
// to the lanes (D / L each). The chain of dependent rotations bounds the
// kernel. The order is the cyclic one by rows, from which the signs of the vectors
// follow. Rounds of a round-robin tournament, their angles found side by side, took
// 65 us for 200 9 x 9 blocks against 84, but gave other signs (pairs that share an
// index change their order there; walking them by p + q would not change it).
template <int D, int L>
__global__ void __launch_bounds__(128) k_block_eigen(const double* __restrict__ packed, int nblk, int src, int off,
                                                     double* vals, double* vecs) {
    static_assert(D % L == 0, "whole rows of V per lane");
    constexpr int R = D / L, kPerWarp = 32 / L;
    const int lane = threadIdx.x & 31, part = lane % L;
    const long blk = ((long)blockIdx.x * (128 / 32) + (threadIdx.x >> 5)) * kPerWarp + lane / L;
    if (lane >= L * kPerWarp || blk >= nblk) return;
    const double* in = packed + blk * (src * (src + 1) / 2);
    double a[D][D], v[R][D];  // a: i <= j used
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
        for (int j = i; j < D; ++j) {
            const int r = off + i;  // upper-triangle index of (off + i, off + j)
            a[i][j] = __ldg(in + r * src - r * (r - 1) / 2 + (j - i));
        }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < D; ++j) v[r][j] = part * R + r == j ? 1.0 : 0.0;
    for (int sweep = 0; sweep < 50; ++sweep) {
        double off2 = 0.0, dg = 0.0;
#pragma unroll
        for (int i = 0; i < D; ++i) {
            dg += a[i][i] * a[i][i];
#pragma unroll
            for (int j = i + 1; j < D; ++j) off2 += a[i][j] * a[i][j];
        }
        if (off2 <= 1e-30 * dg) break;
#pragma unroll
        for (int p = 0; p < D - 1; ++p)
#pragma unroll
            for (int q = p + 1; q < D; ++q) {
                const double apq = a[p][q], app = a[p][p], aqq = a[q][q];
                double c, s, t;
                if (!sym_rotation(app, aqq, apq, c, s, t)) continue;
                a[p][p] = fma(-t, apq, app);
                a[q][q] = fma(t, apq, aqq);
                a[p][q] = 0.0;
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    if (k == p || k == q) continue;
                    double& y = a[k < p ? k : p][k < p ? p : k];
                    double& z = a[k < q ? k : q][k < q ? q : k];
                    const double yk = y, zk = z;
                    y = c * yk - s * zk;
                    z = s * yk + c * zk;
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const double x = v[r][p], y = v[r][q];
                    v[r][p] = c * x - s * y;
                    v[r][q] = s * x + c * y;
                }
            }
    }
    double* const w = vals + blk * D;
    double* const e = vecs ? vecs + blk * (D * D) : nullptr;
    double key[D];  // a NaN counts as infinity, so that the ranks are a permutation and every place is written
#pragma unroll
    for (int j = 0; j < D; ++j) key[j] = a[j][j] == a[j][j] ? a[j][j] : __longlong_as_double(0x7ff0000000000000LL);
#pragma unroll
    for (int j = 0; j < D; ++j) {  // descending order, ties by index
        int rank = 0;
#pragma unroll
        for (int i = 0; i < D; ++i) rank += (key[i] > key[j]) || (key[i] == key[j] && i < j);
        if (part == j / R) w[rank] = a[j][j];
        if (e) {
#pragma unroll
            for (int r = 0; r < R; ++r) e[rank * D + part * R + r] = v[r][j];
        }
    }
}

// Lanes per block: one up to 3 x 3 (V fits beside the block, and there are as
// many blocks as points), one per row above.
template <int D>
void launch_block_eigen(const double* packed, int nblk, int src, int off, double* vals, double* vecs,
                        cudaStream_t sm) {
    constexpr int L = D <= 3 ? 1 : D;
    const long per_cta = 4 * (32 / L);
    k_block_eigen<D, L><<<(unsigned)((nblk + per_cta - 1) / per_cta), 128, 0, sm>>>(packed, nblk, src, off, vals, vecs);
    count_launch();
}

}  // namespace
}  // namespace unc

using namespace unc;

extern "C" int unc_block_eigen_device(const double* d_packed, int num_blocks, int block_params, int sub_offset,
                                      int sub_dim, double* d_values, double* d_vectors, void* stream) {
    g_last_error.clear();
    if (num_blocks < 0 || block_params < 1 || block_params > kMaxDim || sub_offset < 0 || sub_dim < 1 ||
        sub_offset + sub_dim > block_params || (num_blocks && (!d_packed || !d_values))) {
        g_last_error = "unc_block_eigen_device: bad arguments (block_params <= 9, sub-block inside the block)";
        return UNC_ERR_INVALID_ARG;
    }
    if (num_blocks == 0) return UNC_OK;
    cudaStream_t sm = (cudaStream_t)stream;
    using Launch = void (*)(const double*, int, int, int, double*, double*, cudaStream_t);
    static constexpr Launch by_dim[kMaxDim] = {launch_block_eigen<1>, launch_block_eigen<2>, launch_block_eigen<3>,
                                               launch_block_eigen<4>, launch_block_eigen<5>, launch_block_eigen<6>,
                                               launch_block_eigen<7>, launch_block_eigen<8>, launch_block_eigen<9>};
    by_dim[sub_dim - 1](d_packed, num_blocks, block_params, sub_offset, d_values, d_vectors, sm);
    cudaError_t e = cudaStreamSynchronize(sm);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) {
        g_last_error = std::string("unc_block_eigen_device: ") + cudaGetErrorString(e);
        return UNC_ERR_CUDA;
    }
    return UNC_OK;
}

extern "C" int unc_block_eigen(const double* packed, int num_blocks, int block_params, int sub_offset, int sub_dim,
                               double* values, double* vectors) {
    g_last_error.clear();
    if (num_blocks < 0 || block_params < 1 || block_params > kMaxDim || sub_offset < 0 || sub_dim < 1 ||
        sub_offset + sub_dim > block_params || (num_blocks && (!packed || !values))) {
        g_last_error = "unc_block_eigen: bad arguments (block_params <= 9, sub-block inside the block)";
        return UNC_ERR_INVALID_ARG;
    }
    if (num_blocks == 0) return UNC_OK;
    const size_t nin = (size_t)num_blocks * block_params * (block_params + 1) / 2;
    const size_t nv = (size_t)num_blocks * sub_dim, nvec = vectors ? nv * sub_dim : 0;
    Scratch mem;
    cudaError_t e = mem.alloc(sizeof(double) * (nin + nv + nvec), nullptr);
    double* d = static_cast<double*>(mem.p);
    if (e != cudaSuccess) {
        g_last_error = std::string("unc_block_eigen: ") + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? UNC_ERR_OUT_OF_MEMORY : UNC_ERR_CUDA;
    }
    e = cudaMemcpy(d, packed, sizeof(double) * nin, cudaMemcpyHostToDevice);
    int rc = UNC_OK;
    if (e == cudaSuccess)
        rc = unc_block_eigen_device(d, num_blocks, block_params, sub_offset, sub_dim, d + nin,
                                    vectors ? d + nin + nv : nullptr, nullptr);
    if (e == cudaSuccess && rc == UNC_OK) e = cudaMemcpy(values, d + nin, sizeof(double) * nv, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && rc == UNC_OK && vectors)
        e = cudaMemcpy(vectors, d + nin + nv, sizeof(double) * nvec, cudaMemcpyDeviceToHost);
    if (rc != UNC_OK) return rc;
    if (e != cudaSuccess) {
        g_last_error = std::string("unc_block_eigen: ") + cudaGetErrorString(e);
        return UNC_ERR_CUDA;
    }
    return UNC_OK;
}
