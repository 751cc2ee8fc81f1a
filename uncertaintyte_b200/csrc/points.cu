// points.cu - fused point-covariance kernel (sm_100a).
//
// Replaces the per-point loop of uncertaintyTE (compute.cpp:517-527 with
// findCams2Point :370-380, composeCams2PointJacobian :382-420,
// composeCamCovariances :422-441, fillPtUnc2OutArray :443-455):
//
//   Sigma_pt = pinv(A) * B * Sigma * B^T * pinv(A)^T
//
// with A = stacked 2x3 point Jacobians (unscaled), B = [J_cam,o | -I2] per
// observation and Sigma = blockdiag(Sigma_cam(o), I2), Sigma_cam the unscaled
// 9x9 diagonal block of the inverse (block-diagonal: the reference drops
// cross-camera terms). With pinv(A) = D^+ A^T, D = A^T A, this is exactly
//
//   Sigma_pt = D^+ + D^+ (sum_o W_o^T Sigma_cam(o) W_o) D^+,   W_o = J_cam,o^T A_o
//
// in two steps: per observation the six values of W_o^T Sigma_cam(o) W_o, by
// camera tiles (the camera's block in shared memory, the records staged), and
// per point the sum of its observations' six values and the 3 x 3 algebra. No
// 2n x 11n matrices, no O(P*obs) scan (the reference rescans every Jacobian row
// per point, :393).
#include "obs_tiles.cuh"

namespace unc {

// One thread per observation of a camera tile: S = W^T Sigma W (symmetric: 00 01
// 02 11 12 22) by position. Gathering the camera's 81 values per observation
// instead cost as many cache lines as there are lanes on every load (100 us for
// 342k observations, of which the records' bytes are 15).
constexpr size_t kSigTileSmem = sizeof(double) * kObsTile * kRecStride;
__global__ void __launch_bounds__(kObsTile, 2)
    k_camera_sig_tiles(int num_cams, const double* __restrict__ J, const int* __restrict__ cam_ptr,
                       const int* __restrict__ cam_obs, const double* __restrict__ sig, double* __restrict__ S) {
    extern __shared__ __align__(16) double sj[];
    __shared__ int ids[kObsTile];
    __shared__ double sg[81];
    ObsTile tile;
    if (!find_tile(cam_ptr, num_cams, blockIdx.x, tile)) return;
    const int n = tile.end - tile.begin, t = threadIdx.x;
    if (t < 81) sg[t] = sig[81L * tile.cam + t];
    stage_records(sj, ids, J, cam_obs, tile);
    if (t >= n) return;
    const double* r = sj + t * kRecStride;
    double W[9][3];
    {
        const double a0 = r[9], a1 = r[10], a2 = r[11], b0 = r[21], b1 = r[22], b2 = r[23];
#pragma unroll
        for (int j = 0; j < 9; ++j) {
            const double u = r[j], v = r[12 + j];
            W[j][0] = u * a0 + v * b0;
            W[j][1] = u * a1 + v * b1;
            W[j][2] = u * a2 + v * b2;
        }
    }
    double s00 = 0, s01 = 0, s02 = 0, s11 = 0, s12 = 0, s22 = 0;
#pragma unroll
    for (int j = 0; j < 9; ++j) {
        double t0 = 0, t1 = 0, t2 = 0;  // (Sigma W)(j, :)
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const double x = sg[9 * j + k];
            t0 = fma(x, W[k][0], t0);
            t1 = fma(x, W[k][1], t1);
            t2 = fma(x, W[k][2], t2);
        }
        s00 = fma(W[j][0], t0, s00);
        s01 = fma(W[j][0], t1, s01);
        s02 = fma(W[j][0], t2, s02);
        s11 = fma(W[j][1], t1, s11);
        s12 = fma(W[j][1], t2, s12);
        s22 = fma(W[j][2], t2, s22);
    }
    double2* out = reinterpret_cast<double2*>(S + 6L * (tile.begin + t));
    out[0] = make_double2(s00, s01);
    out[1] = make_double2(s02, s11);
    out[2] = make_double2(s12, s22);
}

// Pseudo-inverse of a symmetric PSD 3x3 (a00 a01 a02 a11 a12 a22) through a
// cyclic Jacobi eigen-decomposition. Eigenvalues below 64*eps*max are
// dropped (rank-deficient D when a point has a single observation).
__device__ void sym3_pinv(const double in[6], double out[3][3]) {
    double a[3][3] = {{in[0], in[1], in[2]}, {in[1], in[3], in[4]}, {in[2], in[4], in[5]}};
    double v[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
    for (int sweep = 0; sweep < 12; ++sweep) {
        double off = fabs(a[0][1]) + fabs(a[0][2]) + fabs(a[1][2]);
        double dia = fabs(a[0][0]) + fabs(a[1][1]) + fabs(a[2][2]);
        if (off <= 1e-300 || off < dia * 1e-18) break;
#pragma unroll
        for (int pq = 0; pq < 3; ++pq) {
            const int p = pq == 2 ? 1 : 0, q = pq == 0 ? 1 : 2;
            double apq = a[p][q];
            if (apq == 0.0) continue;
            double theta = (a[q][q] - a[p][p]) / (2.0 * apq);
            double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
            double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                double akp = a[k][p], akq = a[k][q];
                a[k][p] = c * akp - s * akq;
                a[k][q] = s * akp + c * akq;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                double apk = a[p][k], aqk = a[q][k];
                a[p][k] = c * apk - s * aqk;
                a[q][k] = s * apk + c * aqk;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                double vkp = v[k][p], vkq = v[k][q];
                v[k][p] = c * vkp - s * vkq;
                v[k][q] = s * vkp + c * vkq;
            }
        }
    }
    double w[3] = {a[0][0], a[1][1], a[2][2]};
    double wmax = fmax(fabs(w[0]), fmax(fabs(w[1]), fabs(w[2])));
    double iw[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) iw[k] = (w[k] > 64.0 * 2.220446049250313e-16 * wmax) ? 1.0 / w[k] : 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            out[i][j] = v[i][0] * v[j][0] * iw[0] + v[i][1] * v[j][1] * iw[1] + v[i][2] * v[j][2] * iw[2];
}

// One thread per point: its observations' S in list order, then the algebra.
__global__ void __launch_bounds__(128) k_point_cov(int num_points, int3 fix, int has_fix, const int* __restrict__ pt_ptr,
                                                   const int2* __restrict__ pt_list, const double* __restrict__ So,
                                                   const double* __restrict__ Vraw, double* __restrict__ pt_unc) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= num_points) return;
    if (has_fix && (p == fix.x || p == fix.y || p == fix.z)) return;  // fixed points are skipped
    double* out = pt_unc + 6L * p;
    const int b = pt_ptr[p], e = pt_ptr[p + 1];
    if (b == e || e - b > kSchurMaxList) {  // pinv of an empty A: zero covariance; a refused point's list is not there
        out[0] = out[1] = out[2] = out[3] = out[4] = out[5] = 0.0;
        return;
    }
    double s6[6] = {0, 0, 0, 0, 0, 0};
    for (int i0 = b; i0 < e; i0 += 4) {  // four records in flight
        double2 x[4][3];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double2* src = reinterpret_cast<const double2*>(So + 6L * (i0 + q < e ? pt_list[i0 + q].x : 0));
#pragma unroll
            for (int k = 0; k < 3; ++k) x[q][k] = i0 + q < e ? __ldg(src + k) : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                s6[2 * k] += x[q][k].x;
                s6[2 * k + 1] += x[q][k].y;
            }
    }
    const double S[3][3] = {{s6[0], s6[1], s6[2]}, {s6[1], s6[3], s6[4]}, {s6[2], s6[4], s6[5]}};
    double Dp[3][3];
    sym3_pinv(Vraw + 6L * p, Dp);
    // Sigma_pt = D^+ + D^+ S D^+
    double T[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) T[i][j] = S[i][0] * Dp[0][j] + S[i][1] * Dp[1][j] + S[i][2] * Dp[2][j];
    double R[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            R[i][j] = Dp[i][j] + Dp[i][0] * T[0][j] + Dp[i][1] * T[1][j] + Dp[i][2] * T[2][j];
    out[0] = R[0][0];
    out[1] = R[0][1];
    out[2] = R[0][2];
    out[3] = R[1][1];
    out[4] = R[1][2];
    out[5] = R[2][2];
}

void prepare_point_kernels() {
    static std::atomic<unsigned long long> attr{0};
    once_per_device(attr, [] {
        return cudaFuncSetAttribute(k_camera_sig_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSigTileSmem) ==
               cudaSuccess;
    });
}

void launch_point_cov(const SceneDev& s, const double* sig, double* pt_unc, cudaStream_t st) {
    if (s.num_points == 0) return;
    prepare_point_kernels();
    int3 fix = make_int3(s.fix[0], s.fix[1], s.fix[2]);
    double* So = s.Q;  // the Q records are not needed any more
    k_camera_sig_tiles<<<(unsigned)camera_tile_slots(s.num_cams, s.num_obs), kObsTile, kSigTileSmem, st>>>(
        s.num_cams, s.J, s.cam_ptr, s.cam_obs, sig, So);
    k_point_cov<<<(s.num_points + 127) / 128, 128, 0, st>>>(s.num_points, fix, s.has_fix, s.pt_ptr, s.pt_list, So, s.Vraw,
                                                            pt_unc);
    count_launch(2);
}

}  // namespace unc
