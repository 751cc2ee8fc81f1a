// rotation.cuh - the rotation of a symmetric 2 x 2 (Golub & Van Loan): c, s and t = s / c
// with a_pq cleared by (x, y) -> (c x - s y, s x + c y) on columns and rows p, q.
#pragma once

namespace unc {

// The angle from the tangent: entries so large or small that their squares leave the
// FP64 range.
__device__ __noinline__ inline void rotation_by_tangent(double d, double h, double& c, double& s, double& t) {
    const double th = d / h;
    t = fabs(th) > 1e100 ? 0.5 / th : (th >= 0.0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
    c = 1.0 / sqrt(t * t + 1.0);
    s = t * c;
}

// False (nothing to do) when |a_pq| <= 1e-17 sqrt(|a_pp a_qq|). The chain of dependent
// rotations bounds the kernels that use it, so a rotation takes two reciprocal square
// roots and no division: with d = a_qq - a_pp, h = 2 a_pq and r = 1 / sqrt(d^2 + h^2),
//   cos^2 = x = (1 + |d| r) / 2,  c = x / sqrt(x),  |s| = |h| r / (2 sqrt(x)).
__device__ __forceinline__ bool sym_rotation(double app, double aqq, double apq, double& c, double& s, double& t) {
    const double pr = fabs(app * aqq);
    const bool small = fabs(apq) > 1e-140 ? apq * apq <= 1e-34 * pr : fabs(apq) <= 1e-17 * sqrt(pr);
    if (apq == 0.0 || small) return false;
    const double d = aqq - app, h = 2.0 * apq, m = fma(d, d, h * h);
    if (m > 1e-280 && m < 1e280) {
        const double r = rsqrt(m), x = fma(0.5 * fabs(d), r, 0.5), rs = rsqrt(x);
        c = x * rs;
        s = 0.5 * fabs(h) * r * rs;
        if (d != 0.0 && (d < 0.0) != (h < 0.0)) s = -s;
        t = s * rs;
    } else {
        rotation_by_tangent(d, h, c, s, t);
    }
    return true;
}

}  // namespace unc
