// Least-squares 3-D line fit of one detector record, shared by the host
// reader (MutoFile::getMuonData) and the batched GPU fit (fit.cu).
//
// The reference fits each half of a record (src/MutoFile.cpp:248-304) with
// Eigen's JacobiSVD of the centred hits and takes the first right singular
// vector as the direction.  That vector is the principal axis of the hits'
// 3x3 scatter matrix, found here by squaring the matrix until one axis is left
// (hits along a line), or else by cyclic Jacobi rotations on the symmetric
// matrix (Golub & Van Loan, "Matrix Computations", sec. 8.5), then oriented
// with d_z > 0 (the SVD leaves the sign open).  The point is
// the line at the layer next to the grid: pin on layer n_middle-1, pout on
// layer n_middle.
//
// Every product and sum goes through fm/fa/fs, which round each operation
// on its own on the device and on the host (built without contraction), so
// the two builds give the same bits.
#pragma once

#include <cmath>
#include <cstdint>

#include "../../include/muto_gb300.h"

#ifdef __CUDACC__
#define MUTO_FIT_HD __host__ __device__
#else
#define MUTO_FIT_HD
#endif

namespace muto {
namespace fit {

constexpr int kMaxLayers = 64;  // detector layers a record may hold

MUTO_FIT_HD inline double fm(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}
MUTO_FIT_HD inline double fa(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dadd_rn(a, b);
#else
    return a + b;
#endif
}
MUTO_FIT_HD inline double fs(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dsub_rn(a, b);
#else
    return a - b;
#endif
}

// Unit eigenvector of the largest eigenvalue of the symmetric a (which the
// rotations overwrite).
MUTO_FIT_HD inline void principal_axis(double a[3][3], double* out) {
    double v[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
    for (int sweep = 0; sweep < 50; ++sweep) {
        const double off = fa(fa(fm(a[0][1], a[0][1]), fm(a[0][2], a[0][2])), fm(a[1][2], a[1][2]));
        const double diag = fa(fa(fm(a[0][0], a[0][0]), fm(a[1][1], a[1][1])), fm(a[2][2], a[2][2]));
        if (off == 0.0 || off < fm(1e-30, diag)) break;
        for (int p = 0; p < 2; ++p)
            for (int q = p + 1; q < 3; ++q) {
                if (a[p][q] == 0.0) continue;
                const double theta = fs(a[q][q], a[p][p]) / fm(2.0, a[p][q]);
                const double t = (theta >= 0 ? 1.0 : -1.0) / fa(fabs(theta), sqrt(fa(fm(theta, theta), 1.0)));
                const double c = 1.0 / sqrt(fa(fm(t, t), 1.0)), s = fm(t, c);
                for (int k = 0; k < 3; ++k) {  // A <- A J
                    const double akp = a[k][p], akq = a[k][q];
                    a[k][p] = fs(fm(c, akp), fm(s, akq));
                    a[k][q] = fa(fm(s, akp), fm(c, akq));
                }
                for (int k = 0; k < 3; ++k) {  // A <- J^T A
                    const double apk = a[p][k], aqk = a[q][k];
                    a[p][k] = fs(fm(c, apk), fm(s, aqk));
                    a[q][k] = fa(fm(s, apk), fm(c, aqk));
                }
                for (int k = 0; k < 3; ++k) {  // V <- V J
                    const double vkp = v[k][p], vkq = v[k][q];
                    v[k][p] = fs(fm(c, vkp), fm(s, vkq));
                    v[k][q] = fa(fm(s, vkp), fm(c, vkq));
                }
            }
    }
    int best = 0;
    for (int k = 1; k < 3; ++k)
        if (a[k][k] > a[best][best]) best = k;
    for (int k = 0; k < 3; ++k) out[k] = v[k][best];
}

// The same axis, not normalised, where one eigenvalue stands out: the eigenvalue
// ratio of a's powers falls as the square of the power before, so a column of a^4
// is the axis to the last bit for hits along a line (ratio up to 9e-5), of a^8 and
// a^16 for ratios up to 0.009 and 0.09.  A squaring takes 24 operations and a
// rotation above 110, three to five sweeps of three being needed.  A matrix's
// ratio (e2 = the sum of the 2x2 principal minors, over its trace squared) comes
// with its square: trace(a)^2 - trace(a^2) = 2 e2.  Refused, for the rotations to
// decide: no axis that stands out, powers that leave the range, axes within 1e-6
// of the horizontal (whose sign the orientation does not settle), inf and NaN.
MUTO_FIT_HD inline bool outstanding_axis(const double a[3][3], double* out) {
    double m00 = a[0][0], m01 = a[0][1], m02 = a[0][2], m11 = a[1][1], m12 = a[1][2], m22 = a[2][2];
    bool alone = false;
    for (int k = 0; k < 4 && !alone; ++k) {
        const double q01 = fm(m01, m01), q02 = fm(m02, m02), q12 = fm(m12, m12);
        const double n00 = fa(fa(fm(m00, m00), q01), q02);
        const double n11 = fa(fa(fm(m11, m11), q01), q12);
        const double n22 = fa(fa(fm(m22, m22), q02), q12);
        const double n01 = fa(fm(m01, fa(m00, m11)), fm(m02, m12));
        const double n02 = fa(fm(m02, fa(m00, m22)), fm(m01, m12));
        const double n12 = fa(fm(m12, fa(m11, m22)), fm(m01, m02));
        const double tr = fa(fa(m00, m11), m22), tr2 = fm(tr, tr);
        alone = fs(tr2, fa(fa(n00, n11), n22)) <= fm(1.4901161193847656e-08, tr2);  // 2^-26: the square's ratio is below 2^-54
        m00 = n00, m01 = n01, m02 = n02, m11 = n11, m12 = n12, m22 = n22;
    }
    double top;
    if (m22 >= m00 && m22 >= m11) {
        top = m22;
        out[0] = m02, out[1] = m12, out[2] = m22;
    } else if (m11 >= m00) {
        top = m11;
        out[0] = m01, out[1] = m11, out[2] = m12;
    } else {
        top = m00;
        out[0] = m00, out[1] = m01, out[2] = m02;
    }
    return alone && top >= 1e-140 && top <= 1e140 && fabs(out[2]) >= fm(1e-6, top);
}

// Centroid c and unit direction d (d_z >= 0) of the n hits (x, y, z);
// src/MutoFile.cpp:262-276 and :287-299.
MUTO_FIT_HD inline void fit_line(const double* x, const double* y, const double* z, int n, double* c, double* d) {
    c[0] = c[1] = c[2] = 0.0;
    for (int i = 0; i < n; ++i) {
        c[0] = fa(c[0], x[i]);
        c[1] = fa(c[1], y[i]);
        c[2] = fa(c[2], z[i]);
    }
    const double nn = static_cast<double>(n > 0 ? n : 1);
    for (int k = 0; k < 3; ++k) c[k] = c[k] / nn;
    double a[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    for (int i = 0; i < n; ++i) {
        const double r[3] = {fs(x[i], c[0]), fs(y[i], c[1]), fs(z[i], c[2])};
        for (int p = 0; p < 3; ++p)
            for (int q = p; q < 3; ++q) a[p][q] = fa(a[p][q], fm(r[p], r[q]));
    }
    a[1][0] = a[0][1], a[2][0] = a[0][2], a[2][1] = a[1][2];
    if (!outstanding_axis(a, d)) principal_axis(a, d);
    const double nrm = sqrt(fa(fa(fm(d[0], d[0]), fm(d[1], d[1])), fm(d[2], d[2])));
    if (!(nrm > 0)) {
        d[0] = d[1] = 0.0;
        d[2] = 1.0;
        return;
    }
    const double sgn = d[2] < 0 ? -1.0 : 1.0;
    for (int k = 0; k < 3; ++k) d[k] = fm(sgn, d[k]) / nrm;
}

// One record {ein, x0, y0, ..., x_{nz-1}, y_{nz-1}, eout} (nz <= kMaxLayers)
// to its track (src/MutoFile.cpp:248-304).  Returns false, writing nothing,
// for a record holding a NaN (src/MutoFile.cpp:71-76 drops those).
template <typename T>
MUTO_FIT_HD inline bool fit_record(const T* rec, const double* zl, int nz, int n_middle, muto_ray* out) {
    double hx[kMaxLayers], hy[kMaxLayers];
    const double ein = static_cast<double>(rec[0]);
    const double eout = static_cast<double>(rec[2 * nz + 1]);
    bool nan = ein != ein || eout != eout;
    for (int i = 0; i < nz; ++i) {
        hx[i] = static_cast<double>(rec[1 + 2 * i]);
        hy[i] = static_cast<double>(rec[2 + 2 * i]);
        nan = nan || hx[i] != hx[i] || hy[i] != hy[i];
    }
    if (nan) return false;
    muto_ray r;
    r.ein = ein;
    r.eout = eout;
    double c[3], d[3];
    fit_line(hx, hy, zl, n_middle, c, d);  // upper layers
    double t = fs(zl[n_middle - 1], c[2]) / d[2];
    for (int k = 0; k < 3; ++k) r.din[k] = d[k];
    r.pin[0] = fa(fm(t, d[0]), c[0]);
    r.pin[1] = fa(fm(t, d[1]), c[1]);
    r.pin[2] = zl[n_middle - 1];
    fit_line(hx + n_middle, hy + n_middle, zl + n_middle, nz - n_middle, c, d);  // lower layers
    t = fs(zl[n_middle], c[2]) / d[2];
    for (int k = 0; k < 3; ++k) r.dout[k] = d[k];
    r.pout[0] = fa(fm(t, d[0]), c[0]);
    r.pout[1] = fa(fm(t, d[1]), c[1]);
    r.pout[2] = zl[n_middle];
    *out = r;
    return true;
}

}  // namespace fit
}  // namespace muto
