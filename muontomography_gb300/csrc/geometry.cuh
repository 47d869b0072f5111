// Device geometry for the reconstruction path: Siddon/Jacobs voxel walk,
// point of closest approach, projected scattering angles and displacement.
//
// Bit-exactness.  The voxel lists and PoCA voxels must equal the reference's
// (src/MutoSiddon.cpp, src/MutoPoCA.cpp, src/MutoMLSD.cpp) bit for bit, so
// every FP64 operation on those paths goes through the _rn intrinsics, which
// nvcc never contracts into FMA, in the reference's evaluation order.  The
// reference's `static_cast<unsigned>(double)` is given its x86-64 GCC meaning
// (truncate to int64, keep the low 32 bits), which differs from the device's
// saturating conversion for values <= -1.
#pragma once

#include <cstdint>
#include "../../include/muto_gb300.h"

namespace muto {

struct DevGrid {
    uint32_t n[3];
    double lo[3];
    double w[3];
    double rw[3];   // 1 / w
    int ordinary;   // every lo and w of a magnitude for which quotient() is exact
};

inline DevGrid make_dev_grid(const muto_grid& g) {
    DevGrid d;
    d.n[0] = g.nx; d.n[1] = g.ny; d.n[2] = g.nz;
    d.lo[0] = g.x_min; d.lo[1] = g.y_min; d.lo[2] = g.z_min;
    d.w[0] = g.dx; d.w[1] = g.dy; d.w[2] = g.dz;
    d.ordinary = 1;
    for (int k = 0; k < 3; ++k) {
        d.rw[k] = 1.0 / d.w[k];
        if (!(d.w[k] > 1e-100 && d.w[k] < 1e100 && d.lo[k] > -1e100 && d.lo[k] < 1e100)) d.ordinary = 0;
    }
    return d;
}

__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }
// a / b, correctly rounded, from y = 1 / b correctly rounded: the product a y
// corrected by its remainder twice (Markstein's theorem: the second correction of
// a faithful quotient is the rounded quotient; the remainders are exact).  Five
// FP64 operations where several quotients share a divisor, against about twenty
// for a division; for operands within 1e-100 .. 1e100 (or a = 0), so that no
// product or remainder leaves the range.
__device__ __forceinline__ double quotient(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    const double q1 = __fma_rn(__fma_rn(-q, b, a), y, q);
    return __fma_rn(__fma_rn(-q1, b, a), y, q1);
}
__device__ __forceinline__ double positive_zero(double x) {  // -0.0 as 0.0
    const long long b = __double_as_longlong(x);
    return __longlong_as_double((b << 1) == 0 ? 0ll : b);
}
__device__ __forceinline__ bool ordinary(double x) {  // finite and below about 1e100
    return (__double2hiint(x) & 0x7fffffff) < 0x54b00000;
}
// std::max / std::min argument semantics
__device__ __forceinline__ double smax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double smin(double a, double b) { return (b < a) ? b : a; }

// x86-64 GCC `static_cast<unsigned int>(double)`
__device__ __forceinline__ uint32_t u32_cast_x86(double v) {
    if (!(v > -9223372036854775808.0 && v < 9223372036854775808.0)) return 0u;
    return static_cast<uint32_t>(static_cast<unsigned long long>(__double2ll_rz(v)));
}

// Eigen Vector3::dot order: (a0*b0 + a1*b1) + a2*b2
__device__ __forceinline__ double dot3(const double* a, const double* b) {
    return dadd(dadd(dmul(a[0], b[0]), dmul(a[1], b[1])), dmul(a[2], b[2]));
}

// Order of doubles through their bit patterns: for two values whose sign
// bits are clear (non-negative, and not -0.0) the signed 64-bit integers
// order exactly as the doubles do, so the walk's comparisons can run on the
// integer pipe; it falls back to FP64 compares when a sign bit is set.
__device__ __forceinline__ long long dbits(double x) { return __double_as_longlong(x); }

// Upper bound on the steps of one walk: every step crosses one plane of the
// grid, and a segment crosses each of the n+1 planes of an axis at most once.
__device__ __forceinline__ int siddon_step_bound(const DevGrid& g) {
    return static_cast<int>(g.n[0] + g.n[1] + g.n[2]) + 8;
}

// The lanes of a warp that walk paths, for __syncwarp between consecutive
// walks: a thread-per-path kernel calls this once at its start, with every
// lane of the warp present (no lane has returned yet) and `walks` true on the
// lanes that will make every one of the walks.  Without the sync, lanes that
// finish a walk early start the next one on their own and the warp's lanes
// no longer step together.
__device__ __forceinline__ unsigned walk_lanes(bool walks) { return __ballot_sync(0xffffffffu, walks); }

// Voxel walk of the segment p1 -> p2 (src/MutoSiddon.cpp:9-141).  For every
// voxel with a recorded length the sink is called as sink(ix, iy, iz, len).
// Returns the number of voxels, or -1 if the step bound was hit (never for a
// walk that ends, kept as a guard against a non-terminating loop).
// voxels a walk of a -> b can record: 1 + the index span on each axis of
// the endpoints clamped to the grid (the pieces on the grid lie between
// them), +2 per axis for rounding at either end
__device__ __forceinline__ uint32_t walk_bound(const DevGrid& g, const double* a, const double* b) {
    uint32_t n = 1;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float lo = static_cast<float>(g.lo[k]), w = static_cast<float>(g.w[k]);
        const float top = static_cast<float>(g.n[k] - 1);
        const float ia = fminf(fmaxf(floorf((static_cast<float>(a[k]) - lo) / w), 0.f), top);
        const float ib = fminf(fmaxf(floorf((static_cast<float>(b[k]) - lo) / w), 0.f), top);
        n += static_cast<uint32_t>(fabsf(ia - ib)) + 2u;
    }
    return n;
}

// A walk at its first crossings.
struct SiddonStart {
    uint32_t idx[3];   // the voxel
    int dir[3];        // its steps
    double an[3], da[3];  // next crossing and the distance to the one after, per axis
    double alpha, amax, seg;
};

// The steps of a walk (src/MutoSiddon.cpp:108-138) from the first crossings on.
// INTS: every value non-negative and finite, compared by bit pattern; three FP64
// operations a step (the crossing stepped to, the difference, the length).
// TWO: then the steps of the walk w2, with sink.second() in between; returns -1 if
// either walk hit its step bound.
template <bool INTS, bool TWO, class Sink>
__device__ __forceinline__ int siddon_steps(const DevGrid& g, const SiddonStart& w1, const SiddonStart& w2, Sink& sink) {
    const double eps = 1.0e-6;  // :19
    uint32_t idx[3] = {w1.idx[0], w1.idx[1], w1.idx[2]};
    int dir[3] = {w1.dir[0], w1.dir[1], w1.dir[2]};
    double an[3] = {w1.an[0], w1.an[1], w1.an[2]}, da[3] = {w1.da[0], w1.da[1], w1.da[2]};
    double amax = w1.amax, seg = w1.seg, alpha_last = w1.alpha;
    long long amax_b = dbits(amax);
    const long long eps_b = dbits(eps);
    int count = 0;
    int left = siddon_step_bound(g);
    bool more = INTS ? dbits(alpha_last) < amax_b : alpha_last < amax;
    bool first = TWO;
    auto go_on = [&] {  // to the second walk (moves alone)
        first = false;
        if constexpr (TWO) sink.second();
#pragma unroll
        for (int k = 0; k < 3; ++k) idx[k] = w2.idx[k], dir[k] = w2.dir[k], an[k] = w2.an[k], da[k] = w2.da[k];
        amax = w2.amax, seg = w2.seg, alpha_last = w2.alpha;
        amax_b = dbits(amax);
        left = siddon_step_bound(g);
        more = INTS ? dbits(alpha_last) < amax_b : alpha_last < amax;
    };
    if (TWO && !more) go_on();
    // The lanes of a warp that walk together step together: every iteration
    // ends with a ballot over the lanes still walking, which makes it a
    // reconvergence point (the three-way step below would otherwise let the
    // lanes drift apart for the rest of the walk, each then issuing its own
    // FP64 instructions).
    unsigned live = __activemask();
    live = __ballot_sync(live, more);
    while (more) {
        const uint32_t vx = idx[0], vy = idx[1], vz = idx[2];
        // min of the three next crossings, reference tie-break order
        bool t0, t1;
        if (INTS) {
            const long long b0 = dbits(an[0]), b1 = dbits(an[1]), b2 = dbits(an[2]);
            t0 = b0 < b1 && b0 < b2;
            t1 = b1 < b2;
        } else {
            t0 = an[0] < an[1] && an[0] < an[2];
            t1 = an[1] < an[2];
        }
        // the axis stepped, then one FP64 add for it: the lanes of a warp step
        // along different axes, and a branch per axis would issue the add
        // once per axis taken in the warp (selects are integer instructions)
        const int k = t0 ? 0 : (t1 ? 1 : 2);
        const double ak = k == 0 ? an[0] : (k == 1 ? an[1] : an[2]);
        const double dk = k == 0 ? da[0] : (k == 1 ? da[1] : da[2]);
        const double next = dadd(ak, dk);
        an[0] = k == 0 ? next : an[0];
        an[1] = k == 1 ? next : an[1];
        an[2] = k == 2 ? next : an[2];
        idx[0] += k == 0 ? static_cast<uint32_t>(dir[0]) : 0u;
        idx[1] += k == 1 ? static_cast<uint32_t>(dir[1]) : 0u;
        idx[2] += k == 2 ? static_cast<uint32_t>(dir[2]) : 0u;
        // not yet at the end: the next step's test, and min(alpha, amax) here
        const bool before = INTS ? dbits(ak) < amax_b : ak < amax;
        const double upto = INTS ? (before ? ak : amax) : smin(ak, amax);
        const double dalpha = dsub(upto, alpha_last);
        if (INTS ? eps_b < dbits(dalpha) : eps < dalpha) {  // eps is positive
            sink(vx, vy, vz, dmul(dalpha, seg));
            if (!TWO) ++count;
            alpha_last = ak;
        }
        more = before && --left > 0;  // the step bound: never for a walk that ends
        if (before && !more) count = -1;
        if (TWO && !more && first) go_on();
        live = __ballot_sync(live, more);
    }
    return count;
}

// ORDINARY: coordinates and grid of ordinary magnitudes (the divisions go
// through quotient, the steps' comparisons through integers where they can).
template <bool ORDINARY, class Sink>
__device__ __forceinline__ int siddon_walk_as(const DevGrid& g, const double* p1, const double* p2, Sink& sink);
// The walk's start: 1, or 0 if it misses the grid, or -2 where ORDINARY does not hold.
template <bool ORDINARY>
__device__ __forceinline__ int siddon_start(const DevGrid& g, const double* p1, const double* p2, SiddonStart& w);

// Anything else, and the rare walk with a negative crossing: out of line, the
// sink by value, so that the common walk's state stays in registers.
template <class Sink>
struct Walked {
    Sink sink;
    int count;
};
template <class Sink>
__device__ __noinline__ Walked<Sink> siddon_walk_any(DevGrid g, double3 a, double3 b, Sink sink) {
    const double p1[3] = {a.x, a.y, a.z}, p2[3] = {b.x, b.y, b.z};
    const int n = siddon_walk_as<false>(g, p1, p2, sink);
    return Walked<Sink>{sink, n};
}

template <class Sink>
__device__ __forceinline__ int siddon_walk(const DevGrid& g, const double* p1, const double* p2, Sink& sink) {
    int n = -2;
    if (g.ordinary && ordinary(p1[0]) && ordinary(p1[1]) && ordinary(p1[2]) && ordinary(p2[0]) && ordinary(p2[1]) &&
        ordinary(p2[2]))
        n = siddon_walk_as<true>(g, p1, p2, sink);
    if (n == -2) {
        const Walked<Sink> w = siddon_walk_any(g, make_double3(p1[0], p1[1], p1[2]), make_double3(p2[0], p2[1], p2[2]), sink);
        sink = w.sink;
        n = w.count;
    }
    return n;
}

template <bool ORDINARY>
__device__ __forceinline__ int siddon_start(const DevGrid& g, const double* p1, const double* p2, SiddonStart& w) {
    const double eps = 1.0e-6;  // :19
    double d[3], first[3], last[3], y[3];
    for (int k = 0; k < 3; ++k) d[k] = dsub(p2[k], p1[k]);
    const double seg = __dsqrt_rn(dot3(d, d));  // :14
#pragma unroll
    for (int k = 0; k < 3; ++k) {  // :25-48
        double a0 = -0.1, an = 1.1;
        const double hi = dadd(g.lo[k], dmul(g.w[k], static_cast<double>(g.n[k])));
        y[k] = 0.0;
        if (eps < fabs(d[k])) {
            if (ORDINARY) {
                y[k] = __drcp_rn(d[k]);
                a0 = quotient(dsub(g.lo[k], p1[k]), d[k], y[k]);
                an = quotient(dsub(hi, p1[k]), d[k], y[k]);
            } else {
                a0 = ddiv(dsub(g.lo[k], p1[k]), d[k]);
                an = ddiv(dsub(hi, p1[k]), d[k]);
            }
        } else if (p1[k] < g.lo[k] || hi <= p1[k]) {
            return 0;
        }
        first[k] = (an < a0) ? an : a0;
        last[k] = (an < a0) ? a0 : an;
    }
    const double amin = smax(smax(smax(first[0], first[1]), first[2]), 0.0);  // :50
    const double amax = smin(smin(smin(last[0], last[1]), last[2]), 1.0);     // :51
    if (amax <= amin) return 0;

    double alpha = amin;
    uint32_t(&idx)[3] = w.idx;
    int(&dir)[3] = w.dir;
    double(&da)[3] = w.da;
    double(&an)[3] = w.an;
#pragma unroll
    for (int k = 0; k < 3; ++k) {  // :62-81
        const double nudge = (d[k] <= 0) ? -eps : eps;
        const double at = dsub(dadd(dmul(alpha, d[k]), p1[k]), g.lo[k]);
        idx[k] = u32_cast_x86(dadd(ORDINARY ? quotient(at, g.w[k], g.rw[k]) : ddiv(at, g.w[k]), nudge));
        dir[k] = 0;
        da[k] = 0.0;
        if (eps < fabs(d[k])) {
            da[k] = ORDINARY ? quotient(g.w[k], fabs(d[k]), fabs(y[k])) : ddiv(g.w[k], fabs(d[k]));
            dir[k] = d[k] < 0 ? -1 : 1;
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {  // :85-103
        an[k] = 1.1;
        if (fabs(dsub(amin, first[k])) < eps) {
            an[k] = dadd(amin, da[k]);
        } else if (dir[k] != 0) {
            const double plane = dsub(dadd(dmul(static_cast<double>(idx[k]), g.w[k]), g.lo[k]), p1[k]);
            an[k] = dadd(ORDINARY ? quotient(plane, d[k], y[k]) : ddiv(plane, d[k]), dir[k] == 1 ? da[k] : 0.0);
        }
    }
    // Every crossing finite and every sign bit clear (the crossings only grow):
    // the steps' comparisons then run on the integer pipe.  A track that starts
    // on the grid's top plane has a first crossing of -0.0, which stands for 0.0
    // in every operation to come.
    alpha = positive_zero(alpha);
#pragma unroll
    for (int k = 0; k < 3; ++k) an[k] = positive_zero(an[k]);
    w.alpha = alpha;
    w.amax = amax;
    w.seg = seg;
    if (ORDINARY && !(isfinite(amax) && isfinite(an[0]) && isfinite(an[1]) && isfinite(an[2]) &&
                      (dbits(alpha) | dbits(amax) | dbits(an[0]) | dbits(an[1]) | dbits(an[2])) >= 0))
        return -2;
    return 1;
}

// (returns -2, before the sink has seen anything, where ORDINARY does not hold)
template <bool ORDINARY, class Sink>
__device__ __forceinline__ int siddon_walk_as(const DevGrid& g, const double* p1, const double* p2, Sink& sink) {
    SiddonStart w;
    const int st = siddon_start<ORDINARY>(g, p1, p2, w);
    return st <= 0 ? st : siddon_steps<ORDINARY, false>(g, w, w, sink);
}

// The walks p1 -> p2 and p2 -> p3, sink.second() in between; false if either hit
// its step bound.  Both starts are worked out first, so that a lane goes on to its
// second walk with moves alone while others are still on their first: a warp's
// steps are then the most of any lane's two walks together, not the most of the
// first and the most of the second, which for tracks that turn anywhere in the grid
// is up to twice as many.  2 M tracks through 256 x 256 x 128 voxels in the order of
// their lengths: 5.1 ms, 7.4 ms with the lanes in step after the first walk.
template <class Sink>
__device__ __forceinline__ bool siddon_walk_two(const DevGrid& g, const double* p1, const double* p2, const double* p3,
                                                Sink& sink) {
    if (g.ordinary && ordinary(p1[0]) && ordinary(p1[1]) && ordinary(p1[2]) && ordinary(p2[0]) && ordinary(p2[1]) &&
        ordinary(p2[2]) && ordinary(p3[0]) && ordinary(p3[1]) && ordinary(p3[2])) {
        SiddonStart w[2];
        int st[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            st[h] = siddon_start<true>(g, h ? p2 : p1, h ? p3 : p2, w[h]);
            if (st[h] == 0) {  // misses the grid: no steps
                w[h].alpha = w[h].amax = w[h].seg = 0.0;
#pragma unroll
                for (int k = 0; k < 3; ++k) w[h].idx[k] = 0, w[h].dir[k] = 0, w[h].an[k] = w[h].da[k] = 0.0;
            }
        }
        if (st[0] != -2 && st[1] != -2) return siddon_steps<true, true>(g, w[0], w[1], sink) >= 0;
    }
    const double3 a = make_double3(p1[0], p1[1], p1[2]), b = make_double3(p2[0], p2[1], p2[2]),
                  c = make_double3(p3[0], p3[1], p3[2]);
    const Walked<Sink> first = siddon_walk_any(g, a, b, sink);
    sink = first.sink;
    sink.second();
    const Walked<Sink> then = siddon_walk_any(g, b, c, sink);
    sink = then.sink;
    return first.count >= 0 && then.count >= 0;
}

// Point of closest approach of the in and out lines (src/MutoMLSD.cpp:328-348,
// src/MutoPoCA.cpp:192-213).  Returns true when the lines are not parallel.
__device__ __forceinline__ bool poca_point(const muto_ray& r, double eps, double* out) {
    double w0[3];
    for (int k = 0; k < 3; ++k) w0[k] = dsub(r.pin[k], r.pout[k]);
    const double a = dot3(r.din, r.din);
    const double b = dot3(r.din, r.dout);
    const double c = dot3(r.dout, r.dout);
    const double d = dot3(r.din, w0);
    const double e = dot3(r.dout, w0);
    const double den = dsub(dmul(a, c), dmul(b, b));
    if (fabs(den) < eps) {
        for (int k = 0; k < 3; ++k) out[k] = dmul(0.5, dadd(r.pin[k], r.pout[k]));
        return false;
    }
    const double ni = dsub(dmul(b, e), dmul(c, d)), no = dsub(dmul(a, e), dmul(b, d));
    double cin, cout;
    if (ordinary(ni) && ordinary(no) && ordinary(den) && fabs(den) > 1e-100) {
        const double y = __drcp_rn(den);
        cin = quotient(ni, den, y);
        cout = quotient(no, den, y);
    } else {
        cin = ddiv(ni, den);
        cout = ddiv(no, den);
    }
    for (int k = 0; k < 3; ++k)
        out[k] = dmul(0.5, dadd(dadd(dadd(r.pin[k], dmul(cin, r.din[k])), r.pout[k]), dmul(cout, r.dout[k])));
    return true;
}

// Projected scattering angles (src/MutoMLSD.cpp:350-354)
__device__ __forceinline__ void scat_angles(const double* d1, const double* d2, double* ax, double* ay) {
    *ax = dsub(atan2(d1[0], d1[2]), atan2(d2[0], d2[2]));
    *ay = dsub(atan2(d1[1], d1[2]), atan2(d2[1], d2[2]));
}

// PoCA mean squared angle (src/MutoPoCA.cpp:215-224)
__device__ __forceinline__ double scat_angle_square(const double* d1, const double* d2, double mag) {
    const double axz = dmul(dsub(atan2(d1[0], d1[2]), atan2(d2[0], d2[2])), mag);
    const double ayz = dmul(dsub(atan2(d1[1], d1[2]), atan2(d2[1], d2[2])), mag);
    return ddiv(dadd(dmul(axz, axz), dmul(ayz, ayz)), 2.0);
}

// Displacement in the xz and yz planes (src/MutoMLSD.cpp:356-376): with the
// lines' slopes t = tan(angle) = d_x / d_z, the reference's
//   (x_out - x_in) cos(a_in) l_xy cos(a_out) / cos(a_out - a_in)
// is (x_out - x_in) l_xy / (1 + t_in t_out).  The difference, which cancels, is
// formed in the reference's order.
__device__ __forceinline__ void displacement(const muto_ray& r, double z_min, double* dxz, double* dyz) {
    const double sin_ = ddiv(dsub(z_min, r.pin[2]), r.din[2]);
    const double sout = ddiv(dsub(z_min, r.pout[2]), r.dout[2]);
    const double xp = dadd(r.pin[0], dmul(sin_, r.din[0]));
    const double yp = dadd(r.pin[1], dmul(sin_, r.din[1]));
    const double xt = dadd(r.pout[0], dmul(sout, r.dout[0]));
    const double yt = dadd(r.pout[1], dmul(sout, r.dout[1]));
    const double yi = 1.0 / r.din[2], yo = 1.0 / r.dout[2];
    const double tx = r.din[0] * yi, ty = r.din[1] * yi, ox = r.dout[0] * yo, oy = r.dout[1] * yo;
    const double lxy = sqrt(fma(tx, tx, fma(ty, ty, 1.0)));
    *dxz = dsub(xt, xp) * lxy / fma(tx, ox, 1.0);
    *dyz = dsub(yt, yp) * lxy / fma(ty, oy, 1.0);
}

}  // namespace muto
