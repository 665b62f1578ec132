// pairs.cuh -- separations, screening radii and the virial term shared by the
// pair passes (pairs.cu) and the fused runs of steps (run.cu).
#pragma once

#include "engine.h"

namespace moldy {

// Squared FP32 distance of an FP64 fractional difference (any box): the
// difference rounded to FP32 (off by at most 2^-24 |dx|), the minimum image by
// rintf in the periodic directions.
__device__ __forceinline__ float sep2_f32(const float *bf, int ivol, double dxd, double dyd, double dzd) {
    float dx = (float)dxd, dy = (float)dyd, dz = (float)dzd;
    if (ivol == 0 || ivol == 1 || ivol == 4) {
        dx -= rintf(dx); dy -= rintf(dy); dz -= rintf(dz);
    } else if (ivol == 2) {
        dx -= rintf(dx); dy -= rintf(dy);
    } else if (ivol == 5) {
        dz -= rintf(dz);
    }
    const float rx = fmaf(bf[6], dz, fmaf(bf[3], dy, bf[0] * dx));
    const float ry = fmaf(bf[7], dz, fmaf(bf[4], dy, bf[1] * dx));
    const float rz = fmaf(bf[8], dz, fmaf(bf[5], dy, bf[2] * dx));
    return fmaf(rz, rz, fmaf(ry, ry, rx * rx));
}

// Separation of two atoms from their fixed-point coordinates (fully periodic
// box): the 32-bit differences are the minimum image; bs is B0 per fixed-point
// unit.  Returns r^2 and the Cartesian separation, all FP32.
__device__ __forceinline__ float fix_sep(const float *bs, const int4 &qa, const int4 &qj, float &rx, float &ry,
                                         float &rz, float &dx, float &dy, float &dz) {
    dx = fix_to_float((int32_t)((uint32_t)qa.x - (uint32_t)qj.x));
    dy = fix_to_float((int32_t)((uint32_t)qa.y - (uint32_t)qj.y));
    dz = fix_to_float((int32_t)((uint32_t)qa.z - (uint32_t)qj.z));
    rx = fmaf(bs[6], dz, fmaf(bs[3], dy, bs[0] * dx));
    ry = fmaf(bs[7], dz, fmaf(bs[4], dy, bs[1] * dx));
    rz = fmaf(bs[8], dz, fmaf(bs[5], dy, bs[2] * dx));
    return fmaf(rz, rz, fmaf(ry, ry, rx * rx));
}

__device__ __forceinline__ float fix_sep(const float *bs, const int4 &qa, const int4 &qj, float &rx, float &ry,
                                         float &rz) {
    float dx, dy, dz;
    return fix_sep(bs, qa, qj, rx, ry, rz, dx, dy, dz);
}

// --------------------------------------------------------------- screen --
// Squared screening radius for the FP32 pre-selection.  The FP32 copy of a
// fractional coordinate is off by at most 2^-24 |x|; for |x| < 5 (positions
// are never wrapped) the FP32 distance is then within 2e-6 |B0|_F + 1e-4 A of
// the FP64 one.  rintf and NINT pick different images only at |dx| = 1/2,
// i.e. at half a box width; when half the narrowest width is not beyond the
// screening radius every pair goes to the FP64 test.
static __device__ float screen_radius2(const double *b, double rcull2) {
    double nf = 0.0;
    for (int k = 0; k < 9; ++k) nf += b[k] * b[k];
    double rs = sqrt(rcull2) + 2.0e-6 * sqrt(nf) + 1.0e-4;
    double vol = fabs(b[0] * (b[4] * b[8] - b[7] * b[5]) - b[3] * (b[1] * b[8] - b[7] * b[2]) +
                      b[6] * (b[1] * b[5] - b[4] * b[2]));
    double wmin = 1e300;
    for (int k = 0; k < 3; ++k) {   // width across the face spanned by the other two box vectors
        const double *u = b + 3 * ((k + 1) % 3), *w = b + 3 * ((k + 2) % 3);
        double cx = u[1] * w[2] - u[2] * w[1], cy = u[2] * w[0] - u[0] * w[2], cz = u[0] * w[1] - u[1] * w[0];
        double a = sqrt(cx * cx + cy * cy + cz * cz);
        if (a > 0.0) wmin = fmin(wmin, vol / a);
    }
    if (!(0.5 * wmin > rs * (1.0 + 1e-6))) return 3.0e38f;
    return (float)(rs * rs);
}


constexpr int32_t kOwnBit = (int32_t)0x80000000u;
constexpr int32_t kIdMask = 0x7fffffff;

// The exact FP64 test r^2 <= rcull^2 for a pair whose FP32 distance lies in
// the error band around the cut (rare: kept out of line, so its registers do
// not count against the screening loop)
static __device__ __noinline__ bool inside_cut_fp64(const double4 *__restrict__ pos, int a, int j, const double *b,
                                             int ivol, double rcull2) {
    const double4 pa = pos[a], qd = pos[j];
    double ex = pa.x - qd.x, ey = pa.y - qd.y, ez = pa.z - qd.z;
    min_image(ivol, ex, ey, ez);
    double sx = b[0] * ex + b[3] * ey + b[6] * ez;
    double sy = b[1] * ex + b[4] * ey + b[7] * ez;
    double sz = b[2] * ex + b[5] * ey + b[8] * ez;
    return (sx * sx + sy * sy + sz * sz) <= rcull2;
}

// v[1..6] += s * sym(a (x) b) in the order xx, yy, zz, xy, xz, yz
__device__ __forceinline__ void add_sym(double *v, double ax, double ay, double az, double bx, double by,
                                        double bz, double s) {
    v[1] += s * (ax * bx);
    v[2] += s * (ay * by);
    v[3] += s * (az * bz);
    v[4] += (0.5 * s) * (ax * by + ay * bx);
    v[5] += (0.5 * s) * (ax * bz + az * bx);
    v[6] += (0.5 * s) * (ay * bz + az * by);
}

// FP32 keep radius^2 of a list of radius r: r plus twice the FP32 distance
// error bound, or every pair when the box is too small for the FP32 screen
static __device__ float keep_radius2(const double *sb, double r) {
    const float keep = (float)(r + 2.0 * (2.0e-6 * frob(sb) + 1.0e-4));
    return screen_radius2(sb, r * r) > 1e37f ? 3.0e38f : keep * keep;
}

// ------------------------------------------------------- FP64 pair terms --
// r = sqrt(r2) and 1/r of a positive r2 from one reciprocal square root: the
// product r2 y is corrected by half its residual times y and then 1/r by its
// own residual (one Newton step each), which leaves both within an ulp, in 6
// operations where a square root and a division took two full routines.  Two
// atoms at one point: r = 0, the table's first node, and 1/r is not a number
// (the pair has no direction).  The high word tells, without the FP64 units.
__device__ __forceinline__ double root_and_inverse(double r2, double &rr) {
    const double y = rsqrt(r2);
    double r = r2 * y;
    r = fma(fma(-r, r, r2), 0.5 * y, r);
    rr = fma(fma(-r, y, 1.0), y, y);
    return __double2hiint(r2) == 0 ? 0.0 : r;
}

// r alone; of 0 it gives that of the smallest normal number, 1.5e-154 (one
// integer maximum)
__device__ __forceinline__ double root(double r2) {
    r2 = __hiloint2double(max(__double2hiint(r2), 0x00100000), __double2loint(r2));
    const double y = rsqrt(r2);
    const double r = r2 * y;
    return fma(fma(-r, r, r2), 0.5 * y, r);
}

// Interval of r in the stored nodes and the offset in it; beyond the last
// stored node, that node (its step is zero).  floor by a round-down addition.
__device__ __forceinline__ int interval_d(const Tables &t, double r, double &dr) {
    const double x = fma(r, t.vp_recipstep, t.vp_xoff);
    const double b = __dadd_rd(fmin(fmax(x, 0.0), (double)(t.nr - 1)), 4503599627370496.0);   // + 2^52
    dr = x - (b - 4503599627370496.0);
    return __double2loint(b);
}

// The minimum image of min_image: u - NINT(u) in the periodic directions, m =
// NINT(u).  Nearly every difference lies inside (-1/2, 1/2), where NINT is
// zero: true when one does not (the caller's rare case).
__device__ __forceinline__ bool outside_half(double ux, double uy, double uz) {
    return !(fabs(ux) < 0.5 && fabs(uy) < 0.5 && fabs(uz) < 0.5);
}

}  // namespace moldy
