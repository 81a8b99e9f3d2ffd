// FP64 functions of the precession and excitation kernels, written for their
// arguments; each stays within 2e-16 of the exact value (absolute for the cosine
// and sine, relative for the power).
#pragma once

#include <cuda_runtime.h>

namespace homs {

// cos and sin of 2 pi r for |r| <= 1/8: sin(2 pi r) / r is a polynomial of degree 6
// and (cos(2 pi r) - 1) / r^2 one of degree 6 in r^2, the interpolants at the
// Chebyshev nodes of the interval (relative error 4e-18 before the coefficients'
// rounding); 16 FP64 operations.
__device__ __forceinline__ void cis_eighth(double r, double &cs, double &sn) {
    const double z = r * r;
    double s = 3.7808689593022957, c = -1.6990343940660637;
    s = fma(s, z, -15.093804209987114);
    c = fma(c, z, 7.903206911569678);
    s = fma(s, z, 42.058685020160894);
    c = fma(c, z, -26.426253275854723);
    s = fma(s, z, -76.70585970427454);
    c = fma(c, z, 60.24464135270201);
    s = fma(s, z, 81.60524927594804);
    c = fma(c, z, -85.4568172066438);
    s = fma(s, z, -41.341702240399634);
    c = fma(c, z, 64.93939402266824);
    s = fma(s, z, 6.283185307179586);
    c = fma(c, z, -19.739208802178716);
    sn = s * r;
    cs = fma(c, z, 1.0);
}

// cos and sin of 2 pi theta: theta is reduced to its nearest quarter turn (an
// exact subtraction).  Beyond 2^48 turns (infinities and NaN included) it is first
// reduced to the nearest turn.
__device__ __forceinline__ void cis_turns(double th, double &cs, double &sn) {
    if ((__double2hiint(th) & 0x7FFFFFFF) >= 0x42F00000) th -= rint(th);
    constexpr double MAGIC = 6755399441055744.0;  // 1.5 * 2^52: adds round to an integer
    const double t = fma(th, 4.0, MAGIC);
    const int quad = __double2loint(t);
    const double r = fma(t - MAGIC, -0.25, th);
    double s, c;
    cis_eighth(r, c, s);
    // a quarter turn swaps the two and a half turn flips both signs
    const double a = (quad & 1) ? s : c, b = (quad & 1) ? c : s;
    cs = __hiloint2double(__double2hiint(a) ^ (((quad + 1) & 2) << 30), __double2loint(a));
    sn = __hiloint2double(__double2hiint(b) ^ ((quad & 2) << 30), __double2loint(b));
}

// cos and sin of 2 pi theta from a table of 256 points of the circle: theta is
// reduced to the nearest point (an exact subtraction); the rest, below 1/512 turn,
// takes three terms of either series; 14 FP64 operations, within 2e-16.
constexpr int CIS_POINTS = 256;
__device__ __forceinline__ void cis_table(const double2 *table, double th, double &cs, double &sn) {
    if ((__double2hiint(th) & 0x7FFFFFFF) >= 0x42700000) th -= rint(th);
    constexpr double MAGIC = 6755399441055744.0;  // 1.5 * 2^52: adds round to an integer
    const double t = fma(th, (double)CIS_POINTS, MAGIC);
    const double2 p = table[__double2loint(t) & (CIS_POINTS - 1)];
    const double r = fma(t - MAGIC, -1.0 / CIS_POINTS, th), z = r * r;
    double s = fma(81.60524927607506, z, -41.34170224039976), c = fma(-85.45681720669373, z, 64.9393940226683);
    s = fma(s, z, 6.283185307179586) * r;
    c = fma(c, z, -19.739208802178716) * z;
    cs = fma(p.x, c, fma(-p.y, s, p.x));
    sn = fma(p.y, c, fma(p.x, s, p.y));
}

// 2^y: nearest integer k, then 1 + f q(f) on |f| <= 1/2 with q the degree-10
// interpolant of (2^f - 1) / f at the Chebyshev nodes (relative error 1e-17 before
// the coefficients' rounding), and k added to the exponent; 15 FP64 operations.
// |y| >= 1008 (infinities and NaN included) goes to exp2.
__device__ __forceinline__ double pow2(double y) {
    if ((__double2hiint(y) & 0x7FFFFFFF) >= 0x408F8000) return exp2(y);
    constexpr double MAGIC = 6755399441055744.0;
    const double t = y + MAGIC;
    const int k = __double2loint(t);
    const double f = y - (t - MAGIC);
    double p = 4.4549605981865186e-10;
    p = fma(p, f, 7.072585949269223e-09);
    p = fma(p, f, 1.0178062445845774e-07);
    p = fma(p, f, 1.321544258792169e-06);
    p = fma(p, f, 1.525273382983612e-05);
    p = fma(p, f, 0.0001540353044173605);
    p = fma(p, f, 0.0013333558146416936);
    p = fma(p, f, 0.009618129107606888);
    p = fma(p, f, 0.0555041086648216);
    p = fma(p, f, 0.24022650695910097);
    p = fma(p, f, 0.6931471805599453);
    p = fma(p, f, 1.0);
    return __hiloint2double(__double2hiint(p) + (k << 20), __double2loint(p));
}

// 2^y for |y| <= 1/16: the exponential series to degree 8 (remainder 1.5e-18).
constexpr double POW2_SMALL = 0.0625;
__device__ __forceinline__ double pow2_small(double y) {
    double p = 1.3215486790144305e-06;
    p = fma(p, y, 1.5252733804059838e-05);
    p = fma(p, y, 0.00015403530393381606);
    p = fma(p, y, 0.0013333558146428441);
    p = fma(p, y, 0.009618129107628477);
    p = fma(p, y, 0.055504108664821576);
    p = fma(p, y, 0.2402265069591007);
    p = fma(p, y, 0.6931471805599453);
    p = fma(p, y, 1.0);
    return p;
}

// 2^y for |y| <= 1/128: to degree 5 (remainder 3.5e-17).
constexpr double POW2_TINY = 0.0078125;
__device__ __forceinline__ double pow2_tiny(double y) {
    double p = 0.0013333558146428441;
    p = fma(p, y, 0.009618129107628477);
    p = fma(p, y, 0.055504108664821576);
    p = fma(p, y, 0.2402265069591007);
    p = fma(p, y, 0.6931471805599453);
    p = fma(p, y, 1.0);
    return p;
}

}  // namespace homs
