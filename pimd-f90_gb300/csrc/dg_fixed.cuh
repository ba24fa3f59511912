// dg_fixed.cuh -- fixed-point numbers of the FP64 engine's reciprocal sums (ewald_dg.cu, dipole_matrix.cu)
#pragma once
#include "engine.h"

namespace pimd {

constexpr int DG_BAD = 0x7fffffff;  // scale of an operand with a value that is not finite

// x 2^sh rounded to an integer, |x 2^sh| < 2^63, from the bits of x (an FP64 conversion costs the
// FP64 pipe 64 cycles a warp). A value that is not finite gives 0: the caller's scale says so.
PIMD_D long long dg_fix(double x, int sh) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    const int ex = (int)(u >> 52) & 0x7ff;
    const unsigned long long m = (u & 0xfffffffffffffULL) | 0x10000000000000ULL;
    const int s = ex - 1075 + sh;  // x = m 2^(ex - 1075)
    if (ex == 0 || ex == 0x7ff || s < -53) return 0;
    const unsigned long long v = s >= 0 ? m << s : (m + (1ULL << (-s - 1))) >> -s;
    return (long long)u < 0 ? -(long long)v : (long long)v;
}
// exponent e with |x| < 2^e for every x whose high word (sign cleared) is at most hi
PIMD_D int dg_exp(int hi) {
    const int ex = hi >> 20;
    return ex >= 0x7ff ? DG_BAD : ex - 1022;
}
PIMD_D int dg_hi(double x) { return __double2hiint(x) & 0x7fffffff; }
// t 2^e rounded to nearest
PIMD_D double dg_double(long long t, int e) {
    if (t == 0) return 0.0;
    const bool neg = t < 0;
    unsigned long long u = neg ? 0ULL - (unsigned long long)t : (unsigned long long)t;
    const int lz = __clzll((long long)u);
    u <<= lz;
    const int E = 1023 + 63 - lz + e;
    if (E <= 0) return 0.0;
    const unsigned long long r = ((unsigned long long)(E - 1) << 52) + (u >> 11) + ((u >> 10) & 1ULL);
    return __longlong_as_double((long long)(neg ? r | 0x8000000000000000ULL : r));
}
// (t + lo 2^-w) 2^e rounded to nearest, |t| <= 2^62, |lo| < 2^(w + 1): to 62 bits first where those do not hold it
PIMD_D double dg_double(long long t, int lo, int w, int e) {
    const int m = min(w, max(0, __clzll(t < 0 ? -t : t) - 2)), r = w - m;
    return dg_double(t * (1LL << m) + ((lo + ((1 << r) >> 1)) >> r), e - m);
}

// ---- products of fixed-point numbers -----------------------------------------------------------
// A number in [-1, 1] as 2^62 x = hi 2^32 + lo with both halves signed, so that a product needs no
// unsigned corrections. dg_mul: a b / 2^64 without the low halves' product (below one unit).
PIMD_D int2 dg_split(long long v) {
    const int lo = (int)v;
    return make_int2((int)((v - lo) >> 32), lo);
}
PIMD_D long long dg_join(int2 a) { return ((long long)a.x << 32) + a.y; }
PIMD_D long long dg_mul(int2 a, int2 b) {
    return (long long)a.x * b.x + (((long long)a.x * b.y + (long long)a.y * b.x) >> 32);
}
// a1 b1 + a2 b2, a1 b1 - a2 b2 (/ 2^64)
PIMD_D long long dg_mul2(int2 a1, int2 b1, int2 a2, int2 b2) {
    const long long m = (long long)a1.x * b1.y + (long long)a1.y * b1.x + (long long)a2.x * b2.y + (long long)a2.y * b2.x;
    return (long long)a1.x * b1.x + (long long)a2.x * b2.x + (m >> 32);
}
PIMD_D long long dg_mul2m(int2 a1, int2 b1, int2 a2, int2 b2) {
    const long long m = (long long)a1.x * b1.y + (long long)a1.y * b1.x - (long long)a2.x * b2.y - (long long)a2.y * b2.x;
    return (long long)a1.x * b1.x - (long long)a2.x * b2.x + (m >> 32);
}
// the parts of an entry of the phase tables: (cos hi, lo, sin hi, lo)
PIMD_D int2 dg_re(int4 v) { return make_int2(v.x, v.y); }
PIMD_D int2 dg_im(int4 v) { return make_int2(v.z, v.w); }

}  // namespace pimd
