// pair_math.cuh -- FP64 pair arithmetic of the force call with few FP64-pipe instructions. This
// part issues an FP64 instruction (a conversion and a compare too) every 64 cycles on a
// sub-partition; integer ones every other cycle.
#pragma once
#include "engine.h"

namespace pimd {

// min_image_rn(r, box) by the cell r lies in, where that is beyond doubt: anint(r / box) is 0 below 0.49
// box edges and +-1 between 0.51 and 1.49, so the same value with at most one FP64 operation
PIMD_D double min_image_near(double r, const KP &kp, int c) {
    const int h = hi_abs(r);
    if (h < kp.box49[c]) return r;
    if (h >= kp.box51[c] && h < kp.box149[c]) return __dsub_rn(r, copysign(kp.box[c], r));
    return min_image_rn(r, kp.box[c], kp.boxi[c]);
}

// the undamped screened interaction at r^2 = d2 (smear.f90:10-18): 1/r, r, 1/r^2, exp(-a^2 r^2),
// ts0 = erfc(a r) / r (Abramowitz-Stegun 7.1.26, math.f90:287-314) and ts1
struct PairR {
    double dri, dd, drsqi, g, t0, t1;
};
PIMD_D void pair_r(double d2, const EwC &e, PairR &p) {
    p.dri = rsqrt(d2);
    p.dd = d2 * p.dri;
    p.drsqi = p.dri * p.dri;
    p.g = exp(-(e.a2 * d2));
    const double T = rcp_newton(1.0 + 0.3275911 * (e.aewald * p.dd));
    const double TP = T * (0.254829592 + T * (-0.284496736 + T * (1.421413741 + T * (-1.453152027 + T * 1.061405429))));
    p.t0 = TP * p.g * p.dri;
    p.t1 = (p.t0 + e.cts1 * p.g) * p.drsqi;
}

// Q(2/3, x) as the reference's gammq2_3 leaves it (math.f90:188-285), with the number of terms from
// the bounds in tb and pre = x^(2/3) exp(-x) / Gamma(2/3). The continued fraction's convergent by the forward recurrence
// of its numerators and denominators (no division until the end).
PIMD_D double thole_q23(double x, double pre, const GqBounds &tb, unsigned *err) {
    const double a = 2.0 / 3.0;
    if (hi_abs(x) >= 0x7ff00000 && x != x) {
        *err |= 4u;
        return x;
    }
    if (x < a + 1.0) {
        if (x <= 0.0) return 1.0;
        double sum = 1.5, del = 1.5;
        for (int n = 1; n <= GQ_TERMS; n++) {
            del *= x * tb.inv[n];
            sum += del;
            if (__double_as_longlong(x) <= __double_as_longlong(tb.ser[n])) break;
        }
        return 1.0 - sum * pre;
    }
    double b = x + 1.0 - a, A0 = 0.0, A1 = 1.0, B0 = 1.0, B1 = b;
    for (int i = 1; i <= GQ_TERMS; i++) {
        const double an = -(double)i * ((double)i - a);
        b += 2.0;
        const double A2 = b * A1 + an * A0, B2 = b * B1 + an * B0;
        A0 = A1;
        A1 = A2;
        B0 = B1;
        B1 = B2;
        if (__double_as_longlong(x) >= __double_as_longlong(tb.fra[i])) break;
    }
    return pre * (A1 / B1);
}

// A block's sums of the virial (xx yy zz xy xz yz), the centroid virial and the vdW energy into a
// bead's accumulators; warps that hold only zeros skip the FP64 sums.
template <int NT>
PIMD_D void pair_block_sums(const double (&vt)[6], double vc, double uv, double *acc) {
    __shared__ double red[NT / 32][8];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    double v[8] = {vt[0], vt[1], vt[2], vt[3], vt[4], vt[5], vc, uv};
    long long any = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) any |= __double_as_longlong(v[i]) << 1;
    if (__any_sync(0xffffffffu, any != 0)) {
        int at;
        const double s = warp_sums<8>(v, at);
        if ((lane & 3) == 0) red[wp][at] = s;
    } else if (lane < 8) {
        red[wp][lane] = 0.0;
    }
    __syncthreads();
    if (threadIdx.x < 8) {
        double s = 0.0;
        for (int w = 0; w < NT / 32; w++) s += red[w][threadIdx.x];
        if (__double_as_longlong(s) << 1) {
            const int to[8] = {ACC_VIRT + 0, ACC_VIRT + 4, ACC_VIRT + 8, ACC_VIRT + 1, ACC_VIRT + 2, ACC_VIRT + 5, ACC_VIRIALC, ACC_UVDW};
            const int mirror[8] = {-1, -1, -1, ACC_VIRT + 3, ACC_VIRT + 6, ACC_VIRT + 7, -1, -1};
            atomicAdd(acc + to[threadIdx.x], s);
            if (mirror[threadIdx.x] >= 0) atomicAdd(acc + mirror[threadIdx.x], s);
        }
    }
    __syncthreads();
}

}  // namespace pimd
