// dd_real.cuh -- the real-space dipole field of one induced-dipole iteration of the FP64 engine
// (pot_ttm.f90:311-365), from the tensors cached by the charge phase: thread t0 of nt over the pairs
// (and molecules) of bead b, FP64 atomics per site.
#pragma once
#include "engine.h"

namespace pimd {

// site kinds (1-based like the reference): 1 O, 2 H1, 3 H2, 4 M
template <int MODEL>
struct TT {
    static constexpr int FDI = MODEL == 2 ? 1 : 4;
    static constexpr int LDI = MODEL == 2 ? 3 : 4;
    PIMD_HD static constexpr bool dip(int k) { return k >= FDI && k <= LDI; }
};

PIMD_D double3 ld3(const double *p) { return make_double3(p[0], p[1], p[2]); }

template <int MODEL>
PIMD_D void dd_real_pairs(const KP &kp, int b, int t0, int nt) {
    using T = TT<MODEL>;
    const int N = kp.N;
    if (bead_converged(kp, b)) return;
    const int np = kp.npair[b];
    const double *dip = kp.dip + (size_t)b * kp.S * 3;
    double *Ef = kp.Efdr + (size_t)b * kp.S * 3;
    for (int p = t0; p < np; p += nt) {
        const int2 ij = kp.pairs[(size_t)b * kp.cap + p];
        const double *Tp = kp.Tdd + ((size_t)b * kp.cap + p) * kp.ndd * 6;
        double ei[5][3], ej[5][3];
#pragma unroll
        for (int k = 0; k < 5; k++) ei[k][0] = ei[k][1] = ei[k][2] = ej[k][0] = ej[k][1] = ej[k][2] = 0.0;
        int t = 0;
#pragma unroll
        for (int isp = T::FDI; isp <= T::LDI; isp++) {
            const double3 mi = ld3(dip + 3 * ((isp - 1) * N + ij.x));
#pragma unroll
            for (int jsp = T::FDI; jsp <= T::LDI; jsp++, t++) {
                const double3 mj = ld3(dip + 3 * ((jsp - 1) * N + ij.y));
                const double *Tt = Tp + 6 * t;
                const double xx = Tt[0], yy = Tt[1], zz = Tt[2], xy = Tt[3], xz = Tt[4], yz = Tt[5];
                ei[isp][0] += xx * mj.x + xy * mj.y + xz * mj.z;
                ei[isp][1] += xy * mj.x + yy * mj.y + yz * mj.z;
                ei[isp][2] += xz * mj.x + yz * mj.y + zz * mj.z;
                ej[jsp][0] += xx * mi.x + xy * mi.y + xz * mi.z;
                ej[jsp][1] += xy * mi.x + yy * mi.y + yz * mi.z;
                ej[jsp][2] += xz * mi.x + yz * mi.y + zz * mi.z;
            }
        }
#pragma unroll
        for (int k = T::FDI; k <= T::LDI; k++)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                atomicAdd(Ef + 3 * ((k - 1) * N + ij.x) + c, ei[k][c]);
                atomicAdd(Ef + 3 * ((k - 1) * N + ij.y) + c, ej[k][c]);
            }
    }
    if (MODEL == 2) {  // intramolecular O-H1, O-H2, H1-H2 (pot_ttm.f90:344-365)
        for (int w = t0; w < N; w += nt) {
            const double *Tw = kp.Tself + ((size_t)b * N + w) * 18;
            double e[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
            double3 m[3];
#pragma unroll
            for (int k = 0; k < 3; k++) m[k] = ld3(dip + 3 * (k * N + w));
            int t = 0;
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = i + 1; j < 3; j++, t++) {
                    const double *Tt = Tw + 6 * t;
                    const double xx = Tt[0], yy = Tt[1], zz = Tt[2], xy = Tt[3], xz = Tt[4], yz = Tt[5];
                    e[i][0] += xx * m[j].x + xy * m[j].y + xz * m[j].z;
                    e[i][1] += xy * m[j].x + yy * m[j].y + yz * m[j].z;
                    e[i][2] += xz * m[j].x + yz * m[j].y + zz * m[j].z;
                    e[j][0] += xx * m[i].x + xy * m[i].y + xz * m[i].z;
                    e[j][1] += xy * m[i].x + yy * m[i].y + yz * m[i].z;
                    e[j][2] += xz * m[i].x + yz * m[i].y + zz * m[i].z;
                }
#pragma unroll
            for (int k = 0; k < 3; k++)
#pragma unroll
                for (int c = 0; c < 3; c++) atomicAdd(Ef + 3 * (k * N + w) + c, e[k][c]);
        }
    }
}

}  // namespace pimd
