// pot.cu -- real-space, monomer and bookkeeping kernels of the TTM2.1-F / TTM3-F force call
// for all beads at once (FP64). Restates pot_ttm/pot_ttm.f90:3-630 and find_neigh.f90.
//
// Work decomposition: the bead is blockIdx.y (or .z) everywhere. Monomer work is one thread (small
// FP64 systems: four lanes) per molecule; the pairs' sums are in pairs.cu (FP64) and mixed.cu.
// Energies and virials are reduced per block and added once per block to the per-bead accumulators.
#include <cstdio>

#include "dd_real.cuh"
#include "engine.h"
#include "nasa.cuh"
#include "pair_math.cuh"

namespace pimd {

void pot_init_constants(Engine &E) {
    pair_math_init(E);
    if (E.kp.model < 4) nasa_upload_constants();
}

// ---------------------------------------------------------------------------------------
// pot_ttm.f90:56-151 and 232-261: site layout, M sites, NASA PES + DMS charges, monomer
// virials, self energy and intramolecular Ewald exclusions. Two threads per (molecule, bead),
// in two warps of a 64-thread block (32 molecules): the first warp evaluates the PES
// (nasa_pot), the monomer virial and the gradient rows; the second the DMS charges (nasa_dms),
// their gradients, the site rows, the self energy and the intramolecular exclusions. The two
// halves share no data, so the FP64-latency-bound chain of a molecule is split in two; about 7
// warps per SM at 512 x 32, spread over every SM.
constexpr int SITES_NT = 64;

// The mixed engine: the NASA polynomial sums in FP32 (k_sites64 is the FP64 engine's)
template <int MODEL>
__global__ void __launch_bounds__(SITES_NT) k_sites(KP kp) {
    constexpr bool FSUM = true;
    const int w = blockIdx.x * (SITES_NT / 2) + (threadIdx.x & 31);
    const bool pes = threadIdx.x < 32;  // warp-uniform roles
    const int b = blockIdx.y;
    const int N = kp.N, S = kp.S;
    double av[14];
#pragma unroll
    for (int i = 0; i < 14; i++) av[i] = 0.0;
    if (w < N) {
        const double *RR = kp.RRt + (size_t)b * kp.natoms * 3 + 9 * w;
        const int rep = rep_of(kp, b);
        const double *RC = kp.RRc + (size_t)rep * kp.natoms * 3 + 9 * w;
        const bool first_bead = (b == 0) || (kp.brep && kp.brep[b - 1] != rep);
        double R[4][3], Rc[4][3];
#pragma unroll
        for (int k = 0; k < 3; k++)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                R[k][c] = RR[3 * k + c];
                Rc[k][c] = RC[3 * k + c];
            }
        const double hg = 0.5 * kp.gammaM;
        // the O-H minimum images of the bead and the centroid (the M sites, and in the mixed
        // engine the FP32 site offsets of the exclusion pairs)
        double oh[2][3], ohc[2][3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            oh[0][c] = min_image_rn(__dsub_rn(R[1][c], R[0][c]), kp.box[c], kp.boxi[c]);
            oh[1][c] = min_image_rn(__dsub_rn(R[2][c], R[0][c]), kp.box[c], kp.boxi[c]);
            R[3][c] = __dadd_rn(__dmul_rn(hg, __dadd_rn(oh[0][c], oh[1][c])), R[0][c]);
            ohc[0][c] = min_image_rn(__dsub_rn(Rc[1][c], Rc[0][c]), kp.box[c], kp.boxi[c]);
            ohc[1][c] = min_image_rn(__dsub_rn(Rc[2][c], Rc[0][c]), kp.box[c], kp.boxi[c]);
            Rc[3][c] = __dadd_rn(__dmul_rn(hg, __dadd_rn(ohc[0][c], ohc[1][c])), Rc[0][c]);
        }
        if (pes) {
            double dr1[3][3], e1 = 0.0;
            if (!kp.contraction) {
                nasa_pot(R, kp.box, kp.boxi, dr1, &e1, kp.c5z, kp.nasa_f5z, FSUM);
            } else {
#pragma unroll
                for (int k = 0; k < 3; k++)
#pragma unroll
                    for (int c = 0; c < 3; c++) dr1[k][c] = 0.0;
            }
            av[ACC_UMON] = e1;
            if (!kp.contraction) {
                double roh1[3], roh2[3], rc1[3], rc2[3];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    roh1[c] = min_image_rn(__dsub_rn(R[1][c], R[0][c]), kp.box[c], kp.boxi[c]);
                    roh2[c] = min_image_rn(__dsub_rn(R[2][c], R[0][c]), kp.box[c], kp.boxi[c]);
                    rc1[c] = min_image_rn(__dsub_rn(Rc[1][c], Rc[0][c]), kp.box[c], kp.boxi[c]);
                    rc2[c] = min_image_rn(__dsub_rn(Rc[2][c], Rc[0][c]), kp.box[c], kp.boxi[c]);
                }
#pragma unroll
                for (int col = 0; col < 3; col++)
#pragma unroll
                    for (int c = 0; c < 3; c++) av[ACC_VIRT + c + 3 * col] += roh1[c] * dr1[1][col] + roh2[c] * dr1[2][col];
                av[ACC_VIRIALC] += (rc1[0] * dr1[1][0] + rc1[1] * dr1[1][1] + rc1[2] * dr1[1][2]) +
                                   (rc2[0] * dr1[2][0] + rc2[1] * dr1[2][1] + rc2[2] * dr1[2][2]);
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const size_t s = (size_t)b * S + k * N + w;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    kp.dR[3 * s + c] = (k < 3) ? dr1[k][c] : 0.0;
                    kp.dip[3 * s + c] = 0.0;
                    kp.Efdr[3 * s + c] = 0.0;
                }
            }
        } else {
            double q3[3], dq3[3][3][3];
            nasa_dms(R, kp.box, kp.boxi, kp.dms1, kp.dms2, kp.dms3, q3, dq3, FSUM);
#pragma unroll
            for (int k = 0; k < 3; k++) {
                q3[k] *= CHARGECON;
                kp.chg[(size_t)b * kp.natoms + 3 * w + k] = q3[k];
            }
            const double tmp = 0.5 * kp.gammaM / (1.0 - kp.gammaM);
            double q[4];
            q[0] = 0.0;
            q[1] = q3[1] + tmp * (q3[1] + q3[2]);
            q[2] = q3[2] + tmp * (q3[1] + q3[2]);
            q[3] = q3[0] / (1.0 - kp.gammaM);
            double *g = kp.grdq + ((size_t)b * N + w) * 27;
#pragma unroll
            for (int a = 0; a < 3; a++)
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const double s01 = dq3[a][0][c] * CHARGECON + dq3[a][1][c] * CHARGECON;
                    g[9 * a + 0 + c] = dq3[a][0][c] * CHARGECON + tmp * s01;
                    g[9 * a + 3 + c] = dq3[a][1][c] * CHARGECON + tmp * s01;
                    g[9 * a + 6 + c] = dq3[a][2][c] * CHARGECON - 2.0 * tmp * s01;
                }
            // self energy and intramolecular exclusions (pot_ttm.f90:232-261)
            double Ef[4][3], ph[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                ph[k] = (k == 0) ? 0.0 : -kp.ew.aewald * TSP * q[k];
                Ef[k][0] = Ef[k][1] = Ef[k][2] = 0.0;
            }
            if (FSUM && MODEL == 3) {
                // the mixed engine, TTM3-F: the six exclusion pairs in FP32 from the sites' offsets
                // to their O site (a molecule spans far less than half a box, so a pair's minimum
                // image is the difference of the two offsets); sums converted once
                float rel[4][3], relc[4][3];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    rel[0][c] = relc[0][c] = 0.f;
                    rel[1][c] = (float)oh[0][c];
                    rel[2][c] = (float)oh[1][c];
                    rel[3][c] = (float)__dsub_rn(R[3][c], R[0][c]);
                    relc[1][c] = (float)ohc[0][c];
                    relc[2][c] = (float)ohc[1][c];
                    relc[3][c] = (float)__dsub_rn(Rc[3][c], Rc[0][c]);
                }
                const float qf[4] = {(float)q[0], (float)q[1], (float)q[2], (float)q[3]};
                float phf[4] = {0.f, 0.f, 0.f, 0.f}, Eff[4][3], vcf = 0.f, vtf[9];
#pragma unroll
                for (int k = 0; k < 4; k++) Eff[k][0] = Eff[k][1] = Eff[k][2] = 0.f;
#pragma unroll
                for (int k = 0; k < 9; k++) vtf[k] = 0.f;
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = i + 1; j < 4; j++) {
                        const float Rs[3] = {rel[i][0] - rel[j][0], rel[i][1] - rel[j][1], rel[i][2] - rel[j][2]};
                        const float Rcs[3] = {relc[i][0] - relc[j][0], relc[i][1] - relc[j][1], relc[i][2] - relc[j][2]};
                        float ts0, ts1;
                        self1f(Rs[0] * Rs[0] + Rs[1] * Rs[1] + Rs[2] * Rs[2], kp.ewf, &ts0, &ts1);
                        phf[i] += ts0 * qf[j];
                        phf[j] += ts0 * qf[i];
                        float d[3];
#pragma unroll
                        for (int c = 0; c < 3; c++) {
                            Eff[i][c] += ts1 * qf[j] * Rs[c];
                            Eff[j][c] -= ts1 * qf[i] * Rs[c];
                            d[c] = -ts1 * qf[i] * qf[j] * Rs[c];
                        }
                        vcf += Rcs[0] * d[0] + Rcs[1] * d[1] + Rcs[2] * d[2];
#pragma unroll
                        for (int col = 0; col < 3; col++)
#pragma unroll
                            for (int c = 0; c < 3; c++) vtf[c + 3 * col] += d[col] * Rs[c];
                    }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    ph[k] += (double)phf[k];
#pragma unroll
                    for (int c = 0; c < 3; c++) Ef[k][c] = (double)Eff[k][c];
                }
                av[ACC_VIRIALC] += (double)vcf;
#pragma unroll
                for (int k = 0; k < 9; k++) av[ACC_VIRT + k] += (double)vtf[k];
            } else
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = i + 1; j < 4; j++) {
                    double Rs[3], Rcs[3];
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        Rs[c] = min_image_rn(__dsub_rn(R[i][c], R[j][c]), kp.box[c], kp.boxi[c]);
                        Rcs[c] = min_image_rn(__dsub_rn(Rc[i][c], Rc[j][c]), kp.box[c], kp.boxi[c]);
                    }
                    // FP64 (TTM2.1-F's polarisable H sites take the exclusion field into the
                    // dipoles, so its mixed engine keeps these in FP64 as well)
                    double ts0, ts1;
                    self1(dot3_rn(Rs[0], Rs[1], Rs[2]), kp.ew, &ts0, &ts1);
                    ph[i] += ts0 * q[j];
                    ph[j] += ts0 * q[i];
                    double d[3];
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        Ef[i][c] += ts1 * q[j] * Rs[c];
                        Ef[j][c] -= ts1 * q[i] * Rs[c];
                        d[c] = -ts1 * q[i] * q[j] * Rs[c];
                    }
                    av[ACC_VIRIALC] += Rcs[0] * d[0] + Rcs[1] * d[1] + Rcs[2] * d[2];
#pragma unroll
                    for (int col = 0; col < 3; col++)
#pragma unroll
                        for (int c = 0; c < 3; c++) av[ACC_VIRT + c + 3 * col] += d[col] * Rs[c];
                }
            // TTM2.1-F intramolecular dipole tensors (pot_ttm.f90:344-365), cached per molecule
            if (MODEL == 2) {
                int t = 0;
#pragma unroll
                for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int j = i + 1; j < 3; j++, t++) {
                        double Rs[3];
#pragma unroll
                        for (int c = 0; c < 3; c++) Rs[c] = min_image_rn(__dsub_rn(R[i][c], R[j][c]), kp.box[c], kp.boxi[c]);
                        double t1, t2;
                        smear2<double>(dot3_rn(Rs[0], Rs[1], Rs[2]), kp.pt.apol_dd[i + 1][j + 1], kp.ew, &t1, &t2);
                        double *T = kp.Tself + (((size_t)b * N + w) * 3 + t) * 6;
                        T[0] = 3.0 * t2 * Rs[0] * Rs[0] - t1;
                        T[1] = 3.0 * t2 * Rs[1] * Rs[1] - t1;
                        T[2] = 3.0 * t2 * Rs[2] * Rs[2] - t1;
                        T[3] = 3.0 * t2 * Rs[0] * Rs[1];
                        T[4] = 3.0 * t2 * Rs[0] * Rs[2];
                        T[5] = 3.0 * t2 * Rs[1] * Rs[2];
                    }
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const size_t s = (size_t)b * S + k * N + w;
                kp.pos[s] = make_double4_32a(R[k][0], R[k][1], R[k][2], q[k]);
                if (first_bead) kp.posc[(size_t)rep * S + k * N + w] = make_double4_32a(Rc[k][0], Rc[k][1], Rc[k][2], 0.0);
                kp.F[s] = make_double4_32a(Ef[k][0], Ef[k][1], Ef[k][2], ph[k]);
            }
        }
    }
    block_reduce_add<14, SITES_NT>(av, kp.acc + (size_t)b * NACC);
}

// The same in FP64 (the FP64 engine). A molecule is some 2500 FP64 instructions of 64 cycles a warp,
// so in small systems a molecule takes L = 4 lanes: they share the polynomial sums, and each does the
// self energy, exclusions and rows of one site (each exclusion pair twice, its virial at half
// weight); with enough molecules to fill the chip one lane takes them all. Few FP64 instructions:
// reciprocals for divisions, minimum images only where needed, the screened interaction of the
// pair kernels. 128 molecules, one bead: 97 -> 36 us; 512 x 32: 149 -> 95 us.
template <int MODEL, int L>
__global__ void __launch_bounds__(SITES_NT) k_sites64(KP kp) {
    const int lane = threadIdx.x & 31, l = lane % L, b = blockIdx.y, N = kp.N, S = kp.S;
    const int wm = blockIdx.x * (32 / L) + lane / L, w = min(wm, N - 1);
    const bool in = wm < N, pes = threadIdx.x < 32;  // warp-uniform roles
    double av[14];
#pragma unroll
    for (int i = 0; i < 14; i++) av[i] = 0.0;
    const double *RR = kp.RRt + (size_t)b * kp.natoms * 3 + 9 * w;
    const int rep = rep_of(kp, b);
    const double *RC = kp.RRc + (size_t)rep * kp.natoms * 3 + 9 * w;
    const bool first_bead = (b == 0) || (kp.brep && kp.brep[b - 1] != rep);
    double R[4][3], Rc[4][3], oh[2][3], ohc[2][3];
    const double hg = 0.5 * kp.gammaM;
#pragma unroll
    for (int c = 0; c < 3; c++) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            R[k][c] = RR[3 * k + c];
            Rc[k][c] = RC[3 * k + c];
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            oh[h][c] = min_image_fast(__dsub_rn(R[1 + h][c], R[0][c]), kp.box[c], kp.boxi[c]);
            ohc[h][c] = min_image_fast(__dsub_rn(Rc[1 + h][c], Rc[0][c]), kp.box[c], kp.boxi[c]);
        }
        R[3][c] = __dadd_rn(__dmul_rn(hg, __dadd_rn(oh[0][c], oh[1][c])), R[0][c]);
        Rc[3][c] = __dadd_rn(__dmul_rn(hg, __dadd_rn(ohc[0][c], ohc[1][c])), Rc[0][c]);
    }
    if (pes) {
        double dr1[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, e1 = 0.0;
        if (!kp.contraction) {
            nasa_pot<L>(R, kp.box, kp.boxi, dr1, &e1, kp.c5z, kp.nasa_f5z, false, l);
            if (in && l == 0) {
                av[ACC_UMON] = e1;
#pragma unroll
                for (int col = 0; col < 3; col++) {
#pragma unroll
                    for (int c = 0; c < 3; c++) av[ACC_VIRT + c + 3 * col] = oh[0][c] * dr1[1][col] + oh[1][c] * dr1[2][col];
                    av[ACC_VIRIALC] += ohc[0][col] * dr1[1][col] + ohc[1][col] * dr1[2][col];
                }
            }
        }
        if (in)
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (L > 1 && k != l) continue;
                const size_t s = (size_t)b * S + k * N + w;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    kp.dR[3 * s + c] = (k < 3) ? dr1[k < 3 ? k : 0][c] : 0.0;
                    kp.dip[3 * s + c] = 0.0;
                    kp.Efdr[3 * s + c] = 0.0;
                }
            }
    } else {
        double q3[3], dq3[3][3][3];
        nasa_dms<L>(R, kp.box, kp.boxi, kp.dms1, kp.dms2, kp.dms3, q3, dq3, false, l);
#pragma unroll
        for (int k = 0; k < 3; k++) q3[k] *= CHARGECON;
        const double ig = rcp_newton(1.0 - kp.gammaM), tmp = hg * ig;
        const double q[4] = {0.0, q3[1] + tmp * (q3[1] + q3[2]), q3[2] + tmp * (q3[1] + q3[2]), q3[0] * ig};
        if (in) {
            double *g = kp.grdq + ((size_t)b * N + w) * 27;
#pragma unroll
            for (int a = 0; a < 3; a++) {
                if (L > 1 && a != l) continue;
                kp.chg[(size_t)b * kp.natoms + 3 * w + a] = q3[a];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const double g0 = dq3[a][0][c] * CHARGECON, g1 = dq3[a][1][c] * CHARGECON, s01 = g0 + g1;
                    g[9 * a + 0 + c] = g0 + tmp * s01;
                    g[9 * a + 3 + c] = g1 + tmp * s01;
                    g[9 * a + 6 + c] = dq3[a][2][c] * CHARGECON - 2.0 * tmp * s01;
                }
            }
            // self energy and intramolecular exclusions (pot_ttm.f90:232-261): site k's row
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (L > 1 && k != l) continue;
                double Ef[3] = {0, 0, 0}, ph = k == 0 ? 0.0 : -kp.ew.aewald * TSP * q[k];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (j == k) continue;
                    if (MODEL == 3 && (k == 0 || j == 0)) continue;  // O: no charge, and no dipole to see a field
                    double Rs[3], Rcs[3];
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        Rs[c] = min_image_fast(__dsub_rn(R[k][c], R[j][c]), kp.box[c], kp.boxi[c]);
                        Rcs[c] = min_image_fast(__dsub_rn(Rc[k][c], Rc[j][c]), kp.box[c], kp.boxi[c]);
                    }
                    PairR pr;
                    pair_r(dot3_rn(Rs[0], Rs[1], Rs[2]), kp.ew, pr);
                    const double ts0 = pr.t0 - pr.dri, ts1 = pr.t1 - pr.dri * pr.drsqi;
                    ph += ts0 * q[j];
                    const double a = ts1 * q[j], h = -0.5 * a * q[k];
                    double d[3];
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        Ef[c] += a * Rs[c];
                        d[c] = h * Rs[c];
                        av[ACC_VIRIALC] += Rcs[c] * d[c];
                    }
                    av[ACC_VIRT + 0] += d[0] * Rs[0];
                    av[ACC_VIRT + 4] += d[1] * Rs[1];
                    av[ACC_VIRT + 8] += d[2] * Rs[2];
                    av[ACC_VIRT + 1] += d[0] * Rs[1];
                    av[ACC_VIRT + 2] += d[0] * Rs[2];
                    av[ACC_VIRT + 5] += d[1] * Rs[2];
                }
                const size_t s = (size_t)b * S + k * N + w;
                kp.pos[s] = make_double4_32a(R[k][0], R[k][1], R[k][2], q[k]);
                if (first_bead) kp.posc[(size_t)rep * S + k * N + w] = make_double4_32a(Rc[k][0], Rc[k][1], Rc[k][2], 0.0);
                kp.F[s] = make_double4_32a(Ef[0], Ef[1], Ef[2], ph);
            }
            av[ACC_VIRT + 3] = av[ACC_VIRT + 1];  // (symmetric)
            av[ACC_VIRT + 6] = av[ACC_VIRT + 2];
            av[ACC_VIRT + 7] = av[ACC_VIRT + 5];
            if (MODEL == 2) {  // intramolecular dipole tensors (pot_ttm.f90:344-365), cached per molecule
                int t = 0;
#pragma unroll
                for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int j = i + 1; j < 3; j++, t++) {
                        if (L > 1 && t != l) continue;
                        double Rs[3];
#pragma unroll
                        for (int c = 0; c < 3; c++) Rs[c] = min_image_fast(__dsub_rn(R[i][c], R[j][c]), kp.box[c], kp.boxi[c]);
                        double t1, t2;
                        smear2<double>(dot3_rn(Rs[0], Rs[1], Rs[2]), kp.pt.apol_dd[i + 1][j + 1], kp.ew, &t1, &t2);
                        double *T = kp.Tself + (((size_t)b * N + w) * 3 + t) * 6;
                        T[0] = 3.0 * t2 * Rs[0] * Rs[0] - t1;
                        T[1] = 3.0 * t2 * Rs[1] * Rs[1] - t1;
                        T[2] = 3.0 * t2 * Rs[2] * Rs[2] - t1;
                        T[3] = 3.0 * t2 * Rs[0] * Rs[1];
                        T[4] = 3.0 * t2 * Rs[0] * Rs[2];
                        T[5] = 3.0 * t2 * Rs[1] * Rs[2];
                    }
            }
        }
    }
    block_reduce_add<14, SITES_NT>(av, kp.acc + (size_t)b * NACC);
}

// ---------------------------------------------------------------------------------------
// pot_ttm.f90:273-297: charge forces -q Efq, Uelec, and the initial induced dipoles
// (polarisability times the charge field, or the 4-step predictor from the history).
// pot_ttm.f90:649-675 calc_dpcf: the 4-step predictor coefficients for MD step t, from the
// history slots mod(t,4) (oldest first in the reference's rotation)
PIMD_D double4_32a predictor_coefficients(int t) {
    switch (t % 4) {
        case 0: return make_double4_32a(-1, 4, -6, 4);
        case 1: return make_double4_32a(4, -1, 4, -6);
        case 2: return make_double4_32a(-6, 4, -1, 4);
        default: return make_double4_32a(4, -6, 4, -1);
    }
}

template <int MODEL>
__global__ void __launch_bounds__(128) k_after_qq(KP kp) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y;
    const int t = kp.dstep[0];
    const bool use_pred = (t > 4) && kp.guess;
    const double4_32a dpcf = predictor_coefficients(t);
    double av[3] = {0.0, 0.0, 0.0};
    if (s < kp.S) {
        const size_t gs = (size_t)b * kp.S + s;
        double4_32a F = kp.F[gs];
        if ((kp.fx_mode & 1) && s >= kp.fx_s0) {  // the reciprocal charge field from its scratch
            const double4_32a x = kp.Fx[gs];
            F.x += x.x;
            F.y += x.y;
            F.z += x.z;
            F.w += x.w;
            kp.F[gs] = F;
        }
        const double q = kp.pos[gs].w;
        if (s >= kp.N) {
            kp.dR[3 * gs + 0] -= q * F.x;
            kp.dR[3 * gs + 1] -= q * F.y;
            kp.dR[3 * gs + 2] -= q * F.z;
            av[2] = q * F.w;
        }
        if (s >= kp.fd && s < kp.ld) {
            const int kind = s / kp.N + 1;
            double mu[3];
            if (use_pred) {
                const double *h = kp.txdip + (size_t)b * 4 * kp.S * 3;
                const size_t st = (size_t)kp.S * 3;
#pragma unroll
                for (int c = 0; c < 3; c++)
                    mu[c] = dpcf.x * h[3 * s + c] + dpcf.y * h[st + 3 * s + c] + dpcf.z * h[2 * st + 3 * s + c] +
                            dpcf.w * h[3 * st + 3 * s + c];
            } else {
                mu[0] = kp.polar[kind] * F.x;
                mu[1] = kp.polar[kind] * F.y;
                mu[2] = kp.polar[kind] * F.z;
            }
            kp.dip[3 * gs + 0] = mu[0];
            kp.dip[3 * gs + 1] = mu[1];
            kp.dip[3 * gs + 2] = mu[2];
            const float4 mf = make_float4((float)mu[0], (float)mu[1], (float)mu[2], 0.f);
            if (kp.dipf) kp.dipf[gs] = mf;
            mrec_dipole(kp, b, s, mf);
        }
    }
    block_reduce_add<3, 128>(av, kp.acc + (size_t)b * NACC);  // slot 2 = ACC_UELEC2
}

// pot_ttm.f90:311-365: the real-space dipole field of one iteration (dd_real.cuh)
template <int MODEL>
__global__ void __launch_bounds__(128) k_dd_real(KP kp) {
    dd_real_pairs<MODEL>(kp, blockIdx.y, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

__global__ void k_set_step(int *dstep, int t) {
    if (threadIdx.x == 0) {
        dstep[0] = t;
        dstep[1] = 0;
    }
}

// ---------------------------------------------------------------------------------------

// ---------------------------------------------------------------------------------------
// pot_ttm.f90:556-627: charge-derivative forces grdq*phi, their virials, M-site force
// redistribution onto O/H, dipole outputs, and the predictor history (391-392).
template <int MODEL>
__global__ void __launch_bounds__(128) k_finish(KP kp) {
    using T = TT<MODEL>;
    const int w = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y;
    const int N = kp.N;
    double av[14];
#pragma unroll
    for (int i = 0; i < 14; i++) av[i] = 0.0;
    if (w < N) {
        const size_t base = (size_t)b * kp.S;
        const double4_32a *pos = kp.pos + base;
        const double4_32a *Fb = kp.F + base;
        double *dR = kp.dR + 3 * base;
        double phH1 = Fb[N + w].w, phH2 = Fb[2 * N + w].w, phM = Fb[3 * N + w].w;
        if (kp.fx_mode & 2) {  // the force pass's sums from its scratch (sites from fx_s0 on)
            const double4_32a *X = kp.Fx + base;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int s = k * N + w;
                if (s < kp.fx_s0) continue;
                const double4_32a x = X[s];
                dR[3 * s + 0] += x.x;
                dR[3 * s + 1] += x.y;
                dR[3 * s + 2] += x.z;
                if (k == 1) phH1 += x.w;
                if (k == 2) phH2 += x.w;
                if (k == 3) phM += x.w;
            }
        }
        const double *g = kp.grdq + ((size_t)b * N + w) * 27;
        double dg[3][3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            dg[1][c] = g[0 + 0 + c] * phH1 + g[0 + 3 + c] * phH2 + g[0 + 6 + c] * phM;
            dg[2][c] = g[9 + 0 + c] * phH1 + g[9 + 3 + c] * phH2 + g[9 + 6 + c] * phM;
            dg[0][c] = g[18 + 0 + c] * phH1 + g[18 + 3 + c] * phH2 + g[18 + 6 + c] * phM;
        }
        const double4_32a O = pos[w], H1 = pos[N + w], H2 = pos[2 * N + w], M = pos[3 * N + w];
        const double4_32a *pc = posc_of(kp, b);
        const double4_32a Oc = pc[w], H1c = pc[N + w], H2c = pc[2 * N + w];
        const double o[3] = {O.x, O.y, O.z}, h1[3] = {H1.x, H1.y, H1.z}, h2[3] = {H2.x, H2.y, H2.z};
        const double m[3] = {M.x, M.y, M.z};
        const double oc[3] = {Oc.x, Oc.y, Oc.z}, h1c[3] = {H1c.x, H1c.y, H1c.z}, h2c[3] = {H2c.x, H2c.y, H2c.z};
        double r1[3], r2[3], rc1[3], rc2[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            r1[c] = min_image_rn(__dsub_rn(h1[c], o[c]), kp.box[c], kp.boxi[c]);
            r2[c] = min_image_rn(__dsub_rn(h2[c], o[c]), kp.box[c], kp.boxi[c]);
            rc1[c] = min_image_rn(__dsub_rn(h1c[c], oc[c]), kp.box[c], kp.boxi[c]);
            rc2[c] = min_image_rn(__dsub_rn(h2c[c], oc[c]), kp.box[c], kp.boxi[c]);
        }
#pragma unroll
        for (int ix = 0; ix < 3; ix++)
#pragma unroll
            for (int iy = 0; iy < 3; iy++) av[ACC_VIRT + ix + 3 * iy] += r1[ix] * dg[1][iy] + r2[ix] * dg[2][iy];
#pragma unroll
        for (int c = 0; c < 3; c++) av[ACC_VIRIALC] += rc1[c] * dg[1][c] + rc2[c] * dg[2][c];
        double gO[3], gH1[3], gH2[3], gM[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            gO[c] = dR[3 * w + c] + dg[0][c];
            gH1[c] = dR[3 * (N + w) + c] + dg[1][c];
            gH2[c] = dR[3 * (2 * N + w) + c] + dg[2][c];
            gM[c] = dR[3 * (3 * N + w) + c];
        }
        double *out = kp.dRRt + ((size_t)b * kp.natoms + 3 * w) * 3;
        const double hg = 0.5 * kp.gammaM;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            out[3 + c] = gH1[c] + hg * gM[c];
            out[6 + c] = gH2[c] + hg * gM[c];
            out[c] = gO[c] + (1.0 - kp.gammaM) * gM[c];
        }
        // dipole outputs (pot_ttm.f90:605-627)
        double dI[3], dE[3] = {0, 0, 0};
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double a = min_image_rn(__dsub_rn(h1[c], m[c]), kp.box[c], kp.boxi[c]);
            const double bb = min_image_rn(__dsub_rn(h2[c], m[c]), kp.box[c], kp.boxi[c]);
            dI[c] = H1.w * a + H2.w * bb;
        }
        const double *dip = kp.dip + 3 * base;
        const int slot = kp.dstep[0] % 4;
        double *hist = kp.txdip + ((size_t)b * 4 + slot) * kp.S * 3;
#pragma unroll
        for (int k = T::FDI; k <= T::LDI; k++) {
            const int s = (k - 1) * N + w;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const double mu = dip[3 * s + c];
                dI[c] = mu + dI[c];
                dE[c] = mu;
                if (kp.guess) hist[3 * s + c] = mu;
            }
        }
        double *pI = kp.dipI + ((size_t)b * N + w) * 3, *pE = kp.dipE + ((size_t)b * N + w) * 3;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            pI[c] = dI[c];
            pE[c] = dE[c];
        }
    }
    block_reduce_add<14, 128>(av, kp.acc + (size_t)b * NACC);
}

// pot_ttm.f90:588-591, 628 and force_calc.f90:49: per-bead totals
__global__ void k_totals(KP kp, double *Upott, double *virialt, double *virialct, double *virt9) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= kp.P) return;
    const double *a = kp.acc + (size_t)b * NACC;
    const double En = a[ACC_UMON] + a[ACC_UVDW] + 0.5 * a[ACC_UELEC2] + a[ACC_UIND] + kp.Uvdw_lrc;
    double v[9];
#pragma unroll
    for (int i = 0; i < 9; i++) v[i] = a[ACC_VIRT + i];
    v[0] -= kp.Uvdw_lrc;
    v[4] -= kp.Uvdw_lrc;
    v[8] -= kp.Uvdw_lrc;
    if (Upott) Upott[b] = En;
    if (virialt) virialt[b] = v[0] + v[4] + v[8];
    // pot_spc never sets virialc (its value in the reference is whatever the caller held); 0 here
    if (virialct) virialct[b] = (kp.model >= 4) ? 0.0 : a[ACC_VIRIALC] - 3 * kp.Uvdw_lrc;
    if (virt9)
        for (int i = 0; i < 9; i++) virt9[9 * b + i] = v[i];
}

// ---------------------------------------------------------------------------------------
#define DISPATCH_TTM(E, KERN, GRID, BLOCK, ...)                                              \
    do {                                                                                     \
        if ((E).kp.model == 2)                                                               \
            KERN<2><<<GRID, BLOCK, 0, (E).stream>>>((E).kp, ##__VA_ARGS__);                  \
        else                                                                                 \
            KERN<3><<<GRID, BLOCK, 0, (E).stream>>>((E).kp, ##__VA_ARGS__);                  \
        ++(E).nlaunch;                                                                       \
    } while (0)

static int pair_blocks(const Engine &E) {
    // enough blocks to cover the expected pairs of one bead; the kernels grid-stride
    const long est = (long)E.kp.N * 64;
    long nb = (est + 127) / 128;
    if (nb < 8) nb = 8;
    if (nb > 4096) nb = 4096;
    return (int)nb;
}

void launch_sites(Engine &E) {
    const int N = E.kp.N, P = E.kp.P;
    const dim3 g((2 * N + SITES_NT - 1) / SITES_NT, P);
    if (E.precision == PIMD_PREC_MIXED) {
        if (E.kp.model == 2)
            k_sites<2><<<g, SITES_NT, 0, E.stream>>>(E.kp);
        else
            k_sites<3><<<g, SITES_NT, 0, E.stream>>>(E.kp);
    } else if (lanes_per_molecule(N, P) == 4) {
        const dim3 g4((N + 7) / 8, P);
        if (E.kp.model == 2)
            k_sites64<2, 4><<<g4, SITES_NT, 0, E.stream>>>(E.kp);
        else
            k_sites64<3, 4><<<g4, SITES_NT, 0, E.stream>>>(E.kp);
    } else if (E.kp.model == 2) {
        k_sites64<2, 1><<<g, SITES_NT, 0, E.stream>>>(E.kp);
    } else {
        k_sites64<3, 1><<<g, SITES_NT, 0, E.stream>>>(E.kp);
    }
    ++E.nlaunch;
}

void launch_after_qq(Engine &E) {
    dim3 g((E.kp.S + 127) / 128, E.kp.P);
    DISPATCH_TTM(E, k_after_qq, g, 128);
}

// The force call's accumulators, error word, bad-table flags and iteration count to zero, and the step
// (set: not inside a graph, where its caller sets it): one launch, which took three or four memory sets of about
// 1.5 us each on the call's critical path
__global__ void __launch_bounds__(256) k_begin(KP kp, int *xbad, int t, int set) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < kp.P * NACC) kp.acc[i] = 0.0;
    if (xbad && i < kp.P) xbad[i] = 0;
    if (i == 0) {
        *kp.err = 0u;
        if (set) kp.dstep[0] = t;
        kp.dstep[1] = 0;
    }
}
void launch_begin(Engine &E, int t) {
    k_begin<<<(E.kp.P * NACC + 255) / 256, 256, 0, E.stream>>>(E.kp, E.dg.xbad, t, E.capturing ? 0 : 1);
    ++E.nlaunch;
}
void launch_set_step(Engine &E, int t) {
    k_set_step<<<1, 32, 0, E.stream>>>(E.kp.dstep, t);
    ++E.nlaunch;
}

void launch_dd_real(Engine &E) {
    dim3 g(pair_blocks(E), E.kp.P);
    DISPATCH_TTM(E, k_dd_real, g, 128);
}


void launch_finish(Engine &E) {
    dim3 g((E.kp.N + 127) / 128, E.kp.P);
    DISPATCH_TTM(E, k_finish, g, 128);
}

void launch_totals(Engine &E, double *Upott, double *virialt, double *virialct, double *virt9) {
    k_totals<<<(E.kp.P + 63) / 64, 64, 0, E.stream>>>(E.kp, Upott, virialt, virialct, virt9); ++E.nlaunch;
}

}  // namespace pimd
