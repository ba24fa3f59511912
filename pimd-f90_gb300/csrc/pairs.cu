// pairs.cu -- real-space sums of the FP64 engine: O-O van der Waals and the charges' site pairs of
// every neighbour pair (pot_ttm.f90:159-228, pot_spc.f90:142-191) with the dipole tensors of the
// induced-dipole iterations (pot_ttm.f90:311-342), and the forces on charges and dipoles
// (pot_ttm.f90:399-542).
//
// Bound by FP64 instructions (two lanes a cycle and SM; conversions, compares and shuffled adds
// count too), so the kernel is built to issue few of them:
//   - a lane takes one site of molecule i with all sites of molecule j (3 or 4 lanes a pair), a
//     warp a chunk of pairs: three times the parallelism of a thread per pair in a small system;
//   - the van der Waals terms of the chunk run densely first, one lane a pair;
//   - site pairs within 5 A (one in six at a 9 A cutoff), which take the Thole factors and
//     Q(2/3, x), go to a queue in shared memory and are worked off 32 at a time, instead of
//     making every warp walk that path for a few of its lanes;
//   - minimum images are formed only where a component can exceed half the box (an integer
//     compare of high words; the image is the identity elsewhere, exactly);
//   - erfc and the Gaussian share one exponential, 1/r comes from rsqrt, and 1/(1 + p x) from
//     Newton's iteration;
//   - virials are taken from the summed forces of a lane's site and lever arms from the O site of
//     molecule j, not per site pair: sum_ij d_ij (x) (u_i - v_j) = sum_i G_i (x) u_i - sum_j H_j (x) v_j.
// Measured (GB300), a thread per pair with every test of Q(2/3, x) before: TTM3-F 512 x 32
// 9168 -> 2124 us, TTM2.1-F 128 x 32 3600 -> 865 us, TTM3-F 128 x 1 221 -> 63 us, q-SPC/Fw 256 x 16
// 577 -> 432 us and 32 x 1 51 -> 23 us.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "engine.h"
#include "pair_math.cuh"

namespace pimd {

constexpr int PQ_NT = 128;

// MODEL 2 TTM2.1-F (sites O H H M), 3 TTM3-F (H H M: O has neither charge nor dipole), 4 the SPC
// models (O H H, no damping). NR: rounds of 32 / NI pairs a warp takes per chunk.
template <int MODEL, int NR>
__global__ void __launch_bounds__(PQ_NT) k_pair_qq(KP kp) {
    constexpr int NI = MODEL == 2 ? 4 : 3, PW = 32 / NI, KB0 = MODEL == 3 ? 1 : 0, CH = PW * NR;
    constexpr bool THOLE = MODEL != 4;
    constexpr int QCAP = THOLE ? 31 + 32 * NI + 1 : 1;
    __shared__ double qd[PQ_NT / 32][6][QCAP];  // near site pairs: separation, O-O image shift
    __shared__ int4 qi4[PQ_NT / 32][QCAP];      // molecules i, j, pair, site kinds
    const int b = blockIdx.y, N = kp.N, lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int np = kp.npair[b];
    const double4_32a *pos = kp.pos + (size_t)b * kp.S, *posc = posc_of(kp, b);
    double4_32a *Fb = kp.F + (size_t)b * kp.S;
    double *dRb = kp.dR + (size_t)b * kp.S * 3;
    double vt[6] = {0, 0, 0, 0, 0, 0}, vc = 0.0, uv = 0.0;  // virial xx yy zz xy xz yz, centroid trace, energy
    unsigned err = 0;
    int cnt = 0;

    auto dtensor = [&](int p, int ka, int kb, const double (&R)[3], double t1, double t2) {
        const int t = MODEL == 2 ? 3 * ka + kb : 0;
        double *T = kp.Tdd + (((size_t)b * kp.cap + p) * kp.ndd + t) * 6;
        const double t3 = 3.0 * t2, x = t3 * R[0], y = t3 * R[1];
        T[0] = x * R[0] - t1;
        T[1] = y * R[1] - t1;
        T[2] = t3 * R[2] * R[2] - t1;
        T[3] = x * R[1];
        T[4] = x * R[2];
        T[5] = y * R[2];
    };
    auto isdip = [](int k) { return MODEL == 2 ? k < 3 : MODEL == 3 ? k == 3 : false; };

    // the last n <= 32 records of the queue, one a lane
    auto flush = [&](int n) {
        __syncwarp();
        if (lane < n) {
            const int r = cnt - n + lane;
            const int4 id = qi4[wp][r];
            const double R[3] = {qd[wp][0][r], qd[wp][1][r], qd[wp][2][r]};
            const int ka = id.w >> 2, kb = id.w & 3;
            const size_t ia = (size_t)ka * N + id.x, jb = (size_t)kb * N + id.y;
            const double q1 = pos[ia].w, q2 = pos[jb].w;
            const double d2 = dot3_rn(R[0], R[1], R[2]);
            PairR pr;
            pair_r(d2, kp.ew, pr);
            double t0 = pr.t0, t1 = pr.t1;
            const double r3i = pr.dri * pr.drsqi, x = pr.dd * d2 * kp.pt.apol_qq[ka + 1][kb + 1];
            const double e1 = exp(-x), ra = kp.pt.ra_qq[ka + 1][kb + 1];
            const double rr = ra * pr.dd;
            // x^(2/3) exp(-x) / Gamma(2/3) with x^(2/3) = (a^(1/3) r)^2
            const double q23 = thole_q23(x, e1 * (rr * rr) * kp.gq_norm, kp.gq, &err);
            t1 = t1 - e1 * r3i;
            t0 = t0 - e1 * pr.dri + ra * 1.3541179394264 * q23;
            double *fi = reinterpret_cast<double *>(Fb + ia), *fj = reinterpret_cast<double *>(Fb + jb);
            const double a = t1 * q2, c = t1 * q1;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                atomicAdd(fi + k, a * R[k]);
                atomicAdd(fj + k, -c * R[k]);
            }
            if (ka != 0 && kb != 0) {  // (O is uncharged and its potential unused in the TTM models)
                atomicAdd(fi + 3, t0 * q2);
                atomicAdd(fj + 3, t0 * q1);
                const double w = -a * q1, dx = w * R[0], dy = w * R[1], dz = w * R[2];
                vt[0] += dx * R[0];
                vt[1] += dy * R[1];
                vt[2] += dz * R[2];
                vt[3] += dx * R[1];
                vt[4] += dx * R[2];
                vt[5] += dy * R[2];
                const double4_32a ca = posc[ia], cb = posc[jb];
                vc += dx * (ca.x - cb.x + qd[wp][3][r]) + dy * (ca.y - cb.y + qd[wp][4][r]) + dz * (ca.z - cb.z + qd[wp][5][r]);
            } else if (ka != 0) {
                atomicAdd(fj + 3, t0 * q1);
            } else if (kb != 0) {
                atomicAdd(fi + 3, t0 * q2);
            }
            if (isdip(ka) && isdip(kb)) {
                const double ad = kp.pt.apol_dd[ka + 1][kb + 1];
                const double ed = (MODEL == 3 && kp.same_acd) ? e1 : exp(-(pr.dd * d2 * ad));
                const double t2 = (pr.t1 + kp.ew.cts2 * pr.g) * pr.drsqi;
                // -ch + sr terms of PBCsmear2 (smear.f90:60-66): -e / r^3 and -(e / r^3 + e a) / r^2
                dtensor(id.z, ka, kb, R, pr.t1 - ed * r3i, t2 - (ed * r3i + ed * ad) * pr.drsqi);
            }
        }
        cnt -= n;
        __syncwarp();
    };

    const int step = gridDim.x * (PQ_NT / 32) * CH;
    for (int base = (blockIdx.x * (PQ_NT / 32) + wp) * CH; base < np; base += step) {
        // van der Waals, a lane a pair (pot_ttm.f90:168-190)
        int mi = 0, mj = 0;
        double R0[3] = {0, 0, 0};
        if (lane < CH && base + lane < np) {
            const int2 ij = kp.pairs[(size_t)b * kp.cap + base + lane];
            mi = ij.x;
            mj = ij.y;
            const double4_32a oi = pos[mi], oj = pos[mj];
            const double R[3] = {min_image_near(__dsub_rn(oi.x, oj.x), kp, 0), min_image_near(__dsub_rn(oi.y, oj.y), kp, 1),
                                 min_image_near(__dsub_rn(oi.z, oj.z), kp, 2)};
            const double d2 = dot3_rn(R[0], R[1], R[2]);
            double sc;
            if (MODEL == 4) {
                const double R2i = rcp_newton(d2), R6i = R2i * R2i * R2i, R8i = R6i * R2i;
                uv += R6i * (kp.vdwA * R6i + kp.vdwC);
                sc = R8i * (12.0 * kp.vdwA * R6i + 6.0 * kp.vdwC);
            } else {
                const double ri = rsqrt(d2), d = d2 * ri;
                const double R2i = ri * ri, R4i = R2i * R2i, R6i = R2i * R4i, R8i = R6i * R2i;
                const double tv = kp.vdwD * exp(-kp.vdwE * d);
                uv += R6i * ((kp.vdwA * R6i + kp.vdwB * R4i) + kp.vdwC) + tv;
                const double xr = d - kp.rc1;
                sc = R8i * 6.0 * kp.vdwC + tv * kp.vdwE * ri + (kp.shiftA + kp.shiftB * xr) * (xr * xr);
            }
            const double dx = -(sc * R[0]), dy = -(sc * R[1]), dz = -(sc * R[2]);
            double *di = dRb + 3 * mi, *dj = dRb + 3 * mj;
            atomicAdd(di + 0, dx);
            atomicAdd(di + 1, dy);
            atomicAdd(di + 2, dz);
            atomicAdd(dj + 0, -dx);
            atomicAdd(dj + 1, -dy);
            atomicAdd(dj + 2, -dz);
            vt[0] += dx * R[0];
            vt[1] += dy * R[1];
            vt[2] += dz * R[2];
            vt[3] += dx * R[1];
            vt[4] += dx * R[2];
            vt[5] += dy * R[2];
            if (MODEL != 4) {
                const double4_32a ci = posc[mi], cj = posc[mj];
                vc += min_image_near(__dsub_rn(ci.x, cj.x), kp, 0) * dx + min_image_near(__dsub_rn(ci.y, cj.y), kp, 1) * dy +
                      min_image_near(__dsub_rn(ci.z, cj.z), kp, 2) * dz;
            }
            R0[0] = __dadd_rn(__dsub_rn(R[0], oi.x), oj.x);
            R0[1] = __dadd_rn(__dsub_rn(R[1], oi.y), oj.y);
            R0[2] = __dadd_rn(__dsub_rn(R[2], oi.z), oj.z);
        }
#pragma unroll 1
        for (int rd = 0; rd < NR; rd++) {
            const int src = min(31, rd * PW + lane / NI), m = lane % NI, p = base + src;
            const bool act = lane < PW * NI && p < np;
            const int i = __shfl_sync(0xffffffffu, mi, src), j = __shfl_sync(0xffffffffu, mj, src);
            double S0[3];
#pragma unroll
            for (int c = 0; c < 3; c++) S0[c] = __shfl_sync(0xffffffffu, R0[c], src);
            const int ka = KB0 + m;
            double4_32a si, oj;
            double u[3] = {0, 0, 0}, F[4] = {0, 0, 0, 0}, Fj[NI][4];
#pragma unroll
            for (int k = 0; k < NI; k++) Fj[k][0] = Fj[k][1] = Fj[k][2] = Fj[k][3] = 0.0;
            if (act) {  // site ka of molecule i, from the O site of j
                si = pos[(size_t)ka * N + i];
                oj = pos[j];
                u[0] = si.x + S0[0] - oj.x;
                u[1] = si.y + S0[1] - oj.y;
                u[2] = si.z + S0[2] - oj.z;
            }
#pragma unroll
            for (int k = 0; k < NI; k++) {
                const int kb = KB0 + k;
                double R[3] = {0, 0, 0}, d2 = 0.0, q2 = 0.0;
                bool near = false, moved = false;
                double sh[3] = {0, 0, 0};
                if (act) {
                    const double4_32a sj = pos[(size_t)kb * N + j];
                    R[0] = u[0] - (sj.x - oj.x);
                    R[1] = u[1] - (sj.y - oj.y);
                    R[2] = u[2] - (sj.z - oj.z);
                    q2 = sj.w;
                    if (hi_abs(R[0]) >= kp.box49[0] || hi_abs(R[1]) >= kp.box49[1] || hi_abs(R[2]) >= kp.box49[2]) {
#pragma unroll
                        for (int c = 0; c < 3; c++) {
                            const double w = min_image_rn(R[c], kp.box[c], kp.boxi[c]);
                            sh[c] = w - R[c];
                            R[c] = w;
                        }
                        moved = true;
                    }
                    d2 = dot3_rn(R[0], R[1], R[2]);
                    near = THOLE && __double2hiint(d2) < 0x40390000;  // d2 < 25
                }
                if (THOLE) {
                    const unsigned mk = __ballot_sync(0xffffffffu, near);
                    if (near) {
                        const int r = cnt + __popc(mk & ((1u << lane) - 1u));
#pragma unroll
                        for (int c = 0; c < 3; c++) {
                            qd[wp][c][r] = R[c];
                            qd[wp][3 + c][r] = S0[c];
                        }
                        qi4[wp][r] = make_int4(i, j, p, ka * 4 + kb);
                    }
                    cnt += __popc(mk);
                }
                if (act && !near) {
                    PairR pr;
                    pair_r(d2, kp.ew, pr);
                    const double a = pr.t1 * q2, c = pr.t1 * si.w;
#pragma unroll
                    for (int x = 0; x < 3; x++) {
                        F[x] += a * R[x];
                        Fj[k][x] -= c * R[x];
                    }
                    F[3] += pr.t0 * q2;
                    Fj[k][3] += pr.t0 * si.w;
                    if (moved) {  // the part of R that the lever arms below do not hold
                        const double w = -a * si.w, dx = w * R[0], dy = w * R[1], dz = w * R[2];
                        vt[0] += dx * sh[0];
                        vt[1] += dy * sh[1];
                        vt[2] += dz * sh[2];
                        vt[3] += dx * sh[1];
                        vt[4] += dx * sh[2];
                        vt[5] += dy * sh[2];
                    }
                    if (isdip(ka) && isdip(kb)) dtensor(p, ka, kb, R, pr.t1, (pr.t1 + kp.ew.cts2 * pr.g) * pr.drsqi);
                }
            }
            // lane m takes the sums of site m of molecule j from its pair's lanes
            double H[4];
#pragma unroll
            for (int x = 0; x < 4; x++) {
                H[x] = Fj[0][x];
#pragma unroll
                for (int k = 1; k < NI; k++) H[x] = m == k ? Fj[k][x] : H[x];
            }
#pragma unroll
            for (int r = 1; r < NI; r++) {
                const int from = min(31, lane - m + (m + r) % NI), give = (m + NI - r) % NI;
#pragma unroll
                for (int x = 0; x < 4; x++) {
                    double v = Fj[0][x];
#pragma unroll
                    for (int k = 1; k < NI; k++) v = give == k ? Fj[k][x] : v;
                    H[x] += __shfl_sync(0xffffffffu, v, from);
                }
            }
            if (act) {
                const size_t ia = (size_t)ka * N + i, jb = (size_t)ka * N + j;
                const double4_32a sj = pos[jb];
                double *fi = reinterpret_cast<double *>(Fb + ia), *fj = reinterpret_cast<double *>(Fb + jb);
#pragma unroll
                for (int x = 0; x < 3; x++) {
                    atomicAdd(fi + x, F[x]);
                    atomicAdd(fj + x, H[x]);
                }
                if (MODEL == 4 || ka != 0) {
                    atomicAdd(fi + 3, F[3]);
                    atomicAdd(fj + 3, H[3]);
                }
                if (MODEL == 4 || ka != 0) {
                    const double G[3] = {-si.w * F[0], -si.w * F[1], -si.w * F[2]};
                    const double D[3] = {sj.w * H[0], sj.w * H[1], sj.w * H[2]};
                    const double v[3] = {sj.x - oj.x, sj.y - oj.y, sj.z - oj.z};
                    vt[0] += G[0] * u[0] - D[0] * v[0];
                    vt[1] += G[1] * u[1] - D[1] * v[1];
                    vt[2] += G[2] * u[2] - D[2] * v[2];
                    vt[3] += G[0] * u[1] - D[0] * v[1];
                    vt[4] += G[0] * u[2] - D[0] * v[2];
                    vt[5] += G[1] * u[2] - D[1] * v[2];
                    if (MODEL != 4) {
                        const double4_32a ca = posc[ia], cb = posc[jb];
                        vc += G[0] * (ca.x + S0[0] - oj.x) + G[1] * (ca.y + S0[1] - oj.y) + G[2] * (ca.z + S0[2] - oj.z) -
                              D[0] * (cb.x - oj.x) - D[1] * (cb.y - oj.y) - D[2] * (cb.z - oj.z);
                    }
                }
            }
            if (THOLE)
                while (cnt >= 32) flush(32);
        }
    }
    if (THOLE && cnt > 0) flush(cnt);
    if (err) atomicOr(kp.err, err);
    pair_block_sums<PQ_NT>(vt, vc, uv, kp.acc + (size_t)b * NACC);
}

// Chunks of NI rounds where they fill the chip, of one round where they do not; blocks for one
// pass over the expected pairs, at most about five a SM, so that a
// block's closing sums are few.
template <int MODEL>
static void pair_qq(Engine &E) {
    constexpr int NI = MODEL == 2 ? 4 : 3, PW = 32 / NI;
    const long est = std::max(1L, (long)E.pair_est), P = E.kp.P;
    const long full = (est + 4L * PW * NI - 1) / (4L * PW * NI);
    if (full * P >= 2 * E.nsm) {
        const long nb = std::max(1L, std::min(full, (5L * E.nsm + P - 1) / P));
        k_pair_qq<MODEL, NI><<<dim3((unsigned)nb, (unsigned)P), PQ_NT, 0, E.stream>>>(E.kp);
    } else {
        const long nb = std::max(1L, (est + 4L * PW - 1) / (4L * PW));
        k_pair_qq<MODEL, 1><<<dim3((unsigned)nb, (unsigned)P), PQ_NT, 0, E.stream>>>(E.kp);
    }
    ++E.nlaunch;
}

void launch_pair_qq(Engine &E) {
    if (E.kp.model == 2)
        pair_qq<2>(E);
    else if (E.kp.model == 3)
        pair_qq<3>(E);
    else
        pair_qq<4>(E);
}

// pot_ttm.f90:399-542: real-space forces on charges and dipoles (charge-dipole and dipole-dipole), the
// dipole part of phi, and the intramolecular terms. A lane takes one site pair: TTM3-F five a molecule
// pair (H1 M, H2 M, M M, M H1, M H2: six pairs a warp), TTM2.1-F sixteen (two pairs a warp, M M idle);
// the sites' sums are formed by shuffles and added with one atomic a component. Bound by FP64
// instructions like the charge sums; a thread per pair, with exponentials and divisions of its own for
// each term, took 1520 us at TTM3-F 512 x 32, 917 us at TTM2.1-F 128 x 32 and 80 us at 128 x 1.
template <int MODEL>
PIMD_D void force_term(const KP &kp, const double (&R)[3], double d2, int ka, int kb, double q1, double q2, const double (&m1)[3],
                       const double (&m2)[3], double (&f)[3], double &p1, double &p2) {
    const bool dd = MODEL == 2 ? (ka < 3 && kb < 3) : (ka == 3 && kb == 3);
    PairR pr;
    pair_r(d2, kp.ew, pr);
    const double t2 = (pr.t1 + kp.ew.cts2 * pr.g) * pr.drsqi;
    double c1 = pr.t1, c2 = t2, d2t = t2, d3t = (t2 + kp.ew.cts3 * pr.g) * pr.drsqi;
    if (__double2hiint(d2) < 0x40390000) {  // r < 5 A: the Thole factors (smear.f90:36-107)
        const double r3 = pr.dd * d2, r3i = pr.dri * pr.drsqi;
        const double a = kp.pt.apol_cd[ka + 1][kb + 1], e = exp(-r3 * a), s2 = (e * r3i + e * a) * pr.drsqi;
        c1 -= e * r3i;
        c2 -= s2;
        if (dd) {
            const double ad = kp.pt.apol_dd[ka + 1][kb + 1], ed = kp.same_acd ? e : exp(-r3 * ad);
            const double sd = kp.same_acd ? s2 : (ed * r3i + ed * ad) * pr.drsqi;
            d2t -= sd;
            d3t -= (sd + 0.6 * ed * pr.dd * ad * ad) * pr.drsqi;
        }
    }
    f[0] = f[1] = f[2] = p1 = p2 = 0.0;
    if (dd) dd_force(R, m1, m2, d2t, d3t, f);
    const double qd[3] = {q2 * m1[0] - q1 * m2[0], q2 * m1[1] - q1 * m2[1], q2 * m1[2] - q1 * m2[2]};
    if (qd[0] * qd[0] + qd[1] * qd[1] + qd[2] * qd[2] > 1.e-9) {
        const double w = 3.0 * c2 * (R[0] * qd[0] + R[1] * qd[1] + R[2] * qd[2]);
#pragma unroll
        for (int c = 0; c < 3; c++) f[c] += w * R[c] - c1 * qd[c];
        p1 = c1 * (R[0] * m2[0] + R[1] * m2[1] + R[2] * m2[2]);
        p2 = -c1 * (R[0] * m1[0] + R[1] * m1[1] + R[2] * m1[2]);
    }
}

template <int MODEL>
__global__ void __launch_bounds__(PQ_NT) k_pair_force(KP kp) {
    constexpr int NL = MODEL == 2 ? 16 : 5, PW = 32 / NL;  // lanes a pair, pairs a warp
    const int b = blockIdx.y, N = kp.N, lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int np = kp.npair[b], nwarp = gridDim.x * (PQ_NT / 32), w0 = blockIdx.x * (PQ_NT / 32) + wp;
    const double4_32a *pos = kp.pos + (size_t)b * kp.S, *posc = posc_of(kp, b);
    const double *dip = kp.dip + (size_t)b * kp.S * 3;
    double *dR = kp.dR + (size_t)b * kp.S * 3;
    double4_32a *Fb = kp.F + (size_t)b * kp.S;
    double av[14];
#pragma unroll
    for (int i = 0; i < 14; i++) av[i] = 0.0;
    auto isdip = [](int k) { return MODEL == 2 ? k < 3 : k == 3; };
    auto site = [&](int k, int mol, double &q, double (&m)[3]) {
        const size_t s = (size_t)k * N + mol;
        const double4_32a r = pos[s];
        q = r.w;
        m[0] = m[1] = m[2] = 0.0;
        if (isdip(k))
#pragma unroll
            for (int c = 0; c < 3; c++) m[c] = dip[3 * s + c];
        return r;
    };
    auto virial = [&](const double (&f)[3], const double (&R)[3], const double (&Rc)[3]) {
        av[ACC_VIRIALC] += Rc[0] * f[0] + Rc[1] * f[1] + Rc[2] * f[2];
#pragma unroll
        for (int col = 0; col < 3; col++)
#pragma unroll
            for (int c = 0; c < 3; c++) av[ACC_VIRT + c + 3 * col] += f[c] * R[col];
    };
    const int r = lane % NL;
    const int ka = MODEL == 2 ? r >> 2 : r < 2 ? r + 1 : 3, kb = MODEL == 2 ? r & 3 : r < 3 ? 3 : r - 2;
    for (int base = w0 * PW; base < np; base += nwarp * PW) {
        const int p = base + lane / NL;
        const bool act = lane < PW * NL && p < np && !(MODEL == 2 && r == 15);
        int i = 0, j = 0;
        double f[3] = {0, 0, 0}, p1 = 0.0, p2 = 0.0;
        if (act) {
            const int2 ij = kp.pairs[(size_t)b * kp.cap + p];
            i = ij.x, j = ij.y;
            double q1, q2, m1[3], m2[3];
            const double4_32a oi = pos[i], oj = pos[j], s1 = site(ka, i, q1, m1), s2 = site(kb, j, q2, m2);
            // the separation from the O sites' image (a second one only where a component can need it)
            const double R[3] = {min_image_near(min_image_near(oi.x - oj.x, kp, 0) + ((s1.x - oi.x) - (s2.x - oj.x)), kp, 0),
                                 min_image_near(min_image_near(oi.y - oj.y, kp, 1) + ((s1.y - oi.y) - (s2.y - oj.y)), kp, 1),
                                 min_image_near(min_image_near(oi.z - oj.z, kp, 2) + ((s1.z - oi.z) - (s2.z - oj.z)), kp, 2)};
            force_term<MODEL>(kp, R, dot3_rn(R[0], R[1], R[2]), ka, kb, q1, q2, m1, m2, f, p1, p2);
            // (the reference takes the centroids' separation as it is, pot_ttm.f90:468)
            const double4_32a ca = posc[(size_t)ka * N + i], cb = posc[(size_t)kb * N + j];
            const double Rc[3] = {ca.x - cb.x, ca.y - cb.y, ca.z - cb.z};
            virial(f, R, Rc);
        }
        double g[4] = {f[0], f[1], f[2], p1}, h[4] = {-f[0], -f[1], -f[2], p2};
        if (MODEL == 2) {
#pragma unroll
            for (int x = 0; x < 4; x++) {
                g[x] += __shfl_xor_sync(0xffffffffu, g[x], 1);
                g[x] += __shfl_xor_sync(0xffffffffu, g[x], 2);
                h[x] += __shfl_xor_sync(0xffffffffu, h[x], 4);
                h[x] += __shfl_xor_sync(0xffffffffu, h[x], 8);
            }
            // sums of site ka of i in the lanes of a row, of site kb of j in those of a column; the lanes
            // of the diagonal add one of each
            if (lane / NL + base < np && ka == kb) {
                const int2 ij = kp.pairs[(size_t)b * kp.cap + base + lane / NL];
                const size_t s1 = (size_t)ka * N + ij.x, s2 = (size_t)ka * N + ij.y;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    atomicAdd(dR + 3 * s1 + c, g[c]);
                    atomicAdd(dR + 3 * s2 + c, h[c]);
                }
                if (ka != 0) {
                    atomicAdd(&Fb[s1].w, g[3]);
                    atomicAdd(&Fb[s2].w, h[3]);
                }
            }
        } else {
            // M of i takes lanes 2, 3, 4 of its pair, M of j lanes 0, 1, 2; both in lane 2 (the forces only:
            // the other lanes have a potential at their own H site or none)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const double a = __shfl_down_sync(0xffffffffu, f[c], 1), d = __shfl_down_sync(0xffffffffu, f[c], 2);
                const double u = __shfl_up_sync(0xffffffffu, f[c], 1), v = __shfl_up_sync(0xffffffffu, f[c], 2);
                if (r == 2) {
                    g[c] = f[c] + (a + d);
                    h[c] = -(f[c] + (u + v));
                }
            }
            const double a = __shfl_down_sync(0xffffffffu, p1, 1), d = __shfl_down_sync(0xffffffffu, p1, 2);
            const double u = __shfl_up_sync(0xffffffffu, p2, 1), v = __shfl_up_sync(0xffffffffu, p2, 2);
            if (r == 2) {
                g[3] = p1 + (a + d);
                h[3] = p2 + (u + v);
            }
            if (act && r <= 2) {
                const size_t s1 = (size_t)ka * N + i;
#pragma unroll
                for (int c = 0; c < 3; c++) atomicAdd(dR + 3 * s1 + c, g[c]);
                atomicAdd(&Fb[s1].w, g[3]);
            }
            if (act && r >= 2) {
                const size_t s2 = (size_t)kb * N + j;
#pragma unroll
                for (int c = 0; c < 3; c++) atomicAdd(dR + 3 * s2 + c, h[c]);
                atomicAdd(&Fb[s2].w, h[3]);
            }
        }
    }
    // intramolecular (pot_ttm.f90:482-542): a lane a site pair, six a molecule, five molecules a warp
    for (int base = w0 * 5; base < N; base += nwarp * 5) {
        const int w = base + lane / 6, t = lane % 6;
        if (lane >= 30 || w >= N) continue;
        const int k1 = t < 3 ? 0 : t < 5 ? 1 : 2, k2 = t < 3 ? t + 1 : t < 5 ? t - 1 : 3;
        double q1, q2, m1[3], m2[3];
        const double4_32a s1 = site(k1, w, q1, m1), s2 = site(k2, w, q2, m2);
        const double4_32a ca = posc[(size_t)k1 * N + w], cb = posc[(size_t)k2 * N + w];
        const double R[3] = {min_image_near(s1.x - s2.x, kp, 0), min_image_near(s1.y - s2.y, kp, 1), min_image_near(s1.z - s2.z, kp, 2)};
        const double Rc[3] = {min_image_near(ca.x - cb.x, kp, 0), min_image_near(ca.y - cb.y, kp, 1), min_image_near(ca.z - cb.z, kp, 2)};
        const double d2 = dot3_rn(R[0], R[1], R[2]);
        double f[3] = {0, 0, 0};
        if (isdip(k1) && isdip(k2)) {
            double t1, t2, t3;
            smear3<double>(d2, kp.pt.apol_dd[k1 + 1][k2 + 1], kp.ew, &t1, &t2, &t3);
            dd_force(R, m1, m2, t2, t3, f);
        }
        // self2 (smear.f90:133-156): the screened interaction less the whole one
        PairR pr;
        pair_r(d2, kp.ew, pr);
        const double r3i = pr.dri * pr.drsqi, ts1 = pr.t1 - r3i, ts2 = (pr.t1 + kp.ew.cts2 * pr.g) * pr.drsqi - r3i * pr.drsqi;
        const double qd[3] = {q2 * m1[0] - q1 * m2[0], q2 * m1[1] - q1 * m2[1], q2 * m1[2] - q1 * m2[2]};
        const double x = 3.0 * ts2 * (R[0] * qd[0] + R[1] * qd[1] + R[2] * qd[2]);
        const size_t a1 = (size_t)k1 * N + w, a2 = (size_t)k2 * N + w;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            f[c] += x * R[c] - ts1 * qd[c];
            atomicAdd(dR + 3 * a1 + c, f[c]);
            atomicAdd(dR + 3 * a2 + c, -f[c]);
        }
        if (k1 != 0) atomicAdd(&Fb[a1].w, ts1 * (R[0] * m2[0] + R[1] * m2[1] + R[2] * m2[2]));
        atomicAdd(&Fb[a2].w, -ts1 * (R[0] * m1[0] + R[1] * m1[1] + R[2] * m1[2]));
        virial(f, R, Rc);
    }
    block_reduce_add<14, PQ_NT>(av, kp.acc + (size_t)b * NACC);
}

// Blocks for one pass over the expected pairs, at most about four a SM
void launch_pair_force(Engine &E) {
    const long P = E.kp.P, pw = E.kp.model == 2 ? 2 : 6;
    const long full = std::max((long)(E.kp.N + 19) / 20, (long)(E.pair_est / (4 * pw)) + 1);
    const dim3 g((unsigned)std::max(1L, std::min(full, (4L * E.nsm + P - 1) / P)), (unsigned)P);
    if (E.kp.model == 2)
        k_pair_force<2><<<g, PQ_NT, 0, E.stream>>>(E.kp);
    else
        k_pair_force<3><<<g, PQ_NT, 0, E.stream>>>(E.kp);
    ++E.nlaunch;
}

// ---- Q(2/3, x): where the reference's iterations stop --------------------------------------
// math.f90:188-285 sums a series (x < 5/3) or a continued fraction until a term falls below
// 3e-7, so its value depends on the number of terms, which for both is a monotone function of x.
// The bounds where the number changes are found here by bisection with the reference's own loops;
// the device runs that number of terms without the tests (and divisions) of each.
static int series_terms(double x) {
    const double a = 2.0 / 3.0;
    double ap = a, sum = 1.0 / a, del = sum;
    for (int n = 1; n <= 800; n++) {
        ap += 1.0;
        del = del * x / ap;
        sum += del;
        if (std::fabs(del) < std::fabs(sum) * 3.e-7) return n;
    }
    return 800;
}
static int fraction_terms(double x) {
    const double a = 2.0 / 3.0, tiny = 1.e-30;
    double b = x + 1.0 - a, c = 1.0 / tiny, d = 1.0 / b;
    for (int i = 1; i <= 100; i++) {
        const double an = -i * (i - a);
        b += 2.0;
        d = an * d + b;
        if (std::fabs(d) < tiny) d = tiny;
        c = b + an / c;
        if (std::fabs(c) < tiny) c = tiny;
        d = 1.0 / d;
        if (std::fabs(d * c - 1.0) < 3.e-7) return i;
    }
    return 100;
}

static GqBounds q23_bounds() {
    const double split = 2.0 / 3.0 + 1.0;
    GqBounds g;
    for (int n = 0; n <= GQ_TERMS; n++) {
        // largest x < split with at most n series terms; smallest x >= split with at most n of the fraction
        double lo = 0.0, hi = split;
        for (int it = 0; it < 64 && n > 0; it++) {
            const double m = 0.5 * (lo + hi);
            (series_terms(m) <= n ? lo : hi) = m;
        }
        g.ser[n] = lo;
        g.inv[n] = 1.0 / (2.0 / 3.0 + n);
        lo = split;
        hi = 1.0e9;
        if (fraction_terms(split) <= n) hi = split;
        for (int it = 0; it < 96 && n > 0 && hi > lo; it++) {
            const double m = 0.5 * (lo + hi);
            (fraction_terms(m) <= n ? hi : lo) = m;
        }
        g.fra[n] = hi;
    }
    return g;
}

void pair_math_init(Engine &E) {
    KP &kp = E.kp;
    static const GqBounds bounds = q23_bounds();  // of the reference's algorithm alone
    kp.gq = bounds;
    kp.gq_norm = std::exp(-0.303150275147547);  // 1 / Gamma(2/3) as the reference's gln has it
    const double at[3] = {0.49, 0.51, 1.49};
    for (int c = 0; c < 3; c++)
        for (int i = 0; i < 3; i++) {
            const double h = at[i] * kp.box[c];
            unsigned long long u;
            std::memcpy(&u, &h, sizeof u);
            (i == 0 ? kp.box49 : i == 1 ? kp.box51 : kp.box149)[c] = (int)(u >> 32);
        }
}

}  // namespace pimd
