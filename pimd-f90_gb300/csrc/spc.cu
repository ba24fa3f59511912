// spc.cu -- q-SPC/Fw (pot_model 4) and SPC/F (pot_model 5) force call for all beads (FP64).
// Restates pot_ttm/pot_spc.f90:1-277: harmonic (q-SPC/Fw) or Toukan-Rahman (SPC/F)
// monomers, O-O Lennard-Jones, the 3x3 screened-Coulomb site sums of every neighbour
// pair, self and intramolecular exclusion terms, and the Ewald reciprocal sum with its
// virial (ewald.f90:230-291, ewald_pw_std_qq). No induced dipoles, no M site.
//
// Sites per bead are O(0..N-1) H1(N..2N-1) H2(2N..3N-1) with fixed charges. The neighbour
// list and Ewald kernels are the TTM engine's (the Ewald charge sums cover all 3N sites).
// Decomposition: the intramolecular work by roles of a block's warps (k_sites_spc), one thread per
// molecule in the epilogue; the real-space sums are the pair kernel of pairs.cu, and the reciprocal
// passes run beside them.
#include "engine.h"
#include "pair_math.cuh"

namespace pimd {

// r - box*anint(r/box): pot_spc.f90 divides by the box in its intramolecular, self and
// dipole terms (pot_spc.f90:74-75, 211, 261, 264) where pot_ttm multiplies by 1/box.
PIMD_D double min_image_div_rn(double r, double box) {
    return __dsub_rn(r, __dmul_rn(box, round(__ddiv_rn(r, box))));
}

// the same by the cell r lies in, where that is beyond doubt (as min_image_near)
PIMD_D double min_image_near_div(double r, const KP &kp, int c) {
    const int h = hi_abs(r);
    if (h < kp.box49[c]) return r;
    if (h >= kp.box51[c] && h < kp.box149[c]) return __dsub_rn(r, copysign(kp.box[c], r));
    return min_image_div_rn(r, kp.box[c]);
}

// |v| and 1/|v|: the square root by a Newton step from the reciprocal one
PIMD_D void norm_inv(const double (&v)[3], double &d, double &di) {
    const double s = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
    di = rsqrt(s);
    d = s * di;
    d += 0.5 * di * fma(-d, d, s);
}

// pot_spc.f90:54-137, 201-233 and 258-267: site layout, monomer energy/gradient and virial,
// self energy, intramolecular Ewald exclusions, charges and molecular dipoles. A block takes 32
// molecules: warps 0-2 an exclusion each, then a site each; warp 3 the monomer. Bound by the chain of
// FP64 instructions of a warp (64 cycles each) and not by the number of molecules: with all of a
// molecule's terms in one thread 44 us, by roles 10 us at 32 molecules x 1 bead.
template <int MODEL>
__global__ void __launch_bounds__(128) k_sites_spc(KP kp) {
    __shared__ double4_32a xc[3][32];  // an exclusion's ts1 R and ts0
    const int lane = threadIdx.x & 31, role = threadIdx.x >> 5;
    const int w = blockIdx.x * 32 + lane, b = blockIdx.y;
    const int N = kp.N;
    const bool valid = w < N;
    double av[ACC_VIRT + 9];
#pragma unroll
    for (int i = 0; i < ACC_VIRT + 9; i++) av[i] = 0.0;
    const double *RR = kp.RRt + (size_t)b * kp.natoms * 3 + 9 * (valid ? w : 0);
    auto sep = [&](int i, int j, double (&r)[3]) {
#pragma unroll
        for (int c = 0; c < 3; c++) r[c] = min_image_near_div(RR[3 * i + c] - RR[3 * j + c], kp, c);
    };
    const double qO = kp.qO * CHARGECON, qH = kp.qH * CHARGECON;
    if (role < 3) {
        // pot_spc.f90:201-233 the intramolecular exclusions O H1, O H2, H1 H2
        const int i = role == 2, j = role == 0 ? 1 : 2;
        const double qi = i ? qH : qO;
        double Rs[3];
        sep(i, j, Rs);
        PairR pr;
        pair_r(Rs[0] * Rs[0] + Rs[1] * Rs[1] + Rs[2] * Rs[2], kp.ew, pr);
        const double ts0 = pr.t0 - pr.dri, ts1 = pr.t1 - pr.dri * pr.drsqi;
        const double f[3] = {ts1 * Rs[0], ts1 * Rs[1], ts1 * Rs[2]};
        xc[role][lane] = make_double4_32a(f[0], f[1], f[2], ts0);
        if (valid) {
            const double m = -qi * qH;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const double g = m * f[c];
#pragma unroll
                for (int col = 0; col <= c; col++) av[ACC_VIRT + c + 3 * col] = av[ACC_VIRT + col + 3 * c] = g * Rs[col];
            }
        }
    } else {
        double r1[3], r2[3], g1[3], g2[3], d1, d2, i1, i2;  // O-H vectors and the H sites' gradients
        sep(1, 0, r1);
        sep(2, 0, r2);
        norm_inv(r1, d1, i1);
        norm_inv(r2, d2, i2);
        const double x1 = d1 - kp.roh0, x2 = d2 - kp.roh0;
        double e1;
        if (MODEL == 4) {
            // pot_spc.f90:73-104 harmonic O-H stretches and H-O-H bend
            const double ax = r1[1] * r2[2] - r1[2] * r2[1], ay = r1[2] * r2[0] - r1[0] * r2[2], az = r1[0] * r2[1] - r1[1] * r2[0];
            const double a2 = ax * ax + ay * ay + az * az, ai = rsqrt(a2);
            const double dot = r1[0] * r2[0] + r1[1] * r2[1] + r1[2] * r2[2];
            const double xa = atan2(sqrt(a2), dot) - kp.th0;  // (the reference divides both by |r1| |r2|)
            e1 = kp.harmkb * (x1 * x1 + x2 * x2) + kp.harmka * (xa * xa);
            // d(angle)/dr1 = -(r2 / (d1 d2) - cos r1 / d1^2) / sin
            const double ta = -2.0 * kp.harmka * xa * ai;
            const double u1 = 2.0 * kp.harmkb * x1 * i1 - ta * dot * (i1 * i1), u2 = 2.0 * kp.harmkb * x2 * i2 - ta * dot * (i2 * i2);
#pragma unroll
            for (int c = 0; c < 3; c++) {
                g1[c] = u1 * r1[c] + ta * r2[c];
                g2[c] = u2 * r2[c] + ta * r1[c];
            }
        } else {
            // pot_spc.f90:107-137 SPC/F (Toukan-Rahman) stretch-bend polynomial
            const double Ap = 671.288262912, Bp = 164.376, Cp = -211.536, Dp = 111.744;
            const double rhh0 = 2.0 * sin(0.5 * kp.th0) * kp.roh0;
            double rh[3], d3, i3;
            sep(1, 2, rh);
            norm_inv(rh, d3, i3);
            const double x3 = d3 - rhh0;
            e1 = Ap * (x1 * x1 + x2 * x2) + Bp * x3 * x3 + Cp * (x1 + x2) * x3 + Dp * x1 * x2;
            const double u1 = (2.0 * Ap * x1 + Cp * x3 + Dp * x2) * i1, u2 = (2.0 * Ap * x2 + Cp * x3 + Dp * x1) * i2;
            const double u3 = (2.0 * Bp * x3 + Cp * (x1 + x2)) * i3;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                g1[c] = u1 * r1[c] + u3 * rh[c];
                g2[c] = u2 * r2[c] - u3 * rh[c];
            }
        }
        if (valid) {
            av[ACC_UMON] = e1;
#pragma unroll
            for (int iy = 0; iy < 3; iy++)
#pragma unroll
                for (int c = 0; c < 3; c++) av[ACC_VIRT + c + 3 * iy] = r1[c] * g1[iy] + r2[c] * g2[iy];
            double *dR = kp.dR + 3 * ((size_t)b * kp.S + w);
            // pot_spc.f90:258-267 molecular dipoles from the O-H vectors
            double *pI = kp.dipI + ((size_t)b * N + w) * 3, *pE = kp.dipE + ((size_t)b * N + w) * 3;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                dR[c] = -g1[c] - g2[c];
                dR[3 * N + c] = g1[c];
                dR[6 * N + c] = g2[c];
                pI[c] = qH * r1[c] + qH * r2[c];
                pE[c] = 0.0;  // pot_spc has no induced dipoles (Edip_mom is not written)
            }
        }
    }
    __syncthreads();
    if (role < 3 && valid) {
        // the site's field and potential: its own term and those of its two exclusions
        const int k = role;
        const double4_32a a = xc[k == 2 ? 1 : 0][lane], c = xc[k == 0 ? 1 : 2][lane];
        const double q = k == 0 ? qO : qH, qa = k == 0 ? qH : qO, sa = k == 0 ? qH : -qO, sc = k == 2 ? -qH : qH;
        const size_t s = (size_t)b * kp.S + k * N + w;
        kp.pos[s] = make_double4_32a(RR[3 * k], RR[3 * k + 1], RR[3 * k + 2], q);
        kp.F[s] = make_double4_32a(sa * a.x + sc * c.x, sa * a.y + sc * c.y, sa * a.z + sc * c.z,
                                   -kp.ew.aewald * TSP * q + qa * a.w + qH * c.w);
        kp.chg[(size_t)b * kp.natoms + 3 * w + k] = q;
    }
    block_reduce_add<ACC_VIRT + 9, 128>(av, kp.acc + (size_t)b * NACC);
}

// pot_spc.f90:245-249, 270-275: Uelec = 1/2 sum q phi, charge forces -q Efq, and the
// gradient in the caller's O H H atom order. A thread takes a site and adds the reciprocal field's
// slices (sites [s0, s1), kp.Fpart) itself.
__global__ void __launch_bounds__(128) k_finish_spc(KP kp, int s0, int s1, int ns) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y;
    const int N = kp.N;
    double av[1] = {0.0};
    if (s < kp.S) {
        const size_t gs = (size_t)b * kp.S + s;
        double4_32a f = kp.F[gs];
        if (s >= s0 && s < s1) {
            double4_32a e = make_double4_32a(0.0, 0.0, 0.0, 0.0);
            for (int z = 0; z < ns; z++) {
                const double4_32a p = kp.Fpart[((size_t)z * kp.P + b) * (s1 - s0) + (s - s0)];
                e.x += p.x;
                e.y += p.y;
                e.z += p.z;
                e.w += p.w;
            }
            f.x += e.x;
            f.y += e.y;
            f.z += e.z;
            f.w += e.w;
        }
        const double q = kp.pos[gs].w;
        av[0] = q * f.w;
        const int k = s / N, w = s - k * N;
        double *out = kp.dRRt + ((size_t)b * kp.natoms + 3 * w + k) * 3;
        out[0] = kp.dR[3 * gs + 0] - q * f.x;
        out[1] = kp.dR[3 * gs + 1] - q * f.y;
        out[2] = kp.dR[3 * gs + 2] - q * f.z;
    }
    block_reduce_add<1, 128>(av, kp.acc + (size_t)b * NACC + ACC_UELEC2);
}

void launch_sites_spc(Engine &E) {
    dim3 g((E.kp.N + 31) / 32, E.kp.P);
    if (E.kp.model == 4)
        k_sites_spc<4><<<g, 128, 0, E.stream>>>(E.kp);
    else
        k_sites_spc<5><<<g, 128, 0, E.stream>>>(E.kp);
    ++E.nlaunch;
}

// with the charge field's deferred sums
void launch_finish_spc(Engine &E) {
    dim3 g((E.kp.S + 127) / 128, E.kp.P);
    KP kp = E.kp;
    const Engine::FieldFinish f = E.fin.back();
    E.fin.clear();
    kp.Fpart = f.part;
    k_finish_spc<<<g, 128, 0, E.stream>>>(kp, f.s0, f.s1, f.ns);
    ++E.nlaunch;
}

}  // namespace pimd
