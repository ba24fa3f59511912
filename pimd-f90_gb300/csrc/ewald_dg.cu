// ewald_dg.cu -- the FP64 engine's Ewald reciprocal sums as exact digit products on the tensor
// cores (ewald.f90:1-52, 56-119, 123-226, 230-291).
//
// What bounds the plain FP64 passes: this part issues about two FP64 operations per cycle and SM
// (64 cycles a warp instruction on its sub-partition), while FP16 matrix products run at 1017
// multiply-adds per cycle and SM (mma.sync m16n8k16, measured). With e^{ik.r} = exy(kx, ky) ez(kz)
// and ez(-j) = conj ez(j) both halves of the reciprocal sum are real matrix products:
//
//   structure factor  G[(c, j, cos|sin)][(run, Re|Im)] = sum_s Z X,   Z = w_c(s) (cos|sin)(j z_s),
//                     X = Re|Im exy(s, run);   S(kx, ky, +-j) from the four sums of (c, j, run)
//   field             T[s][(run, T0|T1, Re|Im)] = sum_j Q V,   Q = (cos|sin)(j z_s),
//                     V from the weights 4 pi Ak / V conj(S) of kz = +-j,
//                     E += Im(exy T0) (kx, ky) + Im(exy T1) z
//
// Precision. Each operand is a fixed-point number cut into signed base-2^b digits that FP16 holds
// exactly: 7 digits of 8 bits for the structure factor (2^-55 of the largest weight of the bead),
// 6 digits of 9 bits for the field (2^-53 of the largest weight of the run). Products of digits
// and their sums stay below 2^24, so the FP32 accumulators are exact: |digit| <= 2^(b-1), and one
// accumulator takes at most 7 products x 128 sites x 2^14, resp. 6 x 32 x 2^16. The digit products
// of equal weight are added in one accumulator and the accumulators are joined in integers. For the
// structure factor that is exact for any number of sites (64 bits and a word for what they shift
// out above 128 sites), and the sum is rounded to FP64 once; a T of the field is cut to 2^-56 of the
// run's largest weight (2^-53 with more than 32 harmonics). Left out are the products below the last
// digit (weight 2^-56, resp. 2^-54): the result is nearer to the exact sum than FP64 additions in any
// order, and it does not depend on the order of the sums.
//
// Measured (GB300, TTM3-F 512 x 32, |n| <= 12; FP64 passes -> this): structure factor of an iteration
// 866 -> 108 us (98 the product, half of it at the tensor rate, 10 forming Z), field and SOR update
// 1109 -> 102 us; of the charges 2170 -> 260 us, their field 3300 -> 380 us; the force pass
// 6800 -> 800 us. 128 molecules, one bead: 46 -> 22 us and 111 -> 17 us an iteration.
//
// Nearly no FP64 instruction is left: the phase tables are held in fixed point (2^62), the products
// exy T, ex ey and w z are 64-bit integer ones (six or three 32-bit multiply-adds), digits are cut
// and joined in integers, and a (site, run) takes two FP64 FMAs.
#include <algorithm>
#include <cstring>
#include <cuda_fp16.h>
#include <type_traits>
#include <vector>

#include "dd_real.cuh"
#include "dg_fixed.cuh"
#include "dipole_check.cuh"
#include "engine.h"
#include "umma.cuh"

namespace pimd {

enum { OP_Q = 0, OP_MU = 1, OP_DIP = 2 };
enum { F_Q = 0, F_D = 1, F_QD = 2 };

constexpr int DG_SB = 8, DG_SN = 7;      // structure factor: bits per digit, digits
constexpr int DG_FB = 9, DG_FN = 6;      // field
constexpr int DG_DRAIN = 8;              // k-steps (of 16 sites) per exact FP32 accumulation
constexpr int DG_SLOTS = 8;              // run slots per structure-factor block (2 tiles of 4)
constexpr int DG_XT = 1792, DG_ZT = 3584;  // bytes of one X (16 sites x 8 columns) and Z (16 x 16) tile
constexpr int DG_VT = 1536, DG_QT = 3072;  // the same for the field's V (8 columns) and Q (16 sites)
constexpr int DG_SW = 10;                // most warps of a structure-factor block
constexpr int DG_SMEM = 220 * 1024;      // dynamic shared memory of a block
constexpr int DG_FST = 4;                // tiles of the field's V ring
constexpr int DG_ST = 3;                 // k-steps of its operand ring

// ---- fixed point and digits ----------------------------------------------------------------
// the N digits of two fixed-point numbers, most significant first, as FP16 pairs (a low, b high).
// 0x6400 | u is the FP16 number 1024 + u, so a digit is one half2 subtraction from its bits.
template <int B, int N>
PIMD_D void dg_digits(long long a, long long b, uint32_t (&out)[N]) {
    constexpr int half = 1 << (B - 1);
    long long bias = 0;
#pragma unroll
    for (int i = 0; i < N - 1; i++) bias += (long long)half << (B * i);
    a += bias;
    b += bias;
#pragma unroll
    for (int s = 0; s < N; s++) {
        const int sh = B * (N - 1 - s);
        uint32_t x = (uint32_t)(a >> sh), y = (uint32_t)(b >> sh);
        if (s == 0) {
            x += 512u;  // the top digit is signed, |digit| <= half (+ rounding)
            y += 512u;
        } else {
            x &= (1u << B) - 1u;
            y &= (1u << B) - 1u;
        }
        const uint32_t w = x | (y << 16) | 0x64006400u;
        const uint32_t off = (s == 0) ? 0x66006600u : (B == 8 ? 0x64806480u : 0x65006500u);  // 1536; 1152; 1280
        __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&w), *reinterpret_cast<const __half2 *>(&off));
        out[s] = *reinterpret_cast<uint32_t *>(&h);
    }
}

PIMD_D void dg_mma(float (&d)[4], const uint4 &a, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
PIMD_D long long dg_i64(float d) { return (long long)__float2int_rn(d); }

// entry (cos, sin) of the fixed-point phase tables: (cos hi, lo, sin hi, lo)
PIMD_D int4 dg_tab(const KP &kp, const DgArgs &a, int b, int row, int s) { return a.tab[((size_t)b * kp.ntab + row) * kp.S + s]; }
// e^{i(kx x + ky y)} (ewald.f90:30-31: coskxky = cx cy - sx sy, sinkxky = sx cy + cx sy): one part
PIMD_D long long dg_exy(const KP &kp, const DgArgs &a, int b, int kx, int ky, int s, int part) {
    const int4 ex = dg_tab(kp, a, b, kx, s), ey = dg_tab(kp, a, b, kp.hmax + 1 + (ky < 0 ? -ky : ky), s);
    const long long p = dg_mul(part ? dg_im(ex) : dg_re(ex), dg_re(ey)), r = dg_mul(part ? dg_re(ex) : dg_im(ex), dg_im(ey));
    return ((part != 0) == (ky >= 0) ? p + r : p - r) << 2;
}

// ---- operands ------------------------------------------------------------------------------
// ewald.f90:403-437 ssincos: cos/sin(2 pi n x / L) for n = 0..nmax by the angle-addition recurrence from
// n = 1, each product and sum rounded separately like the reference, left in fixed point; and the
// beads whose tables are not finite. A thread takes one coordinate of a site: bound by the
// recurrence's chain of FP64 instructions, 15 us at 96 sites with all three in a thread and a
// conversion pass after it, 7.8 us so. The SPC models' sites are the input atoms (atoms, O H H).
__global__ void __launch_bounds__(128) k_dg_tab(KP kp, DgArgs a, const double *atoms) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y, d = blockIdx.z;
    if (s >= kp.S) return;
    double x;
    if (atoms) {
        const int k = s / kp.N, w = s - k * kp.N;
        x = atoms[((size_t)b * kp.natoms + 3 * w + k) * 3 + d];
    } else {
        x = reinterpret_cast<const double *>(kp.pos + (size_t)b * kp.S + s)[d];
    }
    const int nmax = d == 0 ? kp.hmax : d == 1 ? kp.kmax : kp.lmax;
    const int row = d == 0 ? 0 : d == 1 ? kp.hmax + 1 : kp.hmax + kp.kmax + 2;
    int4 *T = a.tab + ((size_t)b * kp.ntab + row) * kp.S + s;
    bool bad = false;
    auto put = [&](int n, double c, double sn) {
        bad |= dg_hi(c) >= 0x7ff00000 || dg_hi(sn) >= 0x7ff00000;
        const int2 u = dg_split(dg_fix(c, 62)), v = dg_split(dg_fix(sn, 62));
        T[(size_t)n * kp.S] = make_int4(u.x, u.y, v.x, v.y);
    };
    put(0, 1.0, 0.0);
    if (nmax >= 1) {
        const double arg = __dmul_rn(__dmul_rn(TWOPI, kp.boxi[d]), x);
        const double c1 = cos(arg), s1 = sin(arg);
        double c = c1, sn = s1;
        put(1, c1, s1);
        for (int n = 2; n <= nmax; n++) {
            const double cn = __dsub_rn(__dmul_rn(c, c1), __dmul_rn(sn, s1));
            const double snn = __dadd_rn(__dmul_rn(c, s1), __dmul_rn(sn, c1));
            c = cn;
            sn = snn;
            put(n, c, sn);
        }
    }
    if (bad) atomicOr(a.xbad + b, 1);
}

// X: one warp per tile of 4 run slots x 16 sites of a bead, every lane the fragment it holds in the
// product (column n = lane / 4: slot n / 2, part n & 1; sites 2q, 2q + 1, 2q + 8, 2q + 9 of
// q = lane & 3). Two tiles a step, so that a block's step is one copy. With cache also the values
// themselves, for the field's contraction.
__global__ void __launch_bounds__(128) k_dg_x(KP kp, DgArgs a, int s0, int nsites, int nks, int b0, int cache) {
    const int u = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31, xb = blockIdx.y, b = b0 + xb;
    if (u >= a.nx8 * nks) return;
    const int n8 = u / nks, ks = u - n8 * nks;
    const int n = lane >> 2, q = lane & 3, sl = 4 * n8 + (n >> 1), part = n & 1;
    long long v[4] = {0, 0, 0, 0};
    if (sl < a.nslot) {
        const int4 r = a.slot[sl];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int l = 16 * ks + 2 * q + (i & 1) + 8 * (i >> 1);
            if (l >= nsites) continue;
            const long long x = dg_exy(kp, a, b, r.x, r.y, s0 + l, part);
            if (cache) reinterpret_cast<int2 *>(a.exyc)[2 * (((size_t)b * a.nslot + sl) * nsites + l) + part] = dg_split(x);
            v[i] = (x + 64) >> 7;
        }
    }
    uint32_t d0[DG_SN], d1[DG_SN];
    dg_digits<DG_SB, DG_SN>(v[0], v[1], d0);
    dg_digits<DG_SB, DG_SN>(v[2], v[3], d1);
    char *o = reinterpret_cast<char *>(a.Xd) + ((((size_t)xb * (a.nx8 / 2) + n8 / 2) * nks + ks) * 2 + (n8 & 1)) * DG_XT;
#pragma unroll
    for (int p = 0; p < 3; p++)
        *reinterpret_cast<uint4 *>(o + 512 * p + 16 * lane) = make_uint4(d0[2 * p], d1[2 * p], d0[2 * p + 1], d1[2 * p + 1]);
    *reinterpret_cast<uint2 *>(o + 1536 + 8 * lane) = make_uint2(d0[6], d1[6]);
}

// ---- programmatic dependent launch ---------------------------------------------------------------
// In small systems an iteration's kernels are chained so: a kernel starts while the one before ends,
// does what does not depend on it, and waits (no effect on a launch without the attribute).
PIMD_D void dg_after_prior() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
PIMD_D void dg_next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Z: the weights of a bead's sites times the kz tables. Items (j, c), eight a tile, cos in the rows
// 0-7 and sin in 8-15. The scale is the bead's largest weight, which every block finds for itself.
// REAL (2 TTM2.1-F, 3 TTM3-F): the blocks from nzb on take the iteration's real-space dipole field,
// which needs the same dipoles (small systems: one launch less).
template <int NC, int REAL>
__global__ void __launch_bounds__(256) k_dg_z(KP kp, DgArgs a, int s0, int nsites, int nks, int nmt, int skipconv, int nzb) {
    const int b = blockIdx.y;
    dg_next_may_start();
    dg_after_prior();
    if (skipconv && bead_converged(kp, b)) return;
    if (REAL && (int)blockIdx.x >= nzb) {
        // (half a block's threads: FP64 instructions wait for their sub-partition, more blocks spread them)
        if (threadIdx.x < 128) dd_real_pairs<REAL ? REAL : 3>(kp, b, (blockIdx.x - nzb) * 128 + threadIdx.x, (gridDim.x - nzb) * 128);
        return;
    }
    __shared__ int smax;
    if (threadIdx.x == 0) smax = 0;
    __syncthreads();
    int m = 0;
    if (NC == 1) {
        for (int i = threadIdx.x; i < nsites; i += 256) m = max(m, dg_hi(kp.pos[(size_t)b * kp.S + s0 + i].w));
    } else {
        const double *mu = kp.dip + 3 * ((size_t)b * kp.S + s0);
        for (int i = threadIdx.x; i < 3 * nsites; i += 256) m = max(m, dg_hi(mu[i]));
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(&smax, m);
    __syncthreads();
    const int e = dg_exp(smax);
    if (blockIdx.x == 0 && threadIdx.x == 0) a.zexp[b] = e;
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int units = nmt * nks, step = nzb * 8;
    for (int u = blockIdx.x * 8 + (threadIdx.x >> 5); u < units; u += step) {
        const int mt = u / nks, ks = u - mt * nks;
        const int item = 8 * mt + g, j = NC == 1 ? item : item / NC, c = NC == 1 ? 0 : item - NC * j;
        long long vc[4] = {0, 0, 0, 0}, vs[4] = {0, 0, 0, 0};
        if (j < a.jn && e != DG_BAD) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int l = 16 * ks + 2 * q + (i & 1) + 8 * (i >> 1);
                if (l >= nsites) continue;
                const size_t gs = (size_t)b * kp.S + s0 + l;
                const int2 w = dg_split(dg_fix(NC == 1 ? kp.pos[gs].w : kp.dip[3 * gs + c], 61 - e));
                const int4 z = dg_tab(kp, a, b, kp.hmax + 1 + kp.kmax + 1 + j, s0 + l);
                vc[i] = (dg_mul(w, dg_re(z)) + 8) >> 4;  // 2^(59 - e) w z -> 2^(55 - e)
                vs[i] = (dg_mul(w, dg_im(z)) + 8) >> 4;
            }
        }
        uint32_t c0[DG_SN], c1[DG_SN], n0[DG_SN], n1[DG_SN];
        dg_digits<DG_SB, DG_SN>(vc[0], vc[1], c0);
        dg_digits<DG_SB, DG_SN>(vc[2], vc[3], c1);
        dg_digits<DG_SB, DG_SN>(vs[0], vs[1], n0);
        dg_digits<DG_SB, DG_SN>(vs[2], vs[3], n1);
        uint4 *o = reinterpret_cast<uint4 *>(reinterpret_cast<char *>(a.Zd) + (((size_t)b * nks + ks) * nmt + mt) * DG_ZT);
#pragma unroll
        for (int s = 0; s < DG_SN; s++) o[32 * s + lane] = make_uint4(c0[s], n0[s], c1[s], n1[s]);
    }
}

// Q: the kz tables of every site, 16 sites x 8 harmonics (cos, sin) a tile
__global__ void __launch_bounds__(128) k_dg_q(KP kp, DgArgs a) {
    const int u = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31, b = blockIdx.y;
    if (u >= a.nst * a.ksf) return;
    const int mt = u / a.ksf, ks = u - mt * a.ksf, g = lane >> 2, q = lane & 3;
    uint32_t d[4][DG_FN];
#pragma unroll
    for (int i = 0; i < 4; i++) {  // (site g, j), (site g + 8, j), (site g, j + 4), (site g + 8, j + 4)
        const int s = 16 * mt + g + 8 * (i & 1), j = 8 * ks + q + 4 * (i >> 1);
        int4 z = make_int4(0, 0, 0, 0);
        if (s < kp.S && j < a.jn) z = dg_tab(kp, a, b, kp.hmax + 1 + kp.kmax + 1 + j, s);
        dg_digits<DG_FB, DG_FN>((dg_join(dg_re(z)) + 256) >> 9, (dg_join(dg_im(z)) + 256) >> 9, d[i]);
    }
    uint4 *o = reinterpret_cast<uint4 *>(reinterpret_cast<char *>(a.Qd) + (((size_t)b * a.nst + mt) * a.ksf + ks) * DG_QT);
#pragma unroll
    for (int s = 0; s < DG_FN; s++) o[32 * s + lane] = make_uint4(d[0][s], d[1][s], d[2][s], d[3][s]);
}

// V of the nsl run slots from slot0, from their field weights w[slot][lmax + kz] in shared memory
// (zero where there is no k-vector): with P_j = W(+j) + W(-j), M_j = W(+j) - W(-j),
//   T0 = sum_j cos P + i sin M,  T1 = sum_j j (cos M + i sin P),  T2 = sum_j j^2 (cos P + i sin M).
// NT = 2: two slots a tile of 8 columns (T0, T1 each Re, Im); NT = 3: one slot (T0, T1, T2, -).
// Each slot's T has its own scale. pm: shared scratch of nsl jn x 4 doubles, vmax: nsl x NT ints.
template <int NT>
PIMD_D void dg_build_v(const KP &kp, const DgArgs &a, int b, int slot0, int nsl, const double2 *w, double *pm, int *vmax,
                       uint4 *V, int *vexp) {
    const int LZ = 2 * kp.lmax + 1, jn = a.jn;
    for (int i = threadIdx.x; i < nsl * NT; i += blockDim.x) vmax[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < nsl * jn; i += blockDim.x) {
        const int sl = i / jn, j = i - sl * jn;
        const double2 wp = w[sl * LZ + kp.lmax + j], wm = j ? w[sl * LZ + kp.lmax - j] : make_double2(0.0, 0.0);
        const double p[4] = {wp.x + wm.x, wp.y + wm.y, j ? wp.x - wm.x : 0.0, j ? wp.y - wm.y : 0.0};
        double big = 0.0;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            pm[4 * i + c] = p[c];
            const long long u = __double_as_longlong(p[c]) & 0x7fffffffffffffffLL;
            if (u > __double_as_longlong(big)) big = __longlong_as_double(u);
        }
        double f = 1.0;
#pragma unroll
        for (int t = 0; t < NT; t++) {
            atomicMax(&vmax[sl * NT + t], dg_hi(big * f));
            f *= (double)j;
        }
    }
    __syncthreads();
    const int tiles = NT == 2 ? nsl / 2 : nsl, nv8 = NT == 2 ? a.nv8 : a.nvd8;
    const int tile0 = NT == 2 ? slot0 / 2 : slot0;
    for (int i = threadIdx.x; i < tiles * a.ksf * 32; i += blockDim.x) {
        const int lane = i & 31, ks = (i >> 5) % a.ksf, tl = (i >> 5) / a.ksf;
        if (tile0 + tl >= nv8) continue;
        const int n = lane >> 2, q = lane & 3, part = n & 1;
        const int sl = NT == 2 ? 2 * tl + (n >> 2) : tl, T = NT == 2 ? (n >> 1) & 1 : n >> 1;
        const int e = T < NT ? dg_exp(vmax[sl * NT + T]) : DG_BAD;
        uint32_t d[2][DG_FN];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int j = 8 * ks + q + 4 * h;
            double cs = 0.0, sn = 0.0;
            if (j < jn && e != DG_BAD) {
                const double *p = pm + 4 * (sl * jn + j);
                // part Re: (P_re, -M_im) for T0, T2, (M_re, -P_im) for T1; Im: (P_im, M_re), (M_im, P_re)
                const int k0 = (T == 1) ? 2 : 0;
                const double f = T == 0 ? 1.0 : T == 1 ? (double)j : (double)j * j;
                cs = f * p[k0 + part];
                sn = part ? f * p[2 - k0] : -f * p[3 - k0];
            }
            dg_digits<DG_FB, DG_FN>(dg_fix(cs, 53 - e), dg_fix(sn, 53 - e), d[h]);
        }
        uint4 *o = V + (((size_t)b * nv8 + tile0 + tl) * a.ksf + ks) * (DG_VT / 16);
#pragma unroll
        for (int p = 0; p < 3; p++) o[32 * p + lane] = make_uint4(d[0][2 * p], d[1][2 * p], d[0][2 * p + 1], d[1][2 * p + 1]);
    }
    for (int i = threadIdx.x; i < nsl * NT; i += blockDim.x)
        vexp[((size_t)b * a.nslotp + slot0) * NT + i] = dg_exp(vmax[i]);
}

// ---- structure factor ------------------------------------------------------------------------
// Block: 8 run slots of a bead, one warp per tile of 8 items (all sites), so nothing is summed
// across blocks. The slots are sorted by kz extent, and tiles beyond the block's longest run are
// not formed. The operands come through a ring of DG_ST k-steps in shared memory, two bulk copies a
// step by one thread (loads straight to registers left the warps waiting on L2: 181 us an iteration
// at 512 x 32; copies of 16 bytes a thread cost more instructions than the products: 193 us). The
// epilogue forms S of the slots' k-vectors and (OP_Q, OP_MU) the field's V.
PIMD_D void dg_cp16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
PIMD_D void dg_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
PIMD_D void dg_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// size bytes (a multiple of 16, both addresses 16-byte aligned) counted on bar
PIMD_D void dg_bulk(void *dst, const void *src, uint32_t size, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(umma::smem_u32(dst)),
                 "l"(src), "r"(size), "r"(umma::smem_u32(bar))
                 : "memory");
}
PIMD_D void dg_expect(uint64_t *bar, uint32_t size) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(umma::smem_u32(bar)), "r"(size) : "memory");
}
constexpr long long DG_WAIT = 1LL << 28;  // cycles (about 0.13 s) after which a wait gives up

template <int OP>
__global__ void __launch_bounds__(32 * DG_SW) k_dg_sfac(KP kp, DgArgs a, int nks, int nmt, int ksum, int b0, int skipconv, int soff) {
    constexpr int NC = OP == OP_Q ? 1 : 3;
    const int xb = blockIdx.y, b = b0 + xb;
    dg_next_may_start();
    const int slot0 = blockIdx.x * DG_SLOTS, nsl = min(DG_SLOTS, a.nslot - slot0);
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, wp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int LZ = 2 * kp.lmax + 1, nitem = NC * a.jn;
    extern __shared__ __align__(128) double dsm[];
    char *ring = reinterpret_cast<char *>(dsm);          // [DG_ST][nw Z tiles, 2 X tiles]
    const int stage = nw * DG_ZT + 2 * DG_XT;
    // the epilogue's scratch: over the ring where the block makes one round of the tiles
    double2 *sb = reinterpret_cast<double2 *>(ring + soff);  // [8][nitem][2]: S_c(+j), S_c(-j)
    double2 *w = sb + (size_t)DG_SLOTS * nitem * 2;      // [8][LZ]
    double *pm = reinterpret_cast<double *>(w + (size_t)DG_SLOTS * LZ);  // [8][jn][4]
    __shared__ uint64_t full[DG_ST];
    __shared__ int vmax[DG_SLOTS * 2];
    const int4 first = a.slot[slot0];
    const int mts = min(nmt, (NC * (first.z + first.w) + 7) / 8);  // kzlo + nkz = longest |kz| + 1
    if (threadIdx.x < DG_ST) umma::mbar_init(&full[threadIdx.x], 1);
    for (int i = threadIdx.x; i < nsl * LZ; i += blockDim.x) {  // the epilogue's reads, to L2 / L1
        const int sl = i / LZ, kz = i - sl * LZ - kp.lmax;
        const int4 r = a.slot[slot0 + sl];
        if (kz >= r.z && kz < r.z + r.w)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(kp.kinfo + a.slotk[slot0 + sl] + kz - r.z));
    }
    dg_after_prior();
    if (skipconv && bead_converged(kp, b)) return;
    const int ze = a.zexp[b];
    const bool bad = ze == DG_BAD || a.xbad[b];
    const char *Zb = reinterpret_cast<const char *>(a.Zd) + (size_t)b * nmt * nks * DG_ZT;
    const char *X = reinterpret_cast<const char *>(a.Xd) + ((size_t)xb * (a.nx8 / 2) + blockIdx.x) * nks * (2 * DG_XT);
    __syncthreads();
    int it = 0, late = 0;  // steps taken (over all rounds), waits that gave up
    for (int m0 = 0; m0 < mts; m0 += nw) {
        const int nm = min(nw, mts - m0);
        auto load = [&](int ks, int at) {  // (thread 0) step ks into the ring place of step number at
            char *dst = ring + (at % DG_ST) * stage;
            uint64_t *bar = &full[at % DG_ST];
            dg_expect(bar, nm * DG_ZT + 2 * DG_XT);
            dg_bulk(dst, Zb + ((size_t)ks * nmt + m0) * DG_ZT, nm * DG_ZT, bar);
            dg_bulk(dst + nw * DG_ZT, X + (size_t)ks * (2 * DG_XT), 2 * DG_XT, bar);
        };
        if (m0 > 0) __syncthreads();
        if (threadIdx.x == 0)
            for (int k = 0; k < min(DG_ST - 1, nks); k++) load(k, it + k);
        const int mt = m0 + wp;
        // the sums so far in units of 2^(ze - 54 + ksum), and what is below (unsigned, units of 2^(ze - 62))
        long long t[2][4];
        unsigned low[2][4];
        float d[2][DG_SN][4];
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                t[n][i] = 0;
                low[n][i] = 0;
#pragma unroll
                for (int s = 0; s < DG_SN; s++) d[n][s][i] = 0.f;
            }
        for (int ks = 0; ks < nks; ks++, it++) {
            __syncthreads();  // every warp is done with the step before, whose place the next copy takes
            if (threadIdx.x == 0 && ks + DG_ST - 1 < nks) load(ks + DG_ST - 1, it + DG_ST - 1);
            late |= umma::mbar_wait(&full[it % DG_ST], (uint32_t)((it / DG_ST) & 1), DG_WAIT);
            if (wp >= nm) continue;
            const char *st = ring + (it % DG_ST) * stage;
            uint32_t B[2][DG_SN][2];
#pragma unroll
            for (int n = 0; n < 2; n++) {
                const char *x = st + nw * DG_ZT + n * DG_XT;
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    const uint4 v = reinterpret_cast<const uint4 *>(x + 512 * p)[lane];
                    B[n][2 * p][0] = v.x;
                    B[n][2 * p][1] = v.y;
                    B[n][2 * p + 1][0] = v.z;
                    B[n][2 * p + 1][1] = v.w;
                }
                const uint2 v = reinterpret_cast<const uint2 *>(x + 1536)[lane];
                B[n][6][0] = v.x;
                B[n][6][1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < DG_SN; i++) {
                const uint4 A = reinterpret_cast<const uint4 *>(st + wp * DG_ZT)[32 * i + lane];
#pragma unroll
                for (int j = 0; j < DG_SN - i; j++)
#pragma unroll
                    for (int n = 0; n < 2; n++) dg_mma(d[n][i + j], A, B[n][j][0], B[n][j][1]);
            }
            if (ks % DG_DRAIN == DG_DRAIN - 1 || ks == nks - 1) {
#pragma unroll
                for (int n = 0; n < 2; n++)
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        // sum_d D_d 2^(48 - 8 d) of z x 2^(62 - ze), exactly: the upper part to t, the rest to low
                        const long long hi = (dg_i64(d[n][0][i]) << 16) + (dg_i64(d[n][1][i]) << 8) + dg_i64(d[n][2][i]);
                        const long long lo = (dg_i64(d[n][3][i]) << 16) + (dg_i64(d[n][4][i]) << 8) + dg_i64(d[n][5][i]);
                        const int d6 = __float2int_rn(d[n][6][i]);
                        const long long v = (hi << 24) + lo + (d6 >> 8);
                        low[n][i] += (((unsigned)v & ((1u << ksum) - 1u)) << 8) + ((unsigned)d6 & 255u);
                        t[n][i] += (v >> ksum) + (low[n][i] >> (8 + ksum));
                        low[n][i] &= (1u << (8 + ksum)) - 1u;
#pragma unroll
                        for (int s = 0; s < DG_SN; s++) d[n][s][i] = 0.f;
                    }
            }
        }
        if (soff == 0) __syncthreads();
        if (wp >= nm) continue;
        // e^{ik.r} = exy (cos +- i sin): S(+j) = (cc - ss) + i (sc' + cs'), S(-j) with the signs of sin turned
        const int item = 8 * mt + g;
        if (item < nitem) {
            const int e = ze - 54 + ksum, wd = 8 + ksum;
#pragma unroll
            for (int n = 0; n < 2; n++) {
                double2 *o = sb + ((size_t)(4 * n + q) * nitem + item) * 2;
                const int l[4] = {(int)low[n][0], (int)low[n][1], (int)low[n][2], (int)low[n][3]};
                o[0] = make_double2(dg_double(t[n][0] - t[n][3], l[0] - l[3], wd, e), dg_double(t[n][1] + t[n][2], l[1] + l[2], wd, e));
                o[1] = make_double2(dg_double(t[n][0] + t[n][3], l[0] + l[3], wd, e), dg_double(t[n][1] - t[n][2], l[1] - l[2], wd, e));
            }
        }
    }
    if (late) atomicOr(kp.err, 8u);
    for (int i = threadIdx.x; i < DG_SLOTS * LZ; i += blockDim.x) w[i] = make_double2(0.0, 0.0);
    __syncthreads();
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    for (int i = threadIdx.x; i < nsl * LZ; i += blockDim.x) {
        const int sl = i / LZ, kz = i - sl * LZ - kp.lmax;
        const int4 r = a.slot[slot0 + sl];
        if (kz < r.z || kz >= r.z + r.w) continue;
        const int k = a.slotk[slot0 + sl] + kz - r.z, j = kz < 0 ? -kz : kz;
        const double2 *s = sb + ((size_t)sl * nitem + NC * j) * 2 + (kz < 0 ? 1 : 0);
        const size_t gk = (size_t)b * kp.nk + k;
        if (OP == OP_DIP) {
#pragma unroll
            for (int c = 0; c < 3; c++) kp.Sdip[3 * gk + c] = bad ? make_double2(nan, nan) : s[2 * c];
        } else {
            const double4_32a ki = kp.kinfo[k];
            double2 v = s[0];
            if (OP == OP_MU) {
                v.x = ki.x * s[0].x + ki.y * s[2].x + ki.z * s[4].x;
                v.y = ki.x * s[0].y + ki.y * s[2].y + ki.z * s[4].y;
            }
            if (bad) v = make_double2(nan, nan);
            if (OP == OP_MU) v = make_double2(-v.y, v.x);  // (rQm, iQm), ewald.f90:106-107
            (OP == OP_Q ? kp.Sq : kp.Sm)[gk] = v;
            w[sl * LZ + kp.lmax + kz] = make_double2(ki.w * v.x, -ki.w * v.y);  // 4 pi Ak / V conj(S)
        }
    }
    if (OP == OP_DIP) return;
    __syncthreads();
    dg_build_v<2>(kp, a, b, slot0, DG_SLOTS, w, pm, vmax, a.V, a.vexp);
}

// V of a dipole-force pass, from the structure factor A (and B added to it, if given); the second
// set (blockIdx.z = 1) from A2
__global__ void __launch_bounds__(128) k_dg_vqd(KP kp, DgArgs a, const double2 *A, const double2 *B, const double2 *A2) {
    const int b = blockIdx.y, slot0 = blockIdx.x * DG_SLOTS, nsl = min(DG_SLOTS, a.nslot - slot0), LZ = 2 * kp.lmax + 1;
    extern __shared__ __align__(128) double dsm[];
    double2 *w = reinterpret_cast<double2 *>(dsm);
    double *pm = reinterpret_cast<double *>(w + (size_t)DG_SLOTS * LZ);
    __shared__ int vmax[DG_SLOTS * 3];
    if (blockIdx.z) A = A2, B = nullptr;
    for (int i = threadIdx.x; i < DG_SLOTS * LZ; i += blockDim.x) {
        const int sl = i / LZ, kz = i - sl * LZ - kp.lmax;
        double2 v = make_double2(0.0, 0.0);
        if (sl < nsl) {
            const int4 r = a.slot[slot0 + sl];
            if (kz >= r.z && kz < r.z + r.w) {
                const int k = a.slotk[slot0 + sl] + kz - r.z;
                const double2 x = A[(size_t)b * kp.nk + k], y = B ? B[(size_t)b * kp.nk + k] : make_double2(0.0, 0.0);
                const double c = kp.kinfo[k].w;
                v = make_double2(c * (x.x + y.x), -c * (x.y + y.y));
            }
        }
        w[i] = v;
    }
    __syncthreads();
    const size_t set = blockIdx.z;
    dg_build_v<3>(kp, a, b, slot0, DG_SLOTS, w, pm, vmax, a.Vd + set * kp.P * a.nvd8 * a.ksf * (DG_VT / 16),
                  a.vdexp + set * kp.P * a.nslotp * 3);
}

// ---- field -----------------------------------------------------------------------------------
//   DGF_E : dipole field (E);  DGF_Q: charge field and potential;  DGF_QG: force on the charges
//   (-q E) and the dipoles' potential;  DGF_DG: force on the dipoles,
//   G_a = -sum_k k_a (k.mu) Re(e W) from T0, T1, T2
// Warp: 16 sites x the tiles of a slice, block: 4 warps on the same tiles, which come through a ring
// in shared memory (cp.async). Each slice's sums go to Fpart. sor (DGF_E): the last slice of a block
// of 64 sites to arrive adds the slices, in order, and runs the sites' SOR update and block end
// (dipole_check.cuh), so that an iteration needs no finishing launch; else k_field_finish adds them.
enum { DGF_E = 0, DGF_Q = 1, DGF_QG = 2, DGF_DG = 3 };
template <int MODE, int KS, bool XC>
__global__ void __launch_bounds__(128, 4) k_dg_field(KP kp, DgArgs a, int s0, int s1, int tshift, int sor,
                                                      const double *dip2) {
    const int b = blockIdx.y;
    dg_next_may_start();
    constexpr bool DG = MODE == DGF_DG;
    extern __shared__ uint4 fring[];  // [DG_FST][ksf][96]
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int mt = (s0 >> 4) + blockIdx.x * 4 + (threadIdx.x >> 5);
    const bool work = 16 * mt < s1;
    const int nv8 = DG ? a.nvd8 : a.nv8;
    // (DGF_DG with a second set: its slices are the upper half of the grid)
    const int half = DG && dip2 ? gridDim.z / 2 : gridDim.z, set = (int)blockIdx.z >= half, zs = blockIdx.z - set * half;
    const int n0 = (int)((long)zs * nv8 / half), n1 = (int)((long)(zs + 1) * nv8 / half);
    const uint4 *Q = reinterpret_cast<const uint4 *>(reinterpret_cast<const char *>(a.Qd) + ((size_t)b * a.nst + (work ? mt : 0)) * a.ksf * DG_QT) + lane;
    const int tile = a.ksf * (DG_VT / 16);
    const uint4 *V = (DG ? a.Vd : a.V) + ((size_t)set * kp.P + b) * nv8 * tile;
    const int *vexp = (DG ? a.vdexp : a.vexp) + ((size_t)set * kp.P + b) * a.nslotp * (DG ? 3 : 2);
    const double *dip = set ? dip2 : kp.dip;
    auto load = [&](int n8) {
        uint4 *dst = fring + (n8 % DG_FST) * tile;
        for (int i = threadIdx.x; i < tile; i += 128) dg_cp16(dst + i, V + (size_t)n8 * tile + i);
    };
    uint4 A[KS > 0 ? KS : 1][DG_FN];
    if (KS > 0) {
#pragma unroll
        for (int k = 0; k < KS; k++)
#pragma unroll
            for (int s = 0; s < DG_FN; s++) A[k][s] = Q[(size_t)k * (DG_QT / 16) + 32 * s];
    }
    const int site[2] = {16 * mt + g, 16 * mt + g + 8};
    const bool in[2] = {site[0] >= s0 && site[0] < s1, site[1] >= s0 && site[1] < s1};
    const int T = DG ? q : q & 1;
    const double kzu = TWOPI * kp.boxi[2];  // the k-vector's z component is kzu kz
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    double acc[2][3] = {{0, 0, 0}, {0, 0, 0}};
    // (slots past the last run and DG's fourth pair have zero digits: they add zeros)
    auto slot_of = [&](int n8) { return min(DG ? n8 : 2 * n8 + (q >> 1), a.nslot - 1); };
    const int4 *xc = XC ? a.exyc + (size_t)b * a.nslot * (s1 - s0) : nullptr;
    int4 xn[2];
    if (XC) {
#pragma unroll
        for (int h = 0; h < 2; h++) xn[h] = xc[(size_t)slot_of(n0) * (s1 - s0) + (in[h] ? site[h] - s0 : 0)];
    }
    dg_after_prior();
    if (MODE == DGF_E && bead_converged(kp, b)) {
        // (the block still counts towards the convergence test, once for its sites)
        const double zero[2] = {0.0, 0.0};
        if (sor && blockIdx.z == 0) dd_block_end<128>(kp, b, zero, false, gridDim.x * gridDim.y);
        return;
    }
#pragma unroll
    for (int k = 0; k < DG_FST - 1; k++) {
        if (n0 + k < n1) load(n0 + k);
        dg_commit();
    }
    for (int n8 = n0; n8 < n1; n8++) {
        const int slc = slot_of(n8);
        int4 x[2];
        if (XC) {  // exy of the next tile while this one is worked on
#pragma unroll
            for (int h = 0; h < 2; h++) {
                x[h] = xn[h];
                xn[h] = xc[(size_t)slot_of(min(n8 + 1, n1 - 1)) * (s1 - s0) + (in[h] ? site[h] - s0 : 0)];
            }
        }
        dg_wait<DG_FST - 2>();
        __syncthreads();
        if (n8 + DG_FST - 1 < n1) load(n8 + DG_FST - 1);
        dg_commit();
        if (!work) continue;
        long long t[4] = {0, 0, 0, 0};
        const uint4 *v = fring + (n8 % DG_FST) * tile + lane;
        auto step = [&](const uint4 (&Ak)[DG_FN], int ks, float (&d)[DG_FN][4]) {
            uint32_t B[DG_FN][2];
#pragma unroll
            for (int p = 0; p < 3; p++) {
                const uint4 u = v[ks * (DG_VT / 16) + 32 * p];
                B[2 * p][0] = u.x;
                B[2 * p][1] = u.y;
                B[2 * p + 1][0] = u.z;
                B[2 * p + 1][1] = u.w;
            }
#pragma unroll
            for (int i = 0; i < DG_FN; i++)
#pragma unroll
                for (int j = 0; j < DG_FN - i; j++) dg_mma(d[i + j], Ak[i], B[j][0], B[j][1]);
        };
        auto drain = [&](float (&d)[DG_FN][4]) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                // sum_d D_d 2^(40 - 9 d): T = t 2^(e - 56)
                const long long hi = (dg_i64(d[0][i]) << 18) + (dg_i64(d[1][i]) << 9) + dg_i64(d[2][i]);
                const long long lo = (dg_i64(d[3][i]) << 18) + (dg_i64(d[4][i]) << 9) + dg_i64(d[5][i]);
                t[i] += ((hi << 22) + (lo >> 5)) >> tshift;
            }
        };
        if (KS > 0) {
            float d[DG_FN][4];
#pragma unroll
            for (int s = 0; s < DG_FN; s++) d[s][0] = d[s][1] = d[s][2] = d[s][3] = 0.f;
#pragma unroll
            for (int k = 0; k < KS; k++) step(A[k], k, d);
            drain(d);
        } else {
            for (int k0 = 0; k0 < a.ksf; k0 += 2) {  // 16 harmonics per exact accumulation
                float d[DG_FN][4];
#pragma unroll
                for (int s = 0; s < DG_FN; s++) d[s][0] = d[s][1] = d[s][2] = d[s][3] = 0.f;
                for (int k = k0; k < min(a.ksf, k0 + 2); k++) {
                    uint4 Ak[DG_FN];
#pragma unroll
                    for (int s = 0; s < DG_FN; s++) Ak[s] = Q[(size_t)k * (DG_QT / 16) + 32 * s];
                    step(Ak, k, d);
                }
                drain(d);
            }
        }
        const int e = vexp[slc * (DG ? 3 : 2) + min(T, 2)];
        const double2 kv = a.slotkv[slc];
        double cf[3];
        if (DG) {
            cf[0] = T == 0 ? kv.x * kv.x : T == 1 ? kv.x * kzu : kzu * kzu;
            cf[1] = T == 0 ? kv.x * kv.y : T == 1 ? kv.y * kzu : 0.0;
            cf[2] = T == 0 ? kv.y * kv.y : 0.0;
        } else {
            cf[0] = T == 0 ? kv.x : kzu;
            cf[1] = T == 0 ? kv.y : 0.0;
            cf[2] = 1.0;
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (!XC) {
                const int4 r = a.slot[slc];
                const int sx = in[h] ? site[h] : s0;
                const int2 xr = dg_split(dg_exy(kp, a, b, r.x, r.y, sx, 0)), xi = dg_split(dg_exy(kp, a, b, r.x, r.y, sx, 1));
                x[h] = make_int4(xr.x, xr.y, xi.x, xi.y);
            }
            // Im, Re of exy T in fixed point (62 bits of exy: t 2^(e - 56) -> 2^(e - 54))
            const int2 re = dg_split(t[2 * h]), im = dg_split(t[2 * h + 1]);
            const int ez = (e == DG_BAD ? 0 : e) - 54 + tshift;
            double zi = 0.0, zr = 0.0;
            if (!DG) zi = dg_double(dg_mul2(dg_im(x[h]), re, dg_re(x[h]), im), ez);
            if (MODE != DGF_E) zr = dg_double(dg_mul2m(dg_re(x[h]), re, dg_im(x[h]), im), ez);
            if (e == DG_BAD) zi = zr = nan;
            acc[h][0] = fma(cf[0], DG ? zr : zi, acc[h][0]);
            acc[h][1] = fma(cf[1], DG ? zr : zi, acc[h][1]);
            if (MODE != DGF_E) acc[h][2] = fma(cf[2], zr, acc[h][2]);
        }
    }
    // lanes q of a row: T0 in q = 0, 2 and T1 in 1, 3 (DG: T0, T1, T2 in 0, 1, 2)
#pragma unroll
    for (int h = 0; h < 2; h++) {
        double o[4];
        const size_t gs = (size_t)b * kp.S + (in[h] ? site[h] : s0);
        if (DG) {
            const double r1x = __shfl_down_sync(0xffffffffu, acc[h][0], 1), r1y = __shfl_down_sync(0xffffffffu, acc[h][1], 1);
            const double r2 = __shfl_down_sync(0xffffffffu, acc[h][0], 2);
            if (q != 0 || !in[h]) continue;
            const double mu[3] = {dip[3 * gs], dip[3 * gs + 1], dip[3 * gs + 2]};
            o[0] = -(mu[0] * acc[h][0] + mu[1] * acc[h][1] + mu[2] * r1x);
            o[1] = -(mu[0] * acc[h][1] + mu[1] * acc[h][2] + mu[2] * r1y);
            o[2] = -(mu[0] * r1x + mu[1] * r1y + mu[2] * r2);
            o[3] = 0.0;
        } else {
#pragma unroll
            for (int c = 0; c < 3; c++) acc[h][c] += __shfl_xor_sync(0xffffffffu, acc[h][c], 2);
            o[2] = __shfl_down_sync(0xffffffffu, acc[h][0], 1);
            if (q != 0 || !in[h]) continue;
            const double f = MODE == DGF_QG ? -kp.pos[gs].w : 1.0;
            o[0] = f * acc[h][0];
            o[1] = f * acc[h][1];
            o[2] *= f;
            o[3] = MODE == DGF_E ? 0.0 : acc[h][2];
        }
        kp.Fpart[((size_t)blockIdx.z * kp.P + b) * (s1 - s0) + (site[h] - s0)] = make_double4_32a(o[0], o[1], o[2], o[3]);
    }
    if (MODE != DGF_E || !sor) return;
    __shared__ int last;
    __threadfence();  // this thread's sums are visible before the block counts
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned *c = a.fcnt + (size_t)b * gridDim.x + blockIdx.x;
        last = atomicAdd(c, 1u) == gridDim.z - 1;
        if (last) *c = 0u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // pot_ttm.f90:371-381 for the block's 64 sites, a component a thread
    const int iter = kp.dstep[1] + 1;
    double av[2] = {0.0, 0.0};
    for (int i = threadIdx.x; i < 192; i += 128) {
        const int s = 16 * ((s0 >> 4) + (int)blockIdx.x * 4) + i / 3, c = i % 3;
        if (s < s0 || s >= s1) continue;
        const size_t gc = 3 * ((size_t)b * kp.S + s) + c;
        const double mu = kp.dip[gc], efdr = kp.Efdr[gc];
        const double efq = reinterpret_cast<const double *>(kp.F + (size_t)b * kp.S + s)[c];
        const double pol = kp.polar_sor * kp.polar[s / kp.N + 1];
        const double *f = reinterpret_cast<const double *>(kp.Fpart + (size_t)b * (s1 - s0) + (s - s0)) + c;
        double e = 0.0;
        for (int z = 0; z < (int)gridDim.z; z++) e += __ldcg(f + (size_t)z * kp.P * (s1 - s0) * 4);
        const double efd = (efdr + e) + efq + kp.factor * mu;
        const double mn = (1.0 - kp.polar_sor) * mu + pol * efd;
        const double dd = (iter == 1) ? mn : mn - mu;
        av[0] += dd * dd;
        av[1] += mn * efq;
        kp.dip[gc] = mn;
        kp.Efdr[gc] = 0.0;
    }
    dd_block_end<128>(kp, b, av, true, gridDim.x * gridDim.y);
}

// ---- host --------------------------------------------------------------------------------------
static int ceil_div(int a, int b) { return (a + b - 1) / b; }

// a launch that may start while the one before it on the stream ends (dg_after_prior)
template <typename K, typename... A>
static void launch_pdl(bool on, K kernel, dim3 g, int nt, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t c = {};
    c.gridDim = g;
    c.blockDim = dim3(nt);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = on ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, args...);
}

// Small systems, whose iterations are bound by latency: one launch for Z and the real-space field, the
// three launches of an iteration chained (one bead of 128 molecules 1.40 -> 1.24 ms a call; not inside
// a graph, whose plain edges are faster: 101 x 7 0.52 ms a step, 0.59 with programmatic ones). By the
// pairs' work: at 100 thousand tensors the real-space
// field takes about 8 us, as long as Z; beyond, it runs on the second stream beside the structure
// factor (512 x 32: 850 thousand, 58 us).
bool dg_small(const Engine &E) {
    return E.precision != PIMD_PREC_MIXED && E.kp.model < 4 && E.dg_xall && E.pair_est * E.kp.P * E.kp.ndd <= 1.0e5;
}

// Buffers of the context's size. X holds as many beads as fit the limit (a pass over more beads
// forms X in several parts); the FP64 exy values are kept where X holds all dipole sites.
int dg_init(Engine &E) {
    KP &kp = E.kp;
    DgArgs &a = E.dg;
    a = DgArgs{};
    std::vector<int> order(kp.nrun);
    for (int r = 0; r < kp.nrun; r++) order[r] = r;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
        return E.h_runs[x].kzlo + E.h_runs[x].nkz > E.h_runs[y].kzlo + E.h_runs[y].nkz;
    });
    a.jn = kp.lmax + 1;
    a.nslot = kp.nrun;
    a.nslotp = ceil_div(kp.nrun, DG_SLOTS) * DG_SLOTS;
    a.nx8 = a.nslotp / 4;
    a.nv8 = a.nslotp / 2;
    a.nvd8 = a.nslotp;
    a.ksf = ceil_div(a.jn, 8);
    a.nst = ceil_div(kp.S, 16);
    std::vector<int4> slot(a.nslot);
    std::vector<int> slotk(a.nslot);
    std::vector<double2> slotkv(a.nslot);
    for (int i = 0; i < a.nslot; i++) {
        const KRun &r = E.h_runs[order[i]];
        slot[i] = make_int4(r.kx, r.ky, r.kzlo, r.nkz);
        slotk[i] = r.kbeg;
        slotkv[i] = make_double2(E.h_kvec[3 * r.kbeg], E.h_kvec[3 * r.kbeg + 1]);
    }
    const int nq = kp.S - kp.fq, nd = kp.ld - kp.fd;
    const size_t P = kp.P, kq = ceil_div(nq, 16), kd = ceil_div(nd, 16);
    const size_t per_step = (size_t)a.nx8 * DG_XT;  // X of one bead's 16 sites
    // dipole sites of every bead up to 8 GB, charged sites (formed once a force call) up to 1 GB
    const size_t fit_d = std::min(P * kd, ((size_t)8 << 30) / per_step), fit_q = std::min(P * kq, ((size_t)1 << 30) / per_step);
    a.xsteps = (int)std::max(std::max(kq, kd), std::max(fit_d, fit_q));
    E.dg_xall = (size_t)a.xsteps >= P * kd;
    // One allocation, cut on 256-byte boundaries (a first walk measures, a second places). Where the device has
    // no room for it, without the kept exy values and then with X of one bead at a time (formed in parts).
    const size_t zt = std::max((size_t)ceil_div(a.jn, 8) * kq, (size_t)ceil_div(3 * a.jn, 8) * kd);
    char *base = nullptr;
    size_t used = 0;
    auto cut = [&](auto &p, size_t bytes) {
        p = reinterpret_cast<std::decay_t<decltype(p)>>(base ? base + used : nullptr);
        used += (bytes + 255) & ~(size_t)255;
    };
    int4 *d_slot;
    int *d_slotk;
    double2 *d_slotkv;
    bool keep = nd && E.dg_xall;
    auto place = [&] {
        used = 0;
        cut(d_slot, sizeof(int4) * a.nslot);
        cut(d_slotk, sizeof(int) * a.nslot);
        cut(d_slotkv, sizeof(double2) * a.nslot);
        cut(a.zexp, P * sizeof(int));
        cut(a.xbad, P * sizeof(int));
        cut(a.fcnt, P * (size_t)(a.nst / 4 + 2) * sizeof(unsigned));
        cut(a.vexp, P * a.nslotp * 2 * sizeof(int));
        cut(a.vdexp, 2 * P * a.nslotp * 3 * sizeof(int));
        cut(a.Xd, (size_t)a.xsteps * per_step);
        cut(a.Zd, P * zt * DG_ZT);
        cut(a.Qd, P * a.nst * a.ksf * (size_t)DG_QT);
        cut(a.V, P * a.nv8 * a.ksf * (size_t)DG_VT);
        // (two sets where the differentiation form may run)
        if (nd) cut(a.Vd, (kp.model == 3 ? 2 : 1) * P * a.nvd8 * a.ksf * (size_t)DG_VT);
        if (keep) cut(a.exyc, P * a.nslot * (size_t)nd * sizeof(int4));
        cut(a.tab, P * (size_t)kp.ntab * kp.S * sizeof(int4));
    };
    place();
    for (int less = 0; cudaMalloc((void **)&base, used) != cudaSuccess; less++) {
        cudaGetLastError();
        base = nullptr;
        if (less == 2) return 1;
        keep = false;
        if (less == 1) {
            a.xsteps = (int)std::max(kq, kd);
            E.dg_xall = (size_t)a.xsteps >= P * kd;
        }
        place();
    }
    E.allocs.push_back(base);
    place();
    if (!keep) a.exyc = nullptr;
    // the host tables and the zeroed words after them in one copy
    const size_t head = reinterpret_cast<char *>(a.vexp) - base;
    std::vector<char> img(head, 0);
    std::memcpy(img.data(), slot.data(), sizeof(int4) * a.nslot);
    std::memcpy(img.data() + (reinterpret_cast<char *>(d_slotk) - base), slotk.data(), sizeof(int) * a.nslot);
    std::memcpy(img.data() + (reinterpret_cast<char *>(d_slotkv) - base), slotkv.data(), sizeof(double2) * a.nslot);
    cudaMemcpy(base, img.data(), head, cudaMemcpyHostToDevice);
    a.slot = d_slot;
    a.slotk = d_slotk;
    a.slotkv = d_slotkv;
    const int lim = DG_SMEM;
    // the field's V ring; beside a kernel's static words 48 KB (|kz| > 55) are more than a launch gets unasked
    if ((size_t)DG_FST * a.ksf * DG_VT + 1024 > 48 * 1024) {
        cudaFuncSetAttribute(k_dg_field<DGF_E, 0, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
        cudaFuncSetAttribute(k_dg_field<DGF_E, 0, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
        cudaFuncSetAttribute(k_dg_field<DGF_DG, 0, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
        cudaFuncSetAttribute(k_dg_field<DGF_DG, 0, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
        cudaFuncSetAttribute(k_dg_field<DGF_Q, 0, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
        cudaFuncSetAttribute(k_dg_field<DGF_QG, 0, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
    }
    cudaFuncSetAttribute(k_dg_sfac<OP_Q>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
    cudaFuncSetAttribute(k_dg_sfac<OP_MU>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
    cudaFuncSetAttribute(k_dg_sfac<OP_DIP>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
    cudaFuncSetAttribute(k_dg_vqd, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
    return 0;
}

static void launch_x(Engine &E, int s0, int nsites, int b0, int nb, bool cache) {
    const int nks = ceil_div(nsites, 16);
    k_dg_x<<<dim3(ceil_div(E.dg.nx8 * nks, 4), nb), 128, 0, E.stream>>>(E.kp, E.dg, s0, nsites, nks, b0, cache && E.dg.exyc ? 1 : 0);
    ++E.nlaunch;
}

// Site tables of a force call, and their digits for the field (Q, every site)
void launch_dg_tables(Engine &E) {
    E.dg_xdip = false;
    k_dg_tab<<<dim3(ceil_div(E.kp.S, 128), E.kp.P, 3), 128, 0, E.stream>>>(E.kp, E.dg, E.kp.model >= 4 ? E.kp.RRt : nullptr);
    ++E.nlaunch;
    k_dg_q<<<dim3(ceil_div(E.dg.nst * E.dg.ksf, 4), E.kp.P), 128, 0, E.stream>>>(E.kp, E.dg);
    ++E.nlaunch;
}

// X of the dipole sites, the same in every dipole iteration
void launch_dg_dipoles(Engine &E) {
    if (!E.dg_xall || E.kp.ld <= E.kp.fd) return;
    launch_x(E, E.kp.fd, E.kp.ld - E.kp.fd, 0, E.kp.P, true);
    E.dg_xdip = true;
}

template <int OP>
static void sfac(Engine &E, int s0, int nsites, int skipconv) {
    KP &kp = E.kp;
    const DgArgs &a = E.dg;
    constexpr int NC = OP == OP_Q ? 1 : 3;
    const int nks = ceil_div(nsites, 16), nmt = ceil_div(NC * a.jn, 8);
    // blocks of the Z kernel: enough to fill the chip, few enough that finding the bead's largest
    // weight (each block reads all of them) stays small
    const int upb = std::max(1, (int)((long)nmt * nks * kp.P / (8L * 4 * E.nsm)));
    const int nzb = ceil_div(ceil_div(nmt * nks, 8), upb);
    const bool have = OP != OP_Q && E.dg_xdip;
    const int nbmax = have ? kp.P : std::max(1, a.xsteps / nks);
    auto form_x = [&](int b0) {  // X of the beads from b0 that fit
        if (have) return;
        launch_x(E, s0, nsites, b0, std::min(nbmax, kp.P - b0), false);
        E.dg_xdip = false;
    };
    form_x(0);
    if (E.dg_after_x) cudaStreamWaitEvent(E.stream, E.dg_after_x, 0);
    const bool chain = OP == OP_MU && E.dg_chain;
    if (chain) {
        const int nrb = std::max(1, ceil_div((int)E.pair_est, 128));
        const dim3 g(nzb + nrb, kp.P);
        if (kp.model == 2)
            launch_pdl(E.dg_chain == 2 && !E.capturing, k_dg_z<NC, 2>, g, 256, 0, E.stream, kp, a, s0, nsites, nks, nmt, skipconv, nzb);
        else
            launch_pdl(E.dg_chain == 2 && !E.capturing, k_dg_z<NC, 3>, g, 256, 0, E.stream, kp, a, s0, nsites, nks, nmt, skipconv, nzb);
        E.dg_chain = 2;
    } else {
        k_dg_z<NC, 0><<<dim3(nzb, kp.P), 256, 0, E.stream>>>(kp, a, s0, nsites, nks, nmt, skipconv, nzb);
    }
    ++E.nlaunch;
    // keep the 64-bit sums of all sites below 2^61
    int ksum = 0;
    while (((long)nks * 16 >> ksum) > 128) ksum++;
    // one warp a tile, at least 4 for the epilogue; with large |kz| fewer, to leave room for the
    // epilogue's scratch, which shares the ring's place where one round of tiles is enough
    const size_t scratch = sizeof(double2) * ((size_t)DG_SLOTS * NC * a.jn * 2 + (size_t)DG_SLOTS * (2 * kp.lmax + 1) + (size_t)DG_SLOTS * a.jn * 2);
    int nw = std::min(std::max(nmt, 4), DG_SW);
    auto ring = [&](int n) { return (size_t)DG_ST * (n * DG_ZT + 2 * DG_XT); };
    while (nw > 1 && nw < nmt && scratch + ring(nw) > (size_t)DG_SMEM) nw--;
    const int soff = nw >= nmt ? 0 : (int)ring(nw);
    const size_t smem = soff ? scratch + ring(nw) : std::max(scratch, ring(nw));
    for (int b0 = 0; b0 < kp.P; b0 += nbmax) {
        const int nb = std::min(nbmax, kp.P - b0);
        if (b0) form_x(b0);
        launch_pdl(chain && !E.capturing, k_dg_sfac<OP>, dim3(a.nslotp / DG_SLOTS, nb), 32 * nw, smem, E.stream, kp, a, nks, nmt, ksum, b0, skipconv, soff);
        ++E.nlaunch;
    }
}

void launch_dg_sfac(Engine &E, int op, int s0, int nsites, int skipconv) {
    if (op == OP_Q)
        sfac<OP_Q>(E, s0, nsites, skipconv);
    else if (op == OP_MU)
        sfac<OP_MU>(E, s0, nsites, skipconv);
    else
        sfac<OP_DIP>(E, s0, nsites, skipconv);
}

template <int MODE>
static int field(Engine &E, int s0, int s1, int sor, const double *dip2 = nullptr) {
    const KP &kp = E.kp;
    const DgArgs &a = E.dg;
    const int mb = ceil_div(ceil_div(s1, 16) - s0 / 16, 4), tiles = MODE == DGF_DG ? a.nvd8 : a.nv8;
    // slices of the runs, at least four tiles each: the count whose waves of four blocks a SM do
    // the work soonest (512 x 32: 7 slices, 2.9 waves; 3 slices were 1.3 waves)
    const long base = (long)mb * kp.P, room = 4L * E.nsm;
    int ns = 1;
    double best = 1e300;
    const int most = dip2 ? E.max_slices / 2 : E.max_slices;
    for (int c = 1; c <= std::max(1, std::min(most, tiles / 4)); c++) {
        const double t = (double)((base * c + room - 1) / room) / c;
        if (t < best - 1e-12) best = t, ns = c;
    }
    const size_t smem = (size_t)DG_FST * a.ksf * DG_VT;
    if (dip2) ns *= 2;  // (the two sets' slices, ns of each)
    const dim3 g(mb, kp.P, ns);
    // |T| <= sqrt(2) lmax of the run's scale: keep t below 2^62
    const int tshift = a.jn > 32 ? 3 : 0;
    const bool xc = (MODE == DGF_E || MODE == DGF_DG) && E.dg_xdip && a.exyc && s0 == kp.fd && s1 == kp.ld;
    const bool chain = MODE == DGF_E && sor && E.dg_chain && !E.capturing;
#define PIMD_DGF(KS)                                                                                                      \
    if (xc)                                                                                                               \
        launch_pdl(chain, k_dg_field<MODE, KS, MODE == DGF_E || MODE == DGF_DG>, g, 128, smem, E.stream, kp, a, s0, s1, tshift, \
                   sor, dip2);                                                                                            \
    else                                                                                                                  \
        launch_pdl(chain, k_dg_field<MODE, KS, false>, g, 128, smem, E.stream, kp, a, s0, s1, tshift, sor, dip2)
    if (a.ksf == 1) {
        PIMD_DGF(1);
    } else if (a.ksf == 2) {
        PIMD_DGF(2);
    } else {
        PIMD_DGF(0);
    }
#undef PIMD_DGF
    ++E.nlaunch;
    return ns;
}

// One field pass; returns the number of slices whose sums are in Fpart. F_D: part 0 runs the SOR
// update and the convergence test too, part 1 leaves the sums; F_QD: part 0 the charge half of the
// force pass, 1 its dipole half.
int launch_dg_field(Engine &E, int mode, int s0, int s1, int part) {
    if (mode == F_D) return field<DGF_E>(E, s0, s1, part == 0);
    if (mode == F_Q) return field<DGF_Q>(E, s0, s1, 0);
    if (part == 0) return field<DGF_QG>(E, s0, s1, 0);
    return launch_dg_dforce(E, E.kp.Sq, E.kp.Sm, nullptr, nullptr);
}

// Force on the dipoles kp.dip in the field of the structure factor A (+ B), at the dipole sites, and
// with A2 that on the dipoles dip2 in the field of A2: the slices' sums in Fpart, their number.
int launch_dg_dforce(Engine &E, const double2 *A, const double2 *B, const double2 *A2, const double *dip2) {
    const DgArgs &a = E.dg;
    if (dip2 && E.max_slices < 2) return 0;
    const size_t smem = sizeof(double2) * ((size_t)DG_SLOTS * (2 * E.kp.lmax + 1) + (size_t)DG_SLOTS * a.jn * 2);
    k_dg_vqd<<<dim3(a.nslotp / DG_SLOTS, E.kp.P, A2 ? 2 : 1), 128, smem, E.stream>>>(E.kp, a, A, B, A2);
    ++E.nlaunch;
    return field<DGF_DG>(E, E.kp.fd, E.kp.ld, 0, dip2);
}

}  // namespace pimd
