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
// of equal weight are added in one accumulator, the accumulators are joined in 64-bit integers
// (exact), and the sum is rounded to FP64 once. Left out are the products below the last digit
// (weight 2^-56, resp. 2^-54): the result is nearer to the exact sum than FP64 additions in any
// order, and it does not depend on the order of the sums.
//
// Measured (GB300, TTM3-F 512 x 32, |n| <= 12, before -> now): structure factor of an iteration
// 866 -> 190 us, field 1109 -> 137 us; of the charges 2170 -> 500 us, their field 3300 -> 640 us; the
// force pass 6800 -> 1160 us. 128 molecules, one bead: 46 -> 25 us and 111 -> 22 us an iteration.
//
// The FP64 work left per (site, run) is the contraction with exy, four FMAs per T. Splitting into
// digits and joining them are integer instructions (32 per cycle for an FP64 one's two).
#include <algorithm>
#include <cuda_fp16.h>
#include <type_traits>
#include <vector>

#include "engine.h"

namespace pimd {

enum { OP_Q = 0, OP_MU = 1, OP_DIP = 2 };
enum { F_Q = 0, F_D = 1, F_QD = 2 };

constexpr int DG_SB = 8, DG_SN = 7;      // structure factor: bits per digit, digits
constexpr int DG_FB = 9, DG_FN = 6;      // field
constexpr int DG_DRAIN = 8;              // k-steps (of 16 sites) per exact FP32 accumulation
constexpr int DG_SLOTS = 8;              // run slots per structure-factor block (2 tiles of 4)
constexpr int DG_XT = 1792, DG_ZT = 3584;  // bytes of one X (16 sites x 8 columns) and Z (16 x 16) tile
constexpr int DG_VT = 1536, DG_QT = 3072;  // the same for the field's V (8 columns) and Q (16 sites)
constexpr int DG_BAD = 0x7fffffff;       // scale of an operand with a value that is not finite
constexpr int DG_SW = 10;                // most warps of a structure-factor block

// ---- fixed point and digits ----------------------------------------------------------------
// x 2^sh rounded to an integer, |x 2^sh| < 2^56, from the bits of x (an FP64 conversion costs the
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

PIMD_D double2 dg_tab(const KP &kp, int b, int row, int s) { return kp.tab[((size_t)b * kp.ntab + row) * kp.S + s]; }
PIMD_D double2 dg_exy(const KP &kp, int b, int kx, int ky, int s) {
    const double2 ex = dg_tab(kp, b, kx, s), ey0 = dg_tab(kp, b, kp.hmax + 1 + (ky < 0 ? -ky : ky), s);
    const double2 ey = make_double2(ey0.x, ky < 0 ? -ey0.y : ey0.y);
    // ewald.f90:30-31: coskxky = cx cy - sx sy, sinkxky = sx cy + cx sy
    return make_double2(ex.x * ey.x - ex.y * ey.y, ex.y * ey.x + ex.x * ey.y);
}

// ---- operands ------------------------------------------------------------------------------
// X: one warp per tile of 4 run slots x 16 sites of a bead, every lane the fragment it holds in the
// product (column n = lane / 4: slot n / 2, part n & 1; sites 2q, 2q + 1, 2q + 8, 2q + 9 of
// q = lane & 3). With exyc also the FP64 values, for the field's contraction.
__global__ void __launch_bounds__(128) k_dg_x(KP kp, DgArgs a, int s0, int nsites, int nks, int b0, int cache) {
    const int u = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31, xb = blockIdx.y, b = b0 + xb;
    if (u >= a.nx8 * nks) return;
    const int n8 = u / nks, ks = u - n8 * nks;
    const int n = lane >> 2, q = lane & 3, sl = 4 * n8 + (n >> 1), part = n & 1;
    long long v[4] = {0, 0, 0, 0};
    bool bad = false;
    if (sl < a.nslot) {
        const int4 r = a.slot[sl];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int l = 16 * ks + 2 * q + (i & 1) + 8 * (i >> 1);
            if (l >= nsites) continue;
            const double2 e = dg_exy(kp, b, r.x, r.y, s0 + l);
            const double x = part ? e.y : e.x;
            if (cache) reinterpret_cast<double *>(a.exyc)[2 * (((size_t)b * a.nslot + sl) * nsites + l) + part] = x;
            bad |= dg_hi(x) >= 0x7ff00000;
            v[i] = dg_fix(x, 55);
        }
    }
    if (bad) atomicOr(a.xbad + b, 1);
    uint32_t d0[DG_SN], d1[DG_SN];
    dg_digits<DG_SB, DG_SN>(v[0], v[1], d0);
    dg_digits<DG_SB, DG_SN>(v[2], v[3], d1);
    char *o = reinterpret_cast<char *>(a.Xd) + (((size_t)xb * a.nx8 + n8) * nks + ks) * DG_XT;
#pragma unroll
    for (int p = 0; p < 3; p++)
        *reinterpret_cast<uint4 *>(o + 512 * p + 16 * lane) = make_uint4(d0[2 * p], d1[2 * p], d0[2 * p + 1], d1[2 * p + 1]);
    *reinterpret_cast<uint2 *>(o + 1536 + 8 * lane) = make_uint2(d0[6], d1[6]);
}

// Z: the weights of a bead's sites times the kz tables. Items (j, c), eight a tile, cos in the rows
// 0-7 and sin in 8-15. The scale is the bead's largest weight, which every block finds for itself.
template <int NC>
__global__ void __launch_bounds__(256) k_dg_z(KP kp, DgArgs a, int s0, int nsites, int nks, int nmt, int skipconv) {
    const int b = blockIdx.y;
    if (skipconv && bead_converged(kp, b)) return;
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
    // a z table that is not finite has to show too: its first harmonic is looked at with the items
    const int e = dg_exp(smax);
    if (blockIdx.x == 0 && threadIdx.x == 0) a.zexp[b] = e;
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int units = nmt * nks, step = gridDim.x * 8;
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
                const double w = NC == 1 ? kp.pos[gs].w : kp.dip[3 * gs + c];
                const double2 z = dg_tab(kp, b, kp.hmax + 1 + kp.kmax + 1 + j, s0 + l);
                if (dg_hi(z.x) >= 0x7ff00000 || dg_hi(z.y) >= 0x7ff00000) atomicOr(a.xbad + b, 1);
                vc[i] = dg_fix(w * z.x, 55 - e);
                vs[i] = dg_fix(w * z.y, 55 - e);
            }
        }
        uint32_t c0[DG_SN], c1[DG_SN], n0[DG_SN], n1[DG_SN];
        dg_digits<DG_SB, DG_SN>(vc[0], vc[1], c0);
        dg_digits<DG_SB, DG_SN>(vc[2], vc[3], c1);
        dg_digits<DG_SB, DG_SN>(vs[0], vs[1], n0);
        dg_digits<DG_SB, DG_SN>(vs[2], vs[3], n1);
        uint4 *o = reinterpret_cast<uint4 *>(reinterpret_cast<char *>(a.Zd) + (((size_t)b * nmt + mt) * nks + ks) * DG_ZT);
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
        double2 z = make_double2(0.0, 0.0);
        if (s < kp.S && j < a.jn) z = dg_tab(kp, b, kp.hmax + 1 + kp.kmax + 1 + j, s);
        dg_digits<DG_FB, DG_FN>(dg_fix(z.x, 53), dg_fix(z.y, 53), d[i]);
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
// not formed. The epilogue forms S of the slots' k-vectors and (OP_Q, OP_MU) the field's V.
template <int OP>
__global__ void __launch_bounds__(32 * DG_SW) k_dg_sfac(KP kp, DgArgs a, int nks, int nmt, int ksum, int b0, int skipconv) {
    constexpr int NC = OP == OP_Q ? 1 : 3;
    const int xb = blockIdx.y, b = b0 + xb;
    if (skipconv && bead_converged(kp, b)) return;
    const int slot0 = blockIdx.x * DG_SLOTS, nsl = min(DG_SLOTS, a.nslot - slot0);
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int LZ = 2 * kp.lmax + 1, nitem = NC * a.jn;
    extern __shared__ double dsm[];
    double2 *sb = reinterpret_cast<double2 *>(dsm);      // [8][nitem][2]: S_c(+j), S_c(-j)
    double2 *w = sb + (size_t)DG_SLOTS * nitem * 2;      // [8][LZ]
    double *pm = reinterpret_cast<double *>(w + (size_t)DG_SLOTS * LZ);  // [8][jn][4]
    __shared__ int vmax[DG_SLOTS * 2];
    const int4 first = a.slot[slot0];
    const int mts = min(nmt, (NC * (first.z + first.w) + 7) / 8);  // kzlo + nkz = longest |kz| + 1
    const int ze = a.zexp[b];
    const bool bad = ze == DG_BAD || a.xbad[b];
    for (int mt = threadIdx.x >> 5; mt < mts; mt += blockDim.x >> 5) {
        long long t[2][4];
#pragma unroll
        for (int i = 0; i < 8; i++) t[i >> 2][i & 3] = 0;
        const uint4 *Z = reinterpret_cast<const uint4 *>(reinterpret_cast<const char *>(a.Zd) + ((size_t)b * nmt + mt) * nks * DG_ZT);
        const char *X = reinterpret_cast<const char *>(a.Xd) + ((size_t)xb * a.nx8 + 2 * blockIdx.x) * nks * DG_XT;
        for (int k0 = 0; k0 < nks; k0 += DG_DRAIN) {
            float d[2][DG_SN][4];
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int s = 0; s < DG_SN; s++)
#pragma unroll
                    for (int i = 0; i < 4; i++) d[n][s][i] = 0.f;
            const int k1 = min(nks, k0 + DG_DRAIN);
            for (int ks = k0; ks < k1; ks++) {
                uint4 A[DG_SN];
#pragma unroll
                for (int s = 0; s < DG_SN; s++) A[s] = __ldg(Z + (size_t)ks * (DG_ZT / 16) + 32 * s + lane);
                uint32_t B[2][DG_SN][2];
#pragma unroll
                for (int n = 0; n < 2; n++) {
                    const char *x = X + ((size_t)n * nks + ks) * DG_XT;
#pragma unroll
                    for (int p = 0; p < 3; p++) {
                        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(x + 512 * p) + lane);
                        B[n][2 * p][0] = v.x;
                        B[n][2 * p][1] = v.y;
                        B[n][2 * p + 1][0] = v.z;
                        B[n][2 * p + 1][1] = v.w;
                    }
                    const uint2 v = __ldg(reinterpret_cast<const uint2 *>(x + 1536) + lane);
                    B[n][6][0] = v.x;
                    B[n][6][1] = v.y;
                }
#pragma unroll
                for (int i = 0; i < DG_SN; i++)
#pragma unroll
                    for (int j = 0; j < DG_SN - i; j++)
#pragma unroll
                        for (int n = 0; n < 2; n++) dg_mma(d[n][i + j], A[i], B[n][j][0], B[n][j][1]);
            }
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    // sum_d D_d 2^(40 - 8 d): z x = t 2^(ze - 54)
                    const long long hi = (dg_i64(d[n][0][i]) << 16) + (dg_i64(d[n][1][i]) << 8) + dg_i64(d[n][2][i]);
                    const long long lo = (dg_i64(d[n][3][i]) << 16) + (dg_i64(d[n][4][i]) << 8) + dg_i64(d[n][5][i]);
                    t[n][i] += ((hi << 24) + lo + (dg_i64(d[n][6][i]) >> 8)) >> ksum;
                }
        }
        // e^{ik.r} = exy (cos +- i sin): S(+j) = (cc - ss) + i (sc' + cs'), S(-j) with the signs of sin turned
        const int item = 8 * mt + g;
        if (item < nitem) {
            const int e = ze - 54 + ksum;
#pragma unroll
            for (int n = 0; n < 2; n++) {
                double2 *o = sb + ((size_t)(4 * n + q) * nitem + item) * 2;
                o[0] = make_double2(dg_double(t[n][0] - t[n][3], e), dg_double(t[n][1] + t[n][2], e));
                o[1] = make_double2(dg_double(t[n][0] + t[n][3], e), dg_double(t[n][1] - t[n][2], e));
            }
        }
    }
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

// V of the force pass's dipole half, from the charge and dipole structure factors together
__global__ void __launch_bounds__(128) k_dg_vqd(KP kp, DgArgs a) {
    const int b = blockIdx.y, slot0 = blockIdx.x * DG_SLOTS, nsl = min(DG_SLOTS, a.nslot - slot0), LZ = 2 * kp.lmax + 1;
    extern __shared__ double dsm[];
    double2 *w = reinterpret_cast<double2 *>(dsm);
    double *pm = reinterpret_cast<double *>(w + (size_t)DG_SLOTS * LZ);
    __shared__ int vmax[DG_SLOTS * 3];
    for (int i = threadIdx.x; i < DG_SLOTS * LZ; i += blockDim.x) {
        const int sl = i / LZ, kz = i - sl * LZ - kp.lmax;
        double2 v = make_double2(0.0, 0.0);
        if (sl < nsl) {
            const int4 r = a.slot[slot0 + sl];
            if (kz >= r.z && kz < r.z + r.w) {
                const int k = a.slotk[slot0 + sl] + kz - r.z;
                const double2 sq = kp.Sq[(size_t)b * kp.nk + k], sm = kp.Sm[(size_t)b * kp.nk + k];
                const double c = kp.kinfo[k].w;
                v = make_double2(c * (sq.x + sm.x), -c * (sq.y + sm.y));
            }
        }
        w[i] = v;
    }
    __syncthreads();
    dg_build_v<3>(kp, a, b, slot0, DG_SLOTS, w, pm, vmax, a.Vd, a.vdexp);
}

// ---- field -----------------------------------------------------------------------------------
//   DGF_E : dipole field (E);  DGF_Q: charge field and potential;  DGF_QG: force on the charges
//   (-q E) and the dipoles' potential;  DGF_DG: force on the dipoles,
//   G_a = -sum_k k_a (k.mu) Re(e W) from T0, T1, T2
// Warp: 16 sites x the tiles of a slice, block: 4 warps on the same tiles (they share V in L1).
// Each slice's sums go to Fpart, which k_field_finish adds in order.
enum { DGF_E = 0, DGF_Q = 1, DGF_QG = 2, DGF_DG = 3 };
template <int MODE, int KS, bool XC>
__global__ void __launch_bounds__(128) k_dg_field(KP kp, DgArgs a, int s0, int s1, int tshift) {
    const int b = blockIdx.y;
    if (MODE == DGF_E && bead_converged(kp, b)) return;
    constexpr bool DG = MODE == DGF_DG;
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int mt = (s0 >> 4) + blockIdx.x * 4 + (threadIdx.x >> 5);
    if (16 * mt >= s1) return;
    const int nv8 = DG ? a.nvd8 : a.nv8;
    const int n0 = (int)((long)blockIdx.z * nv8 / gridDim.z), n1 = (int)((long)(blockIdx.z + 1) * nv8 / gridDim.z);
    const uint4 *Q = reinterpret_cast<const uint4 *>(reinterpret_cast<const char *>(a.Qd) + ((size_t)b * a.nst + mt) * a.ksf * DG_QT) + lane;
    const uint4 *V = (DG ? a.Vd : a.V) + ((size_t)b * nv8) * a.ksf * (DG_VT / 16) + lane;
    const int *vexp = (DG ? a.vdexp : a.vexp) + (size_t)b * a.nslotp * (DG ? 3 : 2);
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
    for (int n8 = n0; n8 < n1; n8++) {
        // (slots past the last run and DG's fourth pair have zero digits: they add zeros)
        const int slc = min(DG ? n8 : 2 * n8 + (q >> 1), a.nslot - 1);
        double2 x[2];
        if (XC) {
#pragma unroll
            for (int h = 0; h < 2; h++)
                x[h] = a.exyc[((size_t)b * a.nslot + slc) * (s1 - s0) + (in[h] ? site[h] - s0 : 0)];
        }
        long long t[4] = {0, 0, 0, 0};
        const uint4 *v = V + (size_t)n8 * a.ksf * (DG_VT / 16);
        auto step = [&](const uint4 (&Ak)[DG_FN], int ks, float (&d)[DG_FN][4]) {
            uint32_t B[DG_FN][2];
#pragma unroll
            for (int p = 0; p < 3; p++) {
                const uint4 u = __ldg(v + (size_t)ks * (DG_VT / 16) + 32 * p);
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
                x[h] = dg_exy(kp, b, r.x, r.y, in[h] ? site[h] : s0);
            }
            double re = dg_double(t[2 * h], e - 56 + tshift), im = dg_double(t[2 * h + 1], e - 56 + tshift);
            if (e == DG_BAD) re = im = nan;
            const double zi = x[h].y * re + x[h].x * im;
            if (MODE == DGF_E) {
                acc[h][0] = fma(cf[0], zi, acc[h][0]);
                acc[h][1] = fma(cf[1], zi, acc[h][1]);
            } else {
                const double zr = x[h].x * re - x[h].y * im;
                acc[h][0] = fma(cf[0], DG ? zr : zi, acc[h][0]);
                acc[h][1] = fma(cf[1], DG ? zr : zi, acc[h][1]);
                acc[h][2] = fma(cf[2], zr, acc[h][2]);
            }
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
            const double mu[3] = {kp.dip[3 * gs], kp.dip[3 * gs + 1], kp.dip[3 * gs + 2]};
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
}

// ---- host --------------------------------------------------------------------------------------
static int ceil_div(int a, int b) { return (a + b - 1) / b; }

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
    // one allocation, cut on 256-byte boundaries (the first walk measures, the second places)
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
    for (int pass = 0; pass < 2; pass++) {
        used = 0;
        cut(d_slot, sizeof(int4) * a.nslot);
        cut(d_slotk, sizeof(int) * a.nslot);
        cut(d_slotkv, sizeof(double2) * a.nslot);
        cut(a.zexp, P * sizeof(int));
        cut(a.xbad, P * sizeof(int));
        cut(a.vexp, P * a.nslotp * 2 * sizeof(int));
        cut(a.vdexp, P * a.nslotp * 3 * sizeof(int));
        cut(a.Xd, (size_t)a.xsteps * per_step);
        cut(a.Zd, P * zt * DG_ZT);
        cut(a.Qd, P * a.nst * a.ksf * (size_t)DG_QT);
        cut(a.V, P * a.nv8 * a.ksf * (size_t)DG_VT);
        if (nd) cut(a.Vd, P * a.nvd8 * a.ksf * (size_t)DG_VT);
        if (nd && E.dg_xall) cut(a.exyc, P * a.nslot * (size_t)nd * sizeof(double2));
        if (pass == 0) {
            if (cudaMalloc((void **)&base, used) != cudaSuccess) return 1;
            E.allocs.push_back(base);
        }
    }
    if (!nd || !E.dg_xall) a.exyc = nullptr;
    cudaMemcpy(d_slot, slot.data(), sizeof(int4) * a.nslot, cudaMemcpyHostToDevice);
    cudaMemcpy(d_slotk, slotk.data(), sizeof(int) * a.nslot, cudaMemcpyHostToDevice);
    cudaMemcpy(d_slotkv, slotkv.data(), sizeof(double2) * a.nslot, cudaMemcpyHostToDevice);
    a.slot = d_slot;
    a.slotk = d_slotk;
    a.slotkv = d_slotkv;
    cudaMemset(a.zexp, 0, P * sizeof(int));
    cudaMemset(a.xbad, 0, P * sizeof(int));
    const int lim = 200 * 1024;
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

// Site tables in digits (after the ssincos tables of a force call): the field's Q for every site
void launch_dg_tables(Engine &E) {
    E.dg_xdip = false;
    cudaMemsetAsync(E.dg.xbad, 0, sizeof(int) * E.kp.P, E.stream);
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
    const int upb = std::max(1, (int)((long)nmt * nks * kp.P / (8L * 608)));
    k_dg_z<NC><<<dim3(ceil_div(ceil_div(nmt * nks, 8), upb), kp.P), 256, 0, E.stream>>>(kp, a, s0, nsites, nks, nmt, skipconv);
    ++E.nlaunch;
    // keep the 64-bit sums of all sites below 2^61
    int ksum = 0;
    while (((long)nks * 16 >> ksum) > 128) ksum++;
    const int nw = std::min(std::max(nmt, 4), DG_SW);
    const size_t smem = sizeof(double2) * ((size_t)DG_SLOTS * NC * a.jn * 2 + (size_t)DG_SLOTS * (2 * kp.lmax + 1) + (size_t)DG_SLOTS * a.jn * 2);
    const bool have = OP != OP_Q && E.dg_xdip;
    const int nbmax = have ? kp.P : std::max(1, a.xsteps / nks);
    for (int b0 = 0; b0 < kp.P; b0 += nbmax) {
        const int nb = std::min(nbmax, kp.P - b0);
        if (!have) {
            launch_x(E, s0, nsites, b0, nb, false);
            E.dg_xdip = false;
        }
        k_dg_sfac<OP><<<dim3(a.nslotp / DG_SLOTS, nb), 32 * nw, smem, E.stream>>>(kp, a, nks, nmt, ksum, b0, skipconv);
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
static int field(Engine &E, int s0, int s1) {
    const KP &kp = E.kp;
    const DgArgs &a = E.dg;
    const int mb = ceil_div(ceil_div(s1, 16) - s0 / 16, 4), tiles = MODE == DGF_DG ? a.nvd8 : a.nv8;
    // slices of the runs: about four blocks a SM
    int ns = (int)((152L * 4 + (long)mb * kp.P - 1) / ((long)mb * kp.P));
    ns = std::max(1, std::min(ns, std::min(E.max_slices, tiles)));
    const dim3 g(mb, kp.P, ns);
    // |T| <= sqrt(2) lmax of the run's scale: keep t below 2^62
    const int tshift = a.jn > 32 ? 3 : 0;
    const bool xc = (MODE == DGF_E || MODE == DGF_DG) && E.dg_xdip && a.exyc && s0 == kp.fd && s1 == kp.ld;
#define PIMD_DGF(KS)                                                               \
    if (xc)                                                                        \
        k_dg_field<MODE, KS, true><<<g, 128, 0, E.stream>>>(kp, a, s0, s1, tshift); \
    else                                                                           \
        k_dg_field<MODE, KS, false><<<g, 128, 0, E.stream>>>(kp, a, s0, s1, tshift)
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

// The slices' sums of one field pass in Fpart; returns the number of slices. part: 0 the field or
// the charge half of the force pass, 1 its dipole half.
int launch_dg_field(Engine &E, int mode, int s0, int s1, int part) {
    if (mode == F_D) return field<DGF_E>(E, s0, s1);
    if (mode == F_Q) return field<DGF_Q>(E, s0, s1);
    if (part == 0) return field<DGF_QG>(E, s0, s1);
    const DgArgs &a = E.dg;
    const size_t smem = sizeof(double2) * ((size_t)DG_SLOTS * (2 * E.kp.lmax + 1) + (size_t)DG_SLOTS * a.jn * 2);
    k_dg_vqd<<<dim3(a.nslotp / DG_SLOTS, E.kp.P), 128, smem, E.stream>>>(E.kp, a);
    ++E.nlaunch;
    return field<DGF_DG>(E, s0, s1);
}

}  // namespace pimd
