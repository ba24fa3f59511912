// dipole_matrix.cu -- the induced-dipole iterations of small boxes (pot_ttm.f90:298-390) by the matrix of
// the whole dipole field. While the sites stay, the field of the dipoles at the dipole sites is
//   E_s = sum_t D(r_s - r_t) mu_t,   D_ab(d) = -sum_k (4 pi Ak / V) k_a k_b cos k.d + the pair's real-space tensor,
// so D is formed once a force call (k_dm_build, k_dm_real) and the iterations are products with it in
// shared memory (k_dm_solve): one launch for all of them, a cluster of CTAs a bead.
//
// The structure factor and the field of an iteration are two passes over sites x k-vectors that small
// boxes leave almost empty: an iteration took 30-40 us for one bead of 128 molecules and 28 us for
// 8 replicas of 32 to 256 molecules on the mixed engine, whatever its arithmetic. D costs
// pairs x k-vectors once instead.
//
// The sum over k of D folds to the octant kx, ky, kz >= 0 (the k-list is a sphere in an orthorhombic box):
// with c, s the cosine and sine of a component's phase, w = -(4 pi Ak / V) 2^(nonzero components) / 2,
//   A0 = sum_kz w cz, A1 = sum_kz w kz sz, A2 = sum_kz w kz^2 cz                       for each (kx, ky)
//   S0 = sum_ky cy A0, Syy = sum ky^2 cy A0, Sy = sum ky sy A0, S2 = sum cy A2, Sz = sum cy A1, Syz = sum ky sy A1
//   Dxx = sum_kx kx^2 cx S0, Dyy = sum cx Syy, Dzz = sum cx S2, Dxy = -sum kx sx Sy, Dxz = -sum kx sx Sz, Dyz = -sum cx Syz.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "dd_real.cuh"
#include "dg_fixed.cuh"
#include "mixed_pair.cuh"
#include "umma.cuh"

namespace pimd {

constexpr int DM_NP = 4;          // warps of a build block: parts of the kx, for the same 32 pairs
constexpr int DM_TR = 4, DM_TC = 8;  // rows and columns of its tile of sites
constexpr int DM_JMAX = 16;       // |k| components + 1 at most, in each direction
constexpr int DM_NT = 256;        // threads of a solver CTA

template <typename R>
struct DmTypes;
// FP64 engine: fixed point. An FP64 multiply-add takes a warp 64 cycles here, a 32 x 32 + 64 bit one 4
// or less, and three of those carry the product of two fixed-point numbers of 57 to 61 bits.
template <>
struct DmTypes<double> {
    using Z = int4;  // (cos, sin), each hi, lo of 2^56 x
    struct Y {       // 2^56 cy, 2^56 sy
        int2 c, s;
    };
};
template <>
struct DmTypes<float> {
    using Z = float2;
    struct Y {
        float c, q, s;
    };
};

// sums of products: hi hi, and hi lo + lo hi
struct DmAcc {
    long long h, m;
};
PIMD_D void dm_mac(DmAcc &a, int2 x, int2 y) {
    a.h += (long long)x.x * y.x;
    a.m += (long long)x.x * y.y;
    a.m += (long long)x.y * y.x;
}
PIMD_D void dm_mac_lo(DmAcc &a, int2 x, int2 y) {  // with the high half of lo lo
    dm_mac(a, x, y);
    a.m += __mulhi(x.y, y.y);
}

// ---- phases of a pair's difference ------------------------------------------------------------
// cos and sin of n (phi_s - phi_t) from the sites' tables, 2^60 x
PIMD_D void dm_diff(const int4 a, const int4 b, long long &c, long long &s) {
    c = dg_mul2(dg_re(a), dg_re(b), dg_im(a), dg_im(b));
    s = dg_mul2m(dg_im(a), dg_re(b), dg_re(a), dg_im(b));
}
PIMD_D void dm_z(const int4 a, const int4 b, int4 &z) {
    long long c, s;
    dm_diff(a, b, c, s);
    const int2 u = dg_split((c + 8) >> 4), v = dg_split((s + 8) >> 4);
    z = make_int4(u.x, u.y, v.x, v.y);
}
PIMD_D void dm_y(const int4 a, const int4 b, int, DmTypes<double>::Y &y) {
    int4 z;
    dm_z(a, b, z);
    y.c = make_int2(z.x, z.y);
    y.s = make_int2(z.z, z.w);
}
PIMD_D void dm_x(const int4 a, const int4 b, double2 &x) {
    long long c, s;
    dm_diff(a, b, c, s);
    x = make_double2(dg_double(c, -60), dg_double(s, -60));
}
PIMD_D void dm_diff(const float2 a, const float2 b, float &c, float &s) {
    c = a.x * b.x + a.y * b.y;
    s = a.y * b.x - a.x * b.y;
}
PIMD_D void dm_z(const float2 a, const float2 b, float2 &z) { dm_diff(a, b, z.x, z.y); }
PIMD_D void dm_y(const float2 a, const float2 b, int n, DmTypes<float>::Y &y) {
    float s;
    dm_diff(a, b, y.c, s);
    y.q = y.c * (float)(n * n);
    y.s = s * (float)n;
}
PIMD_D void dm_x(const float2 a, const float2 b, float2 &x) { dm_diff(a, b, x.x, x.y); }

// the host's tables in shared memory
struct DmW {
    const int4 *sh, *WA;
    const int2 *WB;
    const float4 *WF;
    const int *xe;
};

// ---- the six sums of one kx ------------------------------------------------------------------
// FP64 engine. Weights: WA (w kz^0, w kz^2), WB (w kz), each run's scaled to just below 2^58 and kz in
// units, so that A0, A1, A2 keep 58 bits of the run's own size; they are multiplied by 1, ky, ky^2
// (after a shift that makes room, the bits of the factor) and shifted to a common scale of the kx
// (a.sh, per run; a.xe, per kx). c is below 2^56 and there are at most 16 terms, so the sums of
// products stay below 2^63: hi hi 2^(24 + 26 + 4), hi lo 2^(31 + 26 + 4). The error of D is that of
// the same sums in FP64 (3e-17 of D(0) rms, |n| <= 9).
PIMD_D int2 dm_to(long long x, int sh) { return dg_split((x + ((1LL << sh) >> 1)) >> sh); }
template <int NQ>
PIMD_D void dm_kx(const DmW &a, int i0, int r0, int nky, const int2 (&zc)[4 * NQ], const int2 (&zs)[4 * NQ],
                  const DmTypes<double>::Y *yt, double (&S)[6]) {
    DmAcc t[6];
#pragma unroll
    for (int i = 0; i < 6; i++) t[i].h = t[i].m = 0;
    for (int y = 0; y < nky; y++) {
        const int r = r0 + y;
        const int4 sh = a.sh[r];  // groups of four kz, then the six shifts
        const int4 *WA = a.WA + (size_t)r * 4 * NQ;
        const int2 *WB = a.WB + (size_t)r * 4 * NQ;
        DmAcc u[3];
#pragma unroll
        for (int i = 0; i < 3; i++) u[i].h = u[i].m = 0;
#pragma unroll
        for (int q = 0; q < NQ; q++)
            if (q < sh.x) {
#pragma unroll
                for (int j = 4 * q; j < 4 * q + 4; j++) {
                    const int4 wa = WA[j];
                    const int2 wb = WB[j];
                    dm_mac(u[0], zc[j], make_int2(wa.x, wa.y));
                    dm_mac(u[1], zs[j], wb);
                    dm_mac(u[2], zc[j], make_int2(wa.z, wa.w));
                }
            }
        long long A[3];
#pragma unroll
        for (int i = 0; i < 3; i++) A[i] = (u[i].h << 4) + ((u[i].m + (1LL << 27)) >> 28);
        const int p1 = 32 - __clz(y), p2 = 32 - __clz(y * y);
        const DmTypes<double>::Y v = yt[y * 32];
        dm_mac_lo(t[0], v.c, dm_to(A[0], sh.y & 63));
        dm_mac_lo(t[1], v.c, dm_to((A[0] >> p2) * (y * y), (sh.y >> 8) & 63));
        dm_mac_lo(t[2], v.c, dm_to(A[2], (sh.y >> 16) & 63));
        dm_mac_lo(t[3], v.s, dm_to((A[0] >> p1) * y, sh.z & 63));
        dm_mac_lo(t[4], v.c, dm_to(A[1], (sh.z >> 8) & 63));
        dm_mac_lo(t[5], v.s, dm_to((A[1] >> p1) * y, (sh.z >> 16) & 63));
    }
#pragma unroll
    for (int i = 0; i < 6; i++) S[i] = dg_double((t[i].h << 8) + (t[i].m >> 24), a.xe[8 * i0 + i]);
}
// mixed engine
template <int NQ>
PIMD_D void dm_kx(const DmW &a, int, int r0, int nky, const float (&zc)[4 * NQ], const float (&zs)[4 * NQ],
                  const DmTypes<float>::Y *yt, float (&S)[6]) {
#pragma unroll
    for (int i = 0; i < 6; i++) S[i] = 0.f;
    for (int y = 0; y < nky; y++) {
        const int r = r0 + y, nq = a.sh[r].x;
        const float4 *W = a.WF + (size_t)r * NQ;
        float A0 = 0.f, A1 = 0.f, A2 = 0.f;
#pragma unroll
        for (int q = 0; q < NQ; q++)
            if (q < nq) {
                const float4 w4 = W[q];
                const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int j = 4 * q + i;
                    const float wc = w[i] * zc[j];
                    A0 += wc;
                    A2 = fmaf((float)(j * j), wc, A2);
                    A1 = fmaf(w[i], zs[j], A1);  // (zs holds kz sz)
                }
            }
        const DmTypes<float>::Y v = yt[y * 32];
        S[0] += v.c * A0;
        S[1] += v.q * A0;
        S[2] += v.c * A2;
        S[3] += v.s * A0;
        S[4] += v.c * A1;
        S[5] += v.s * A1;
    }
}

template <typename R>
PIMD_D typename DmTypes<R>::Z dm_tab(const KP &kp, const DgArgs &g, int b, int row, int s);
template <>
PIMD_D int4 dm_tab<double>(const KP &kp, const DgArgs &g, int b, int row, int s) {
    return g.tab[((size_t)b * kp.ntab + row) * kp.S + s];
}
template <>
PIMD_D float2 dm_tab<float>(const KP &kp, const DgArgs &, int b, int row, int s) {
    return kp.tabf[((size_t)b * kp.ntab + row) * kp.S + s];
}

// The reciprocal part of D. A block takes a tile of 4 x 8 sites (those with row <= column; the mirror
// image is stored with it): its four warps form the phases of the 32 pairs together, then each the
// kx of its part, and the parts' sums are added. FP64: bound by the issue of integer instructions (and
// with few beads by a warp's chain of them): 28 us for 128 sites, |n| <= 9 (43 with the weights read
// through L1 and the low products in the kz sums; about 22 us of FP64 pipe alone with FP64 sums).
template <typename R, int NQ>
__global__ void __launch_bounds__(32 * DM_NP) k_dm_build(KP kp, DgArgs g, DmArgs a) {
    using Z = typename DmTypes<R>::Z;
    using Y = typename DmTypes<R>::Y;
    using X = typename std::conditional<sizeof(R) == 8, double2, float2>::type;
    extern __shared__ __align__(16) unsigned char dm_sm[];
    Y *yt = reinterpret_cast<Y *>(dm_sm);                              // [kmax + 1][32]
    X *xt = reinterpret_cast<X *>(yt + (kp.kmax + 1) * 32);            // [hmax + 1][32]
    Z *zt = reinterpret_cast<Z *>(xt + (kp.hmax + 1) * 32);            // [4 NQ][32]
    R *part = reinterpret_cast<R *>(zt);                               // [DM_NP][6][32], after the phases
    // the host's tables (16-byte words, in the order of the allocation)
    const int4 *tb = reinterpret_cast<const int4 *>(dm_sm + a.phase);
    for (int i = threadIdx.x; i < a.words; i += 32 * DM_NP) reinterpret_cast<int4 *>(dm_sm + a.phase)[i] = a.tables[i];
    const int4 *kxs = tb;
    const DmW w{tb + a.at[0], tb + a.at[2], reinterpret_cast<const int2 *>(tb + a.at[3]), reinterpret_cast<const float4 *>(tb + a.at[2]),
                reinterpret_cast<const int *>(tb + a.at[1])};
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, b = blockIdx.y;
    // column tile J has 2 J + 2 row tiles
    int J = (int)((sqrtf(4.f * (float)blockIdx.x + 1.f) - 1.f) * 0.5f);
    while (J * (J + 1) > (int)blockIdx.x) J--;
    while ((J + 1) * (J + 2) <= (int)blockIdx.x) J++;
    const int s = DM_TR * ((int)blockIdx.x - J * (J + 1)) + (lane >> 3), t = DM_TC * J + (lane & 7);
    const int ss = kp.fd + min(s, a.nd - 1), st = kp.fd + min(t, a.nd - 1);
    for (int n = wp; n <= kp.kmax; n += DM_NP)
        dm_y(dm_tab<R>(kp, g, b, kp.hmax + 1 + n, ss), dm_tab<R>(kp, g, b, kp.hmax + 1 + n, st), n, yt[n * 32 + lane]);
    for (int n = wp; n <= kp.hmax; n += DM_NP) dm_x(dm_tab<R>(kp, g, b, n, ss), dm_tab<R>(kp, g, b, n, st), xt[n * 32 + lane]);
    const int rz = kp.hmax + kp.kmax + 2;
    for (int n = wp; n < 4 * NQ; n += DM_NP) {
        Z z{};
        if (n <= kp.lmax) dm_z(dm_tab<R>(kp, g, b, rz + n, ss), dm_tab<R>(kp, g, b, rz + n, st), z);
        zt[n * 32 + lane] = z;
    }
    __syncthreads();
    typename std::conditional<sizeof(R) == 8, int2, float>::type zc[4 * NQ], zs[4 * NQ];
#pragma unroll
    for (int j = 0; j < 4 * NQ; j++) {
        const Z z = zt[j * 32 + lane];
        if constexpr (sizeof(R) == 8) {
            zc[j] = make_int2(z.x, z.y);
            zs[j] = make_int2(z.z, z.w);
        } else {
            zc[j] = z.x;
            zs[j] = (float)j * z.y;
        }
    }
    R D[6] = {0, 0, 0, 0, 0, 0};  // xx yy zz xy xz yz
    for (int i = 0; i < a.nkx; i++) {
        const int4 kx = kxs[i];  // (kx, first run, ky of it, part)
        if (kx.w != wp) continue;
        R S[6];
        dm_kx<NQ>(w, i, kx.y, kx.z, zc, zs, yt + lane, S);
        const X x = xt[kx.x * 32 + lane];
        const R n = (R)kx.x, cn = x.x * n * n, sn = x.y * n;
        D[0] += cn * S[0];
        D[1] += x.x * S[1];
        D[2] += x.x * S[2];
        D[3] -= sn * S[3];
        D[4] -= sn * S[4];
        D[5] -= x.x * S[5];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 6; i++) part[(wp * 6 + i) * 32 + lane] = D[i];
    __syncthreads();
    const bool bad = sizeof(R) == 8 && g.xbad && g.xbad[b];
    if (s > t || t >= a.nd) return;
    R *M = reinterpret_cast<R *>(a.M) + (size_t)b * a.nd * 6 * a.ndp;
    const R f[6] = {(R)(a.gk[0] * a.gk[0]), (R)(a.gk[1] * a.gk[1]), (R)(a.gk[2] * a.gk[2]),
                    (R)(a.gk[0] * a.gk[1]), (R)(a.gk[0] * a.gk[2]), (R)(a.gk[1] * a.gk[2])};
    for (int i = wp; i < 6; i += DM_NP) {
        R v = 0;
#pragma unroll
        for (int p = 0; p < DM_NP; p++) v += part[(p * 6 + i) * 32 + lane];
        v *= f[i];
        if (bad) v = (R)__longlong_as_double(0x7ff8000000000000LL);
        M[((size_t)s * 6 + i) * a.ndp + t] = v;
        M[((size_t)t * 6 + i) * a.ndp + s] = v;
    }
}

// The real-space tensors of the charge phase's pair list (and TTM2.1-F's intramolecular ones) into D, a
// component of a pair a thread (a pair of sites is listed once)
template <int MODEL>
__global__ void __launch_bounds__(128) k_dm_real(KP kp, DmArgs a) {
    const int b = blockIdx.y, N = kp.N, np = kp.npair[b];
    double *M = reinterpret_cast<double *>(a.M) + (size_t)b * a.nd * 6 * a.ndp;
    constexpr int ND = MODEL == 2 ? 9 : 1;
    const int n = np * ND, all = n + (MODEL == 2 ? 3 * N : 0);
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < 6 * all; u += gridDim.x * blockDim.x) {
        const int i = u / 6, c = u - 6 * i;
        int s, t;
        const double *T;
        if (i < n) {
            const int p = i / ND, k = i - p * ND;
            const int2 ij = kp.pairs[(size_t)b * kp.cap + p];
            s = MODEL == 2 ? (k / 3) * N + ij.x : ij.x, t = MODEL == 2 ? (k % 3) * N + ij.y : ij.y;
            T = kp.Tdd + (((size_t)b * kp.cap + p) * ND + k) * 6;
        } else {
            const int w = (i - n) / 3, k = (i - n) - 3 * w;  // O H1, O H2, H1 H2
            s = (k == 2 ? N : 0) + w, t = (k == 0 ? N : 2 * N) + w;
            T = kp.Tself + ((size_t)b * N + w) * 18 + 6 * k;
        }
        double *x = M + ((size_t)s * 6 + c) * a.ndp + t, *y = M + ((size_t)t * 6 + c) * a.ndp + s;
        const double v = T[c], vx = *x, vy = *y;
        *x = vx + v;
        *y = vy + v;
    }
}

// The same on the mixed engine, from the full lists (a warp a molecule's row): the smeared tensor as the
// iterations' gather forms it (k_dd_real_m with OTF). TTM2.1-F's intramolecular tensors stay out of D: their field is
// taken in FP64 (k_dm_solve), as the gather takes it.
template <int MODEL>
__global__ void __launch_bounds__(128) k_dm_real_m(KP kp, DmArgs a) {
    using T = TT<MODEL>;
    const int lane = threadIdx.x & 31, i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, b = blockIdx.y, N = kp.N;
    if (i >= N) return;
    float *M = reinterpret_cast<float *>(a.M) + (size_t)b * a.nd * 6 * a.ndp;
    const int2 *fl = reinterpret_cast<const int2 *>(kp.fnbr) + (size_t)b * kp.fcap;
    const int ne = kp.fntot[b];  // offsets run past the stored length when the list overflowed
    const int e0 = min(kp.foff[(size_t)b * N + i], ne);
    const int e1 = (i + 1 < N) ? min(kp.foff[(size_t)b * N + i + 1], ne) : ne;
    auto add = [&](int s, int t, const float (&R)[3], float t1, float t3) {
        float *m = M + (size_t)s * 6 * a.ndp + t;
        const int p = a.ndp;
        m[0] += t3 * R[0] * R[0] - t1;
        m[p] += t3 * R[1] * R[1] - t1;
        m[2 * p] += t3 * R[2] * R[2] - t1;
        m[3 * p] += t3 * R[0] * R[1];
        m[4 * p] += t3 * R[0] * R[2];
        m[5 * p] += t3 * R[1] * R[2];
    };
    if (MODEL == 3) {
        const float4 *rec = kp.mrec + (size_t)b * N * 2;
        const float4 ri = rec[2 * i];
        for (int e = e0 + lane; e < e1; e += 32) {
            const int j = fl[e].y;
            const float4 rj = rec[2 * j];
            const float R[3] = {(float)(int)(__float_as_uint(ri.x) - __float_as_uint(rj.x)) * kp.boxq[0],
                                (float)(int)(__float_as_uint(ri.y) - __float_as_uint(rj.y)) * kp.boxq[1],
                                (float)(int)(__float_as_uint(ri.z) - __float_as_uint(rj.z)) * kp.boxq[2]};
            float t1, t2;
            smear2<float>(R[0] * R[0] + R[1] * R[1] + R[2] * R[2], kp.ptf.apol_dd[4][4], kp.ewf, &t1, &t2);
            add(i, j, R, t1, 3.f * t2);
        }
        return;
    }
    const float4 *pf = kp.posf + (size_t)b * kp.S;
    const uint4 *of = kp.ofix + (size_t)b * N;
    const uint4 oi = of[i];
    for (int e = e0 + lane; e < e1; e += 32) {
        const int j = fl[e].y;
        float Rf[3];
        oo_min_image(kp, oi, of[j], Rf);
#pragma unroll
        for (int isp = T::FDI; isp <= T::LDI; isp++)
#pragma unroll
            for (int jsp = T::FDI; jsp <= T::LDI; jsp++) {
                const float4 u = pf[(isp - 1) * N + i], c = pf[(jsp - 1) * N + j];
                const float R[3] = {wrapf(Rf[0] + u.x - c.x, kp.ptf.box[0], kp.ptf.boxi[0]),
                                    wrapf(Rf[1] + u.y - c.y, kp.ptf.box[1], kp.ptf.boxi[1]),
                                    wrapf(Rf[2] + u.z - c.z, kp.ptf.box[2], kp.ptf.boxi[2])};
                float t1, t2;
                smear2<float>(R[0] * R[0] + R[1] * R[1] + R[2] * R[2], kp.ptf.apol_dd[isp][jsp], kp.ewf, &t1, &t2);
                add((isp - 1) * N + i, (jsp - 1) * N + j, R, t1, 3.f * t2);
            }
    }
}

// ---- the iterations ------------------------------------------------------------------------------
template <typename T>
PIMD_D void dm_put(const T *local, uint32_t rank, T v) {
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(umma::smem_u32(local)), "r"(rank));
    if constexpr (sizeof(T) == 8)
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(v) : "memory");
    else
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(ra), "f"(v) : "memory");
}

// Sums over a warp's lanes of four 64-bit integers: lanes 8 i to 8 i + 7 get number i (as warp_sums)
PIMD_D long long dm_warp_sum4(long long (&x)[4]) {
    const int lane = threadIdx.x & 31;
    long long y[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const long long give = lane & 16 ? x[i] : x[i + 2], keep = lane & 16 ? x[i + 2] : x[i];
        y[i] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
    }
    const long long give = lane & 8 ? y[0] : y[1], keep = lane & 8 ? y[1] : y[0];
    long long z = keep + __shfl_xor_sync(0xffffffffu, give, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    return z;
}

// All of a bead's iterations (pot_ttm.f90:371-385) by a cluster: each CTA keeps the rows of D of its
// sites in shared memory, forms their field from every CTA's dipoles (a warp a row), updates their
// dipoles (a thread a component) and puts them and its sums into every CTA's shared memory; one
// cluster barrier an iteration (two sets of dipoles and sums in turn). The CTAs add the same sums
// in the same order, so they stop together.
// On the FP64 engine the products are in fixed point: the row's entries at 2^58 of its largest, the
// dipoles at 2^58 of the bead's largest (known with the sums), exact 64-bit sums of the high halves'
// products (2^(26 + 26) each, 552 at most) and of the mixed ones with the high half of lo lo (2^(26 + 31)
// each, 36 a lane), joined once a row: 2^-59 of the row's largest entry or of the largest dipole in a
// term, below the rounding of FP64 sums (rms error of an iteration's dipoles at 128 sites 7e-17 of them;
// 1.4e-16 with FP64 sums, 2.9e-16 with 2^52 and 2^54 and each lane's sum rounded, 1 % faster where many
// small beads share the SMs), and 20 cycles a product instead of 64. Four CTAs a SM (64 registers): 48 spill,
// and 80 leave small boxes of 64 beads in two waves (32 x 64 790 us a call, 715 so). Bound by latency: 3.9 us an
// iteration of 128 sites in a cluster of 16 CTAs (6.0 with FP64 products).
// intra: on the mixed engine TTM2.1-F's intramolecular field, the largest of a site's fields, is added by the updating
// threads from the FP64 tensors and dipoles (six products a component, the dipoles kept a second time in FP64: 60 x 8
// 409 us a call as with all in FP32, a step of 30 x 2 347 instead of 336).
constexpr int DM_MAXROWS = 42;  // of a CTA: their components are four warps' lanes
template <typename R, bool INTRA>
__global__ void __launch_bounds__(DM_NT, sizeof(R) == 8 ? 4 : 0) k_dm_solve(KP kp, DmArgs a, int rows) {
    constexpr bool D = sizeof(R) == 8;
    using W = typename std::conditional<D, int2, float>::type;  // an entry of D in shared memory
    extern __shared__ __align__(16) unsigned char dm_sm[];
    __shared__ int stop;
    const uint32_t rank = umma::cluster_rank(), C = umma::cluster_size();
    const int b = blockIdx.x / C, lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int nd = a.nd, ndp = a.ndp, s0 = (int)rank * rows, nr = max(0, min(rows, nd - s0)), nw = (3 * rows + 31) / 32;
    double *sums = reinterpret_cast<double *>(dm_sm);  // [2][32][2], of the CTAs' updating warps
    int *top = reinterpret_cast<int *>(sums + 128);    // [2][32] their largest dipole component's high word
    int *rexp = top + 64;                              // [44] the rows' scales
    double *ef = reinterpret_cast<double *>(rexp + 44);  // [3 rows + 1] field
    const bool intra = INTRA && kp.model == 2;          // (a branch: without it the FP64 chain is hoisted, 3 % slower)
    double *md = ef + 3 * rows + (rows & 1);            // [2][3][ndp] intra: the dipoles in FP64
    R *mu = reinterpret_cast<R *>(md + (intra ? 6 * ndp : 0));  // [2][3][ndp]
    W *mf = reinterpret_cast<W *>(mu + 6 * ndp);       // [3][ndp] FP64 engine: the dipoles in fixed point
    W *Ms = mf + (D ? 3 * ndp : 0);                    // [rows][6][ndp]
    const R *M = reinterpret_cast<const R *>(a.M) + ((size_t)b * nd + s0) * 6 * ndp;
    const double *dip = kp.dip + 3 * ((size_t)b * kp.S + kp.fd);
    int mt = 0;  // largest dipole component of the bead (high word)
    for (int i = threadIdx.x; i < 3 * nd; i += DM_NT) {
        mu[(i % 3) * ndp + i / 3] = (R)dip[i];
        if (intra) md[(i % 3) * ndp + i / 3] = dip[i];
    }
    if constexpr (D) {
        for (int i = lane; i < 3 * nd; i += 32) mt = max(mt, dg_hi(dip[i]));
        mt = __reduce_max_sync(0xffffffffu, mt);
        for (int r = wp; r < nr; r += DM_NT / 32) {
            int m = 0;
            for (int c = 0; c < 6; c++)
                for (int t = lane; t < nd; t += 32) m = max(m, dg_hi(M[((size_t)r * 6 + c) * ndp + t]));
            const int e = dg_exp(__reduce_max_sync(0xffffffffu, m));
            if (lane == 0) rexp[r] = e;
            for (int c = 0; c < 6; c++)
                for (int t = lane; t < nd; t += 32)
                    Ms[((size_t)r * 6 + c) * ndp + t] = e == DG_BAD ? make_int2(0, 0) : dg_split(dg_fix(M[((size_t)r * 6 + c) * ndp + t], 58 - e));
        }
    } else {
        for (int i = threadIdx.x; i < nr * 6 * ndp / 4; i += DM_NT) reinterpret_cast<uint4 *>(Ms)[i] = reinterpret_cast<const uint4 *>(M)[i];
    }
    // this thread's component of a site
    const int ur = threadIdx.x / 3, uc = threadIdx.x - 3 * ur;
    const bool upd = (int)threadIdx.x < 3 * nr;
    double mine = 0.0, before = 0.0, eq = 0.0, pol = 0.0;
    if (upd) {
        const int s = kp.fd + s0 + ur;
        mine = dip[3 * (s0 + ur) + uc];
        eq = reinterpret_cast<const double *>(kp.F + (size_t)b * kp.S + s)[uc];
        pol = kp.polar_sor * kp.polar[s / kp.N + 1];
    }
    // intra: the rows of the tensors to the molecule's other two sites (pairs O H1, O H2, H1 H2 of Tself)
    double tr[2][3] = {{0, 0, 0}, {0, 0, 0}};
    int other[2] = {0, 0};
    if (intra && upd) {
        const int k = (s0 + ur) / kp.N, w = s0 + ur - k * kp.N;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int j = i + (i >= k);
            const double *T = kp.Tself + ((size_t)b * kp.N + w) * 18 + 6 * (k + j - 1);
            other[i] = j * kp.N + w;
#pragma unroll
            for (int c = 0; c < 3; c++) tr[i][c] = T[c == uc ? c : c + uc + 2];  // xx yy zz xy xz yz
        }
    }
    umma::cluster_barrier();  // every CTA has started; this CTA's shared memory is filled
    int it = 0, em = D ? dg_exp(mt) : 0;
    while (true) {
        const R *cur = mu + (size_t)(it & 1) * 3 * ndp;
        it++;
        R *nxt = mu + (size_t)(it & 1) * 3 * ndp;
        if constexpr (D) {
            for (int i = threadIdx.x; i < 3 * ndp; i += DM_NT)
                mf[i] = i % ndp < nd && em != DG_BAD ? dg_split(dg_fix(cur[i], 58 - em)) : make_int2(0, 0);
            __syncthreads();
        }
        for (int r = wp; r < nr; r += DM_NT / 32) {
            const W *m = Ms + (size_t)r * 6 * ndp;
            if constexpr (D) {
                DmAcc e[3];
#pragma unroll
                for (int c = 0; c < 3; c++) e[c].h = e[c].m = 0;
                for (int t = lane; t < nd; t += 32) {
                    const int2 x = mf[t], y = mf[ndp + t], z = mf[2 * ndp + t];
                    const int2 xx = m[t], yy = m[ndp + t], zz = m[2 * ndp + t], xy = m[3 * ndp + t], xz = m[4 * ndp + t], yz = m[5 * ndp + t];
                    dm_mac_lo(e[0], xx, x);
                    dm_mac_lo(e[0], xy, y);
                    dm_mac_lo(e[0], xz, z);
                    dm_mac_lo(e[1], xy, x);
                    dm_mac_lo(e[1], yy, y);
                    dm_mac_lo(e[1], yz, z);
                    dm_mac_lo(e[2], xz, x);
                    dm_mac_lo(e[2], yz, y);
                    dm_mac_lo(e[2], zz, z);
                }
                long long h[4] = {e[0].h, e[1].h, e[2].h, 0}, m8[4] = {0, 0, 0, 0};
#pragma unroll
                for (int c = 0; c < 3; c++) m8[c] = (e[c].m + 128) >> 8;
                const long long H = dm_warp_sum4(h), L = dm_warp_sum4(m8);  // 2^-52 and 2^-76 of 2^(er + em)
                const int er = rexp[r], c = lane >> 3;
                if ((lane & 7) == 0 && c < 3)
                    ef[3 * r + c] = er == DG_BAD || em == DG_BAD ? __longlong_as_double(0x7ff8000000000000LL)
                                                                 : dg_double(H + (L >> 24), (int)(L & 0xffffff), 24, er + em - 52);
            } else {
                float e[3] = {0.f, 0.f, 0.f};
                for (int t = lane; t < nd; t += 32) {
                    const float x = cur[t], y = cur[ndp + t], z = cur[2 * ndp + t];
                    const float xx = m[t], yy = m[ndp + t], zz = m[2 * ndp + t], xy = m[3 * ndp + t], xz = m[4 * ndp + t], yz = m[5 * ndp + t];
                    e[0] += xx * x + xy * y + xz * z;
                    e[1] += xy * x + yy * y + yz * z;
                    e[2] += xz * x + yz * y + zz * z;
                }
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) e[c] += __shfl_xor_sync(0xffffffffu, e[c], o);
                if (lane < 3) ef[3 * r + lane] = (double)(lane == 0 ? e[0] : lane == 1 ? e[1] : e[2]);
            }
        }
        __syncthreads();
        if (wp < nw) {
            double av[2] = {0.0, 0.0};
            int m = 0;
            if (upd) {
                double f = ef[threadIdx.x];
                if (intra) {
                    const double *m = md + ((it - 1) & 1) * 3 * ndp;
#pragma unroll
                    for (int i = 0; i < 2; i++) f += tr[i][0] * m[other[i]] + tr[i][1] * m[ndp + other[i]] + tr[i][2] * m[2 * ndp + other[i]];
                }
                const double efd = f + eq + kp.factor * mine;
                const double mn = (1.0 - kp.polar_sor) * mine + pol * efd;
                const double d = it == 1 ? mn : mn - mine;
                av[0] = d * d;
                av[1] = mn * eq;
                before = mine;
                mine = mn;
                m = dg_hi(mn);
                const R v = (R)mn;
                for (uint32_t k = 0; k < C; k++) {
                    dm_put(nxt + uc * ndp + s0 + ur, k, v);
                    if (intra) dm_put(md + (it & 1) * 3 * ndp + uc * ndp + s0 + ur, k, mn);
                }
            }
            int at;
            const double v = warp_sums<2>(av, at);  // lanes 0 and 16
            if (D) m = __reduce_max_sync(0xffffffffu, m);
            const int slot = (it & 1) * 32 + (int)rank * nw + wp;
            for (uint32_t k = lane & 15; k < C; k += 16) {
                dm_put(sums + 2 * slot + at, k, v);
                if (D && at == 0) dm_put(reinterpret_cast<const float *>(top + slot), k, __int_as_float(m));
            }
        }
        umma::cluster_barrier();
        const int n = (int)C * nw;
        if (D) em = dg_exp(__reduce_max_sync(0xffffffffu, lane < n ? top[(it & 1) * 32 + lane] : 0));
        if (wp == DM_NT / 32 - 1) {
            double av[2] = {0.0, 0.0};
            if (lane < n) {
                av[0] = sums[2 * ((it & 1) * 32 + lane)];
                av[1] = sums[2 * ((it & 1) * 32 + lane) + 1];
            }
            int at;
            const double v = warp_sums<2>(av, at);
            const double dsq = __shfl_sync(0xffffffffu, v, 0);
            const bool conv = dsq < kp.dsq_eps;
            if (lane == 0) {
                stop = conv || it >= kp.polar_maxiter;
                if (stop && rank == 0) {
                    double *acc = kp.acc + (size_t)b * NACC;
                    acc[ACC_NITER] = (double)it;
                    acc[ACC_DELTADIP] = dsq;  // pimd_get_dipole_info takes stath sqrt of it
                    acc[ACC_CONV] = conv ? 1.0 : 2.0;
                    *kp.allconv = 1;
                }
            }
            if (lane == 16 && rank == 0) kp.acc[(size_t)b * NACC + ACC_UIND] = -0.5 * v;
        }
        __syncthreads();
        if (stop) break;
    }
    // the dipoles, and those of the iteration before, whose structure factor ewald_std_qd takes
    // (in Efdr, which is not otherwise used in such a call, and dipf_alt)
    if (upd) {
        const size_t at = 3 * ((size_t)b * kp.S + kp.fd + s0 + ur) + uc;
        kp.dip[at] = mine;
        kp.Efdr[at] = before;
        if (kp.dipf) {
            const size_t gs = (size_t)b * kp.S + kp.fd + s0 + ur;
            reinterpret_cast<float *>(kp.dipf + gs)[uc] = (float)mine;
            reinterpret_cast<float *>(kp.dipf_alt + gs)[uc] = (float)before;
            if (kp.mrec) reinterpret_cast<float *>(kp.mrec + 2 * ((size_t)b * kp.N + s0 + ur) + 1)[uc] = (float)mine;
        }
    }
}

// ---- host ----------------------------------------------------------------------------------------
static size_t solve_smem(const DmArgs &a, int rows, size_t rs, int model) {
    const size_t row = (size_t)a.ndp * rs, intra = rs == 4 && model == 2 ? 48 * (size_t)a.ndp : 0;
    return 128 * 8 + (64 + 44) * 4 + 8 * (size_t)(3 * rows + (rows & 1)) + intra + row * (6 + (rs == 8 ? 3 : 0) + 6 * (size_t)rows);
}

template <typename R, int NQ>
static void build(Engine &E) {
    const DmArgs &a = E.dm;
    const int nJ = (a.nd + DM_TC - 1) / DM_TC;
    const KP &kp = E.kp;
    const size_t smem = a.phase + 16 * (size_t)a.words;
    k_dm_build<R, NQ><<<dim3(nJ * (nJ + 1), kp.P), 32 * DM_NP, smem, E.stream>>>(kp, E.dg, a);
    ++E.nlaunch;
}
template <typename R>
static void build(Engine &E) {
    switch (E.dm.nqmax) {
        case 1: return build<R, 1>(E);
        case 2: return build<R, 2>(E);
        case 3: return build<R, 3>(E);
        default: return build<R, 4>(E);
    }
}

template <typename R>
static const void *build_kernel(int nq) {
    return nq == 1 ? (const void *)k_dm_build<R, 1> : nq == 2 ? (const void *)k_dm_build<R, 2> : nq == 3 ? (const void *)k_dm_build<R, 3> : (const void *)k_dm_build<R, 4>;
}
static void build_attr(const DmArgs &a, bool mixed) {
    cudaFuncSetAttribute(mixed ? build_kernel<float>(a.nqmax) : build_kernel<double>(a.nqmax), cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
}

// the reciprocal part, after the site tables
void launch_dm_build(Engine &E) {
    if (E.precision == PIMD_PREC_MIXED)
        build<float>(E);
    else
        build<double>(E);
}

// the real-space part, after the pair lists (and the charge phase on the FP64 engine), and the iterations
void launch_dm_solve(Engine &E) {
    const KP &kp = E.kp;
    const DmArgs &a = E.dm;
    const bool mixed = E.precision == PIMD_PREC_MIXED;
    if (mixed) {
        const dim3 g((kp.N + 3) / 4, kp.P);
        if (kp.model == 2)
            k_dm_real_m<2><<<g, 128, 0, E.stream>>>(kp, a);
        else
            k_dm_real_m<3><<<g, 128, 0, E.stream>>>(kp, a);
    } else {
        const dim3 g(std::max(1, std::min(4096, (int)(E.pair_est * kp.ndd * 6 / 128) + 1)), kp.P);
        if (kp.model == 2)
            k_dm_real<2><<<g, 128, 0, E.stream>>>(kp, a);
        else
            k_dm_real<3><<<g, 128, 0, E.stream>>>(kp, a);
    }
    // clusters of 16 where they all run at once
    const int C = a.c16 && kp.P <= a.c16 ? 16 : 8, rows = (a.nd + C - 1) / C;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(C * kp.P);
    c.blockDim = dim3(DM_NT);
    c.dynamicSmemBytes = solve_smem(a, rows, mixed ? 4 : 8, kp.model);
    c.stream = E.stream;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = C;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    if (!mixed)
        cudaLaunchKernelEx(&c, k_dm_solve<double, false>, kp, a, rows);
    else if (kp.model == 2)
        cudaLaunchKernelEx(&c, k_dm_solve<float, true>, kp, a, rows);
    else
        cudaLaunchKernelEx(&c, k_dm_solve<float, false>, kp, a, rows);
    E.nlaunch += 2;
}

// Where the matrix pays: forming it costs pairs x k-vectors once, the passes it replaces sites x
// k-vectors an iteration and about 30 us of latency. FP64 engine (a force call, passes -> matrix):
// 32 x 1 978 -> 453 us, 128 x 8 1599 -> 820, 128 x 64 4570 -> 3325, TTM2.1-F 60 x 16 (180 dipole sites)
// 2075 -> 1617: wherever its rows fit the shared memory of 8 CTAs (up to 184 sites). Mixed: 32 x 8
// 3474 -> 272 us, 128 x 32 1120 -> 400, 216 x 32 1024 -> 803, 270 x 8 1055 -> 487, 270 x 32 1209 -> 1129,
// but 270 x 64 1833 -> 1954: beyond 216 sites only up to 40 beads of 270 (the rows fit up to 272, TTM2.1-F
// 264). A k shell's tables are to fit 100 KB beside the phases, two blocks a SM: cubes up to |n| = 15, FP64 14.
static bool dm_wanted(const Engine &E) {
    const KP &kp = E.kp;
    if (kp.model >= 4 || std::max(kp.hmax, std::max(kp.kmax, kp.lmax)) >= DM_JMAX) return false;
    const double nd = kp.ld - kp.fd, mixed = E.precision == PIMD_PREC_MIXED;
    if (mixed && nd > 216 && nd * nd * kp.P > 40.0 * 270 * 270) return false;
    return nd * nd * kp.P * 6 * (mixed ? 4 : 8) <= 2147483648.0;  // (its memory: at most 2 GB)
}

void dm_init(Engine &E) {
    KP &kp = E.kp;
    DmArgs &a = E.dm;
    a = DmArgs{};
    const bool mixed = E.precision == PIMD_PREC_MIXED;
    if (!dm_wanted(E)) return;
    a.nd = kp.ld - kp.fd;
    a.ndp = (a.nd + 3) & ~3;
    const size_t rs = mixed ? 4 : 8;
    const size_t lim = (size_t)226 * 1024;  // (beside the static words)
    if ((a.nd + 7) / 8 > DM_MAXROWS || solve_smem(a, (a.nd + 7) / 8, rs, kp.model) > lim) return;
    for (int c = 0; c < 3; c++) a.gk[c] = TWOPI * kp.boxi[c];
    a.nqmax = (kp.lmax + 4) / 4;
    const int JM = 4 * a.nqmax;
    // the octant's runs, ordered by kx then ky (the list has every ky from 0 to a largest one, and
    // every kz from 0 likewise)
    std::vector<int4> kx;
    std::vector<int> nq, load;
    std::vector<double> w;
    int nrun = 0;
    for (const KRun &r : E.h_runs) {
        if (r.ky < 0) continue;
        if (kx.empty() || kx.back().x != r.kx) {
            kx.push_back(make_int4(r.kx, nrun, 0, 0));
            load.push_back(6);
        }
        if (r.ky != kx.back().z) return;
        kx.back().z++;
        w.resize((size_t)(nrun + 1) * JM, 0.0);
        int top = 0;
        for (int k = r.kbeg; k < r.kbeg + r.nkz; k++) {
            const int kz = r.kzlo + (k - r.kbeg);
            if (kz < 0) continue;
            const double m = (r.kx ? 2.0 : 1.0) * (r.ky ? 2.0 : 1.0) * (kz ? 2.0 : 1.0);
            w[(size_t)nrun * JM + kz] = -0.5 * m * FOURPI * E.h_Ak[k] / kp.volume;
            top = kz;
        }
        nq.push_back(top / 4 + 1);
        load.back() += 8 + 12 * nq.back();
        nrun++;
    }
    // the kx dealt to the parts, the largest first to the part with the least
    std::vector<int> order(kx.size());
    for (size_t i = 0; i < kx.size(); i++) order[i] = (int)i;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return load[x] > load[y]; });
    std::vector<int> sum(DM_NP, 0);
    std::vector<int4> list;
    for (int i : order) {
        kx[i].w = (int)(std::min_element(sum.begin(), sum.end()) - sum.begin());
        list.push_back(kx[i]);
        sum[kx[i].w] += load[i];
    }
    a.nkx = (int)list.size();
    // fixed-point weights, each run and power of kz at a scale of its own, and the shifts to the kx's
    std::vector<int4> WA(w.size()), sh(nrun, make_int4(0, 0, 0, 0));
    std::vector<int2> WB(w.size());
    std::vector<float> WF(w.size());
    std::vector<int> xe(8 * list.size(), 0);
    for (size_t i = 0; i < w.size(); i++) WF[i] = (float)w[i];
    auto bits = [](int x) {
        int n = 0;
        while (x >> n) n++;
        return n;
    };
    for (size_t i = 0; i < list.size(); i++) {
        constexpr int NONE = INT_MAX;  // a run of zeros
        std::vector<int> at(6 * list[i].z);  // exponents of the six sums' terms, of each run
        for (int y = 0; y < list[i].z; y++) {
            const size_t r0 = (size_t)(list[i].y + y) * JM;
            int e[3];
            for (int n = 0; n < 3; n++) {
                double big = 0.0;
                for (int j = 0; j < JM; j++) big = std::max(big, std::fabs(w[r0 + j] * std::pow((double)j, n)));
                int x = 0;
                std::frexp(big, &x);
                e[n] = big > 0.0 ? 58 - x : NONE;
                for (int j = 0; j < JM; j++) {
                    const long long v = big > 0.0 ? std::llrint(std::ldexp(w[r0 + j] * std::pow((double)j, n), e[n])) : 0;
                    const int lo = (int)(uint32_t)(unsigned long long)v, hi = (int)((v - lo) >> 32);
                    if (n == 0) WA[r0 + j].x = hi, WA[r0 + j].y = lo;
                    if (n == 1) WB[r0 + j] = make_int2(hi, lo);
                    if (n == 2) WA[r0 + j].z = hi, WA[r0 + j].w = lo;
                }
            }
            const int from[6] = {0, 0, 2, 0, 1, 1}, pre[6] = {0, bits(y * y), 0, bits(y), 0, bits(y)};
            for (int n = 0; n < 6; n++) at[6 * y + n] = e[from[n]] == NONE ? NONE : e[from[n]] - 4 - pre[n];
        }
        for (int n = 0; n < 6; n++) {
            int g = NONE;
            for (int y = 0; y < list[i].z; y++) g = std::min(g, at[6 * y + n]);
            xe[8 * i + n] = g == NONE ? 0 : g;  // of the terms; the sums' below
            for (int y = 0; y < list[i].z; y++) {
                const int v = at[6 * y + n] == NONE ? 0 : std::min(62, at[6 * y + n] - g);
                int4 &o = sh[list[i].y + y];
                o.x = nq[list[i].y + y];
                (n < 3 ? o.y : o.z) |= v << (8 * (n % 3));
            }
            xe[8 * i + n] = -xe[8 * i + n];  // (2^56 x 2^g / 2^56)
        }
    }
    // one allocation: the host tables, then D
    std::vector<char> img;
    auto put = [&](const void *p, size_t bytes) {
        const int at = (int)(img.size() / 16);
        img.resize((img.size() + bytes + 15) & ~(size_t)15, 0);
        std::memcpy(img.data() + 16 * (size_t)at, p, bytes);
        return at;
    };
    put(list.data(), sizeof(int4) * list.size());
    a.at[0] = put(sh.data(), sizeof(int4) * sh.size());
    a.at[1] = put(xe.data(), sizeof(int) * xe.size());
    a.at[2] = mixed ? put(WF.data(), sizeof(float) * WF.size()) : put(WA.data(), sizeof(int4) * WA.size());
    a.at[3] = mixed ? 0 : put(WB.data(), sizeof(int2) * WB.size());
    a.words = (int)(img.size() / 16);
    a.phase = (int)(32 * ((mixed ? sizeof(DmTypes<float>::Y) : sizeof(DmTypes<double>::Y)) * (kp.kmax + 1) + 2 * rs * (kp.hmax + 1) +
                          std::max(JM * 2 * (size_t)(mixed ? 4 : 8), DM_NP * 6 * rs)));
    const size_t bsm = a.phase + img.size();
    if (bsm > (size_t)100 * 1024) return;
    const size_t head = (img.size() + 255) & ~(size_t)255;
    char *base = nullptr;
    if (cudaMalloc((void **)&base, head + (size_t)kp.P * a.nd * 6 * a.ndp * rs) != cudaSuccess) {
        cudaGetLastError();  // (no room: the passes)
        return;
    }
    E.allocs.push_back(base);
    cudaMemcpy(base, img.data(), img.size(), cudaMemcpyHostToDevice);
    a.tables = reinterpret_cast<const int4 *>(base);
    a.M = base + head;
    build_attr(a, mixed);
    const void *solve = !mixed ? (const void *)k_dm_solve<double, false> : kp.model == 2 ? (const void *)k_dm_solve<float, true> : (const void *)k_dm_solve<float, false>;
    cudaFuncSetAttribute(solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lim);
    if (!mixed) {
        // clusters of 16 are beyond the portable size: as many as the device says it holds at once
        cudaFuncSetAttribute(solve, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3(16);
        c.blockDim = dim3(DM_NT);
        c.dynamicSmemBytes = solve_smem(a, (a.nd + 15) / 16, rs, kp.model);
        cudaLaunchAttribute at = {};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = 16;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        c.attrs = &at;
        c.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, solve, &c) == cudaSuccess) a.c16 = n;
        cudaGetLastError();
    }
}

}  // namespace pimd
