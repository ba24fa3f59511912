// Tensor-core (tcgen05) dipole structure factor of the mixed engine:
//   S(k) = sum_s (k.mu_s) e^{i k.r_s}            (ewald.f90:99-108, the per-iteration ewald_std_dd sum)
// over the dipole sites of every bead, as GEMMs on FP16 hi + lo splits (hi.hi + hi.lo + lo.hi,
// ~22-bit operands) with FP32 accumulators in TMEM, followed by the sum over site groups and the
// FP32 field weights (k_sreduce's job) in the same launch.
//
// Formulation. For a run (kx, ky) with kz in [kzlo, kzlo + nkz) and a site s, e^{ik.r} =
// exy(s) ez(s, kz) with exy = ex(kx) ey(ky) (ewald.f90:30-31), and
//   S(kz) = kx Gx(kz) + ky Gy(kz) + kz Gz(kz),   Gc(kz) = sum_s mu_c(s) exy(s) ez(s, kz).
// With ez(-j) = conj ez(j) = c_j - i s_j, every Gc(+-j) follows from four real sums over s,
//   Re.c = sum Re(exy) mu_c c_j,  Re.s,  Im.c,  Im.s :
//   Gc(+j) = (Re.c - Im.s) + i (Re.s + Im.c),   Gc(-j) = (Re.c + Im.s) + i (Im.c - Re.s),
// so one real GEMM per bead gives every k-vector:
//   D[(c, j, cos|sin)][(run, Re|Im)] = sum_s Z[(c, j, cos|sin)][s] X[(run, Re|Im)][s],
//   Z = mu_c(s) (c_j(s) | s_j(s)),   X = Re|Im exy(s, run).
// The M side holds 6 (max |kz| + 1) <= 128 rows, the N side two columns per run (<= 256 runs,
// two MMAs of N <= 256 per K step). A tcgen05 MMA costs about the same for any N <= 256 on this
// part (measured: ~200 cycles for M = 128 and 32 bytes of K), so the wide, run-dependent operand
// goes on N, and kind::f16 (16 sites per 32 bytes of K) halves the MMAs per site of kind::tf32;
// each K step of 16 sites is three MMAs per N half. Z is scaled by 2^6 (exact) so that small
// mu_c ez values keep normal FP16 lo parts; the epilogue takes the scale out.
//
// A CTA owns one bead, one group of <= 256 runs and one group of consecutive sites; the site
// groups of a (bead, run group) form a thread-block cluster. Warp roles:
//   * producer warp: per 32-site stage, TMA (cp.async.bulk.tensor.2d, two boxes of 16 sites x all
//     ntab table rows, 128-byte swizzle) plus a bulk copy of the 32 FP32 dipoles, completing on an
//     mbarrier; it then turns the dipoles into scaled, masked per-component rows and releases the
//     stage to the builders;
//   * 16 builder warps: per 16 sites build X (exy of every run, one item per thread) and Z
//     (mu_c ez, on the threads without an X item) in the canonical no-swizzle K-major layout,
//     split into FP16 hi + lo, into one of up to four buffers (X cached: 8 warps a step, in turn);
//   * MMA warp: one thread issues the MMAs into TMEM and commits to the buffer's mbarrier, which
//     releases the buffer to the builders.
// Only mbarriers connect the roles, so building, copying and MMAs overlap. The epilogue reads
// TMEM (tcgen05.ld) 64 runs at a time, combines each k-vector's 12 sums, and keeps the CTA's FP32
// partial S in shared memory; after a cluster barrier each CTA adds the partials of all CTAs of
// its cluster over a slice of the k-vectors (distributed shared memory, FP32, site groups in a
// fixed order) and writes Sm, the FP32 weights Wf and the field pass's operand V.
// Every mbarrier wait is bounded (~0.13 s); after a timeout a role stops, the CTA waits (bounded)
// for its copies and MMAs in flight, frees its TMEM, still meets its cluster barriers, and bit 8
// of the context's error word is set.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <tuple>
#include <utility>
#include <vector>

#include <cuda_fp16.h>

#include "dipole_check.cuh"
#include "engine.h"
#include "umma.cuh"

namespace pimd {

constexpr int TC_NB = 16;                 // builder warps
constexpr int TC_MMA_WARP = TC_NB;        // MMA-issuing warp (then the producer warp)
constexpr int TC_NT = (TC_NB + 2) * 32;   // 576 threads
constexpr int TC_SS = 32;                 // sites per table stage
constexpr int TC_KS = 16;                 // sites per MMA step (kind::f16: 32 bytes of K)
constexpr float TC_ZS = 64.f;             // power-of-two scale of Z (keeps small mu_c ez normal in FP16)
constexpr int TC_NABUF_MAX = 4;           // operand buffers (4: 708 -> 712 graph steps/s over 3)
constexpr int TC_NST = 4;                 // table stage buffers (a CTA's 128 sites at 512 x 32)
constexpr int TC_ZMAX = 4;                // Z items per builder thread (6 (|kz|max + 1) x 2 <= 256)
constexpr int TC_CLMAX = 8;               // site groups per cluster (portable cluster size)
constexpr int TC_MAXRUN = 256;            // runs per group: 512 TMEM columns
constexpr int TC_CH = 64;                 // runs per epilogue chunk
constexpr int TC_LD = 2 * TC_CH + 4;      // staging row pitch (floats)
constexpr float TP_WS = 512.f;            // power-of-two scale of the field passes' V (a row adds up to four weights)
constexpr long long TC_WAIT = 1LL << 28;  // cycles before a wait gives up (~0.13 s)

// structure-factor sums (values as in ewald.cu): charge q e, dipole (k.mu) e, dipole components mu_c e
enum { TC_OP_Q = 0, TC_OP_MU = 1, TC_OP_DIP = 2 };
// field passes (values as in ewald.cu): charge field and potential, dipole field + SOR update,
// and the two halves of the force pass ewald_std_qd: TF_QG the charge force and potential from
// the dipole structure factor, TF_DG the dipole force from the total (charge + dipole) one; TF_DE is TF_DG
// with the field itself, into Fx (the reverse sweep)
enum { TF_Q = 0, TF_D = 1, TF_QG = 2, TF_DG = 3, TF_DE = 4 };

// A run group: slots [p0, p0 + nr), MMA columns, the |kz| rows j0 .. j0 + jm - 1 of its Z
// operand (6 jm <= 128: |kz| above 20 goes to band groups, j0 = 21, of the same runs), k-vectors
// (local indices; those of a run outside the group's |kz| rows are entries with k = -1), and np pairs of runs
// (kx, +-ky) from vp0 of the pair table
struct TcGroup {
    int p0, nr, ncol, jm, nkl, kgoff, j0, np, vp0;
};

// k-vector of a local index and its 4 pi Ak / V
struct TcKW {
    int k;
    float w;
};

struct TcArgs {
    const int4 *slot;     // per slot: kx + 256 (ky + 128), local k offset, kzlo, nkz
    const float2 *skv;    // per slot: FP32 (k_x, k_y)
    const TcGroup *grp;
    const TcKW *kw;       // k-vector and weight of each local index
    const float *kzv;     // k_z by kz + lmax
    int sbase;            // first site of site group 0 (multiple of 32, <= s_lo)
    int s_lo, s_hi;       // dipole sites [s_lo, s_hi)
    int tsg;              // sites per group (multiple of 32)
    int ncolmax;          // max MMA columns over run groups
    int nabuf;            // operand buffers
    int skipconv;
    uint4 *xcache;        // X operand blocks of the dipole sites (null: no cache), see k_sfac_tc
    int xsub, xblock;     // 16-site blocks per bead and run group, bytes per block
    int xkeep;            // load the cached X blocks with the L2 evict-last policy
    int pdl;              // 1: launched as a programmatic dependent of the previous iteration's field pass; 2: of
                          // the band groups' launch, beside which it runs
    int tg0, ntg;         // the launch's first run group, all of them
    const int4 *vp;       // per pair: group slots of its +ky | -ky << 16 runs (0xffff: none), where its rows of
                          // the field pass's V begin and how far the lo rows are from there (16-byte words), |kz| rows
    uint4 *V;             // [P][vstride] that operand (null: none)
    int vstride;
};

// Shared-memory carve-up (bytes from a 1024-aligned base), used by the kernel and the launcher.
// A table stage holds two TMA boxes of 16 sites x ntab rows, each written with the 128-byte
// swizzle (16-byte chunk c of row r lands at chunk c ^ (r & 7), so loads of the same sites from
// different rows fall in different banks), followed by the stage's 32 dipoles (as copied, then
// as 3 rows of 2^6 mu_c with the sites outside the group zeroed). An operand
// buffer holds Z hi, Z lo (128 rows x 16 FP16 sites each) and X hi, X lo (ncolmax rows x 16 sites).
struct TcSmem {
    int boxb, mu, muz, stage, buf, xoff, bufstride, total;
    __host__ __device__ TcSmem(int ntab, int ncolmax, int nabuf) {
        boxb = ((ntab * 128 + 1023) / 1024) * 1024;
        mu = 2 * boxb;
        muz = mu + TC_SS * 16;
        stage = ((muz + 3 * TC_SS * 4 + 1023) / 1024) * 1024;
        buf = TC_NST * stage;
        xoff = 2 * 128 * 32;
        bufstride = xoff + 2 * ncolmax * 32;
        total = buf + nabuf * bufstride + 1024;  // + alignment slack of the dynamic base
    }
};

// 16-byte chunk holding sites (site, site + 1) of table row `row` in a swizzled stage
PIMD_D const float4 *tab_chunk(const unsigned char *stage, int boxb, int row, int site) {
    const int c = (site & 15) >> 1;
    return reinterpret_cast<const float4 *>(stage + (site >> 4) * boxb + row * 128 + ((c ^ (row & 7)) << 4));
}
PIMD_D float2 tab_elem(const unsigned char *stage, int boxb, int row, int site) {
    const float2 *p = reinterpret_cast<const float2 *>(tab_chunk(stage, boxb, row, site & ~1));
    return p[site & 1];
}

PIMD_D void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            umma::smem_u32(dst)),
        "l"((unsigned long long)map), "r"(x), "r"(y), "r"(umma::smem_u32(bar))
        : "memory");
}
// contiguous global -> shared copy (addresses 16-byte aligned, bytes a multiple of 16)
PIMD_D void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     umma::smem_u32(dst)),
                 "l"((unsigned long long)src), "r"(bytes), "r"(umma::smem_u32(bar))
                 : "memory");
}
// the same with an L2 eviction policy: evict-first (data read once per kernel that should not
// displace the working set of the other kernels) or, with keep, evict-last (data read again by
// every dipole iteration of the force call, kept in L2 across them)
PIMD_D void bulk_load_stream(void *dst, const void *src, uint32_t bytes, uint64_t *bar, bool keep = false) {
    uint64_t pol;
    if (keep)
        asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    else
        asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
                     umma::smem_u32(dst)),
                 "l"((unsigned long long)src), "r"(bytes), "r"(umma::smem_u32(bar)), "l"(pol)
                 : "memory");
}
// programmatic dependent launch: the next kernel of the stream may start (its CTAs wait with
// pdl_wait before they read what this grid writes); pdl_wait returns once the previous grid
// has completed and its writes are visible (a no-op without the launch attribute)
PIMD_D void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
PIMD_D void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
PIMD_D void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(umma::smem_u32(bar)), "r"(bytes) : "memory");
}
PIMD_D void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::smem_u32(bar)) : "memory");
}
PIMD_D void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
PIMD_D uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
PIMD_D float2 ld_cluster_f2(uint32_t local_addr, uint32_t rank) {
    uint32_t ra;
    float2 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(local_addr), "r"(rank));
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(ra));
    return v;
}
// Eight FP32 values as FP16 hi + lo (x = hi + lo to ~22 bits): two 16-byte rows of 8 halves
PIMD_D void split8_h(const float (&x)[8], uint4 &hi, uint4 &lo) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const __half2 hh = __floats2half2_rn(x[2 * i], x[2 * i + 1]);
        const float2 hf = __half22float2(hh);
        const __half2 ll = __floats2half2_rn(x[2 * i] - hf.x, x[2 * i + 1] - hf.y);
        h[i] = *reinterpret_cast<const uint32_t *>(&hh);
        l[i] = *reinterpret_cast<const uint32_t *>(&ll);
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}
// byte offset of the 16-byte chunk c (sites 8 c .. 8 c + 7) of row n in a K-major operand of 16
// FP16 sites (two core matrices along K)
PIMD_D int rowchunk(int n, int c) { return (((n >> 3) * 2 + c) << 7) + ((n & 7) << 4); }

// The rows of the field passes' V of a run pair at one |kz|: w the weights of (+ky, +kz), (+ky, -kz), (-ky, +kz),
// (-ky, -kz); out(row, cos part, sin part) for T0's Ts re, im, Td re, im, the same of T1, and with T2 of T2.
template <bool T2 = false, typename F>
PIMD_D void v_rows(const float2 (&w)[4], float kz, F &&out) {
    float2 p[2], m[2];  // W(+kz) + W(-kz) and W(+kz) - W(-kz), by the sign of ky
#pragma unroll
    for (int y = 0; y < 2; y++) {
        const float2 a = make_float2(TP_WS * w[2 * y].x, TP_WS * w[2 * y].y), c = make_float2(TP_WS * w[2 * y + 1].x, TP_WS * w[2 * y + 1].y);
        p[y] = make_float2(a.x + c.x, a.y + c.y);
        m[y] = make_float2(a.x - c.x, a.y - c.y);
    }
#pragma unroll
    for (int d = 0; d < 2; d++) {
        const float2 wp = d ? make_float2(p[0].x - p[1].x, p[0].y - p[1].y) : make_float2(p[0].x + p[1].x, p[0].y + p[1].y);
        const float2 wm = d ? make_float2(m[0].x - m[1].x, m[0].y - m[1].y) : make_float2(m[0].x + m[1].x, m[0].y + m[1].y);
        out(2 * d, wp.x, -wm.y);
        out(2 * d + 1, wp.y, wm.x);
        out(4 + 2 * d, kz * wm.x, -kz * wp.y);
        out(5 + 2 * d, kz * wm.y, kz * wp.x);
        if (T2) {
            const float k2 = kz * kz;
            out(8 + 2 * d, k2 * wp.x, -k2 * wm.y);
            out(9 + 2 * d, k2 * wp.y, k2 * wm.x);
        }
    }
}

// 64 registers a thread (a few bytes spill): one CTA of 576 threads then leaves 28 K registers
// of the SM to the real-space dipole field running beside it on the second stream (4 blocks
// instead of 1 at 95 registers); the graph step at 512 x 32 measured 677 -> 702 steps/s
// (72 registers: 695, 56: 697, 48: 680)
template <int OP>
__global__ void __maxnreg__(64) k_sfac_tc(const __grid_constant__ CUtensorMap tmap, KP kp, TcArgs a) {
    // Z components: q (charges) or mu_x, mu_y, mu_z; partial sums per k: S, or the three G_c
    constexpr int NCZ = (OP == TC_OP_Q) ? 1 : 3;
    constexpr int NPT = (OP == TC_OP_DIP) ? 3 : 1;
    const int grp = blockIdx.x, tg = a.tg0 + blockIdx.y, b = blockIdx.z;
    // a programmatic launch starts under the previous field pass: the convergence flags, the
    // dipoles and the weights are that grid's output
    if (a.pdl == 1) pdl_wait();
    // Beside the band groups' launch (pdl 2) the previous field pass is the launch before the one that this grid
    // depends on: it has ended, since every CTA of the band groups waited for it before it let this grid start, but
    // nothing has made its writes visible to this grid's cached loads. What it wrote and this kernel reads (the
    // convergence flag, the iteration count, the dipoles by bulk copies) is read from L2. The whole cluster (same
    // bead) leaves together.
    if (a.skipconv && bead_converged(kp, b)) {
        if (a.pdl == 2) pdl_wait();
        return;
    }
    const TcGroup G = a.grp[tg];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const TcSmem L(kp.ntab, a.ncolmax, a.nabuf);
    extern __shared__ __align__(1024) unsigned char sm_raw[];
    // the swizzle pattern follows shared-memory address bits 7-9: align the base to 1024 bytes
    unsigned char *sm = sm_raw + ((1024u - (umma::smem_u32(sm_raw) & 1023u)) & 1023u);
    __shared__ uint64_t tfull[TC_NST], mfull[TC_NST], tempty[TC_NST], afull[TC_NABUF_MAX], aempty[TC_NABUF_MAX];
    __shared__ uint64_t xfull[TC_NABUF_MAX];  // a cached X block has landed in the buffer
    __shared__ uint32_t tslot;
    __shared__ int4 sslot[TC_MAXRUN];
    __shared__ float2 sskv[TC_MAXRUN];
    __shared__ float skz[256];

    const int g0 = a.sbase + grp * a.tsg;
    const int g1 = min(a.s_hi, g0 + a.tsg);
    const int nstage = max(0, (g1 - g0 + TC_SS - 1) / TC_SS);
    const int nsub = nstage * (TC_SS / TC_KS);
    const int yrow = kp.hmax + 1;            // first ey row (ky = 0); ez rows follow the ky rows
    const int nab = a.nabuf, jm = G.jm, nr = G.nr;
    const int xlo = a.ncolmax * 32;          // X lo after X hi
    // X = exy(site, run) depends on the positions only, so the dipole structure factor of the
    // iterations builds it once per force call: the first iteration (no iteration done yet)
    // builds and stores it (xm 1), later ones load it by bulk copies (xm 2) and build only Z.
    // A block holds the X rows [0, 2 nr) rounded to 8-row groups, hi then lo, in the operand
    // layout; the cache is zeroed once, so the rows past 2 nr stay zero.
    const int xm = (OP == TC_OP_MU && a.xcache) ? (dd_done(kp) == 0 ? 1 : 2) : 0;
    const int xbytes = ((2 * nr + 7) / 8) * 256;
    uint4 *xc = xm ? a.xcache + ((size_t)(b * a.ntg + tg) * a.xsub + (g0 - a.sbase) / TC_KS) * (a.xblock / 16)
                   : nullptr;

    if (tid < nr) {
        sslot[tid] = a.slot[G.p0 + tid];
        sskv[tid] = a.skv[G.p0 + tid];
    }
    if (tid < 2 * kp.lmax + 1) skz[tid] = a.kzv[tid];
    if (warp == 0) umma::tmem_alloc(&tslot, 512);
    // table stage ts of this group: TMA boxes of the tables and a bulk copy of the dipoles
    const uint32_t box_tx = (uint32_t)(kp.ntab * 128);
    const float4 *const wsrc = (OP == TC_OP_Q) ? kp.posf : dipf_cur(kp);  // (offset, q) or (mu, 0)
    auto issue_stage = [&](int ts) {
        const int sfirst = g0 + ts * TC_SS, tb = ts % TC_NST;
        unsigned char *dst = sm + tb * L.stage;
        const int nmu = min(TC_SS, kp.S - sfirst);  // dipoles inside this bead's rows
        const uint32_t mub = (uint32_t)nmu * 16u;
        mbar_expect_tx(&tfull[tb], 2 * box_tx + mub);
        tma_load_2d(dst, &tmap, 2 * sfirst, b * kp.ntab, &tfull[tb]);
        tma_load_2d(dst + L.boxb, &tmap, 2 * sfirst + 32, b * kp.ntab, &tfull[tb]);
        bulk_load(dst + L.mu, wsrc + (size_t)b * kp.S + sfirst, mub, &tfull[tb]);
    };
    if (tid == 0) {
        for (int i = 0; i < TC_NST; i++) {
            umma::mbar_init(&tfull[i], 1);
            umma::mbar_init(&mfull[i], 1);
            umma::mbar_init(&tempty[i], TC_NB);
        }
        for (int i = 0; i < nab; i++) {
            umma::mbar_init(&afull[i], xm == 2 ? TC_NB / 2 : TC_NB);
            umma::mbar_init(&aempty[i], 1);
            umma::mbar_init(&xfull[i], 1);
        }
        // the first stages go out now, under the rest of the set-up
        for (int ts = 0; ts < min(nstage, TC_NST); ts++) issue_stage(ts);
    }
    {   // padding stays zero in every buffer (hi and lo): Z rows >= 6 jm, X rows >= 2 nr
        const int zp = 128 - 2 * NCZ * jm, xp = G.ncol - 2 * nr;
        for (int i = tid; i < nab * 2 * (zp + xp) * 2; i += TC_NT) {
            const int q = i & 1, rr = i >> 1;
            const int row = rr % (zp + xp), hl = (rr / (zp + xp)) & 1, bi = rr / (2 * (zp + xp));
            unsigned char *B0 = sm + L.buf + bi * L.bufstride;
            unsigned char *dst = row < zp ? B0 + hl * 128 * 32 + rowchunk(2 * NCZ * jm + row, q)
                                          : B0 + L.xoff + hl * a.ncolmax * 32 + rowchunk(2 * nr + row - zp, q);
            *reinterpret_cast<float4 *>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    umma::fence_smem_to_async();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    // the iteration's field pass may start its set-up (tables, Q) on the SMs this grid leaves free
    pdl_launch_dependents();
    const uint32_t tm = tslot;
    uint32_t err = 0;

    if (warp < TC_NB) {
        // ---------------- builders: X = exy of every run (8 sites per item), Z = mu_c ez
        const int bt = tid;  // 0 .. 32 TC_NB - 1
        int it_n = 0, it_off[2], it_xr[2], it_yr[2], it_o[2];
        float it_ys[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int it = bt + u * 32 * TC_NB;
            it_off[u] = it_xr[u] = it_yr[u] = it_o[u] = 0;
            it_ys[u] = 1.f;
            if (it >= 2 * nr || xm == 2) continue;
            it_n = u + 1;
            const int p = it >> 1, o = it & 1;
            const int kxy = sslot[p].x, kx = kxy & 255, ky = (kxy >> 8) - 128;
            it_off[u] = rowchunk(2 * p, o);  // Re row; the Im row 2 p + 1 is 16 bytes further
            it_o[u] = o;
            it_xr[u] = kx;
            it_yr[u] = yrow + (ky < 0 ? -ky : ky);
            it_ys[u] = ky < 0 ? -1.f : 1.f;
        }
        // Z items: one row (c, j, cos|sin) x 8 sites each, on the whole warps after the X items
        // (or as many of the last as TC_ZMAX items per thread need); row decoded once here
        // (X cached: the halves of the builders take the two MMA steps of a stage, one Z item a thread -- at most
        // 252 -- so that a step's chain of loads, splits and fences runs beside the next one's)
        const int nzi = 2 * NCZ * jm * 2;
        const int half = xm == 2 ? warp / (TC_NB / 2) : 0;
        const int zwarps = xm == 2 ? TC_NB / 2 : max((nzi + 32 * TC_ZMAX - 1) / (32 * TC_ZMAX), TC_NB - (2 * nr + 31) / 32);
        const int zthreads = 32 * zwarps, zbase = xm == 2 ? half * zthreads : 32 * TC_NB - zthreads;
        int zn = 0, zoff[TC_ZMAX], zmo[TC_ZMAX], zer[TC_ZMAX], zcs[TC_ZMAX], zq[TC_ZMAX];
#pragma unroll
        for (int u = 0; u < TC_ZMAX; u++) {
            const int zi = bt - zbase + u * zthreads;
            zoff[u] = zmo[u] = zer[u] = zcs[u] = zq[u] = 0;
            if (bt < zbase || zi >= nzi) continue;
            zn = u + 1;
            const int zr = zi >> 1, c = zr / (2 * jm);
            zoff[u] = rowchunk(zr, zi & 1);
            zmo[u] = c * TC_SS + 8 * (zi & 1);         // component row of muz, first site
            zer[u] = yrow + kp.kmax + 1 + G.j0 + ((zr >> 1) % jm);  // ez row of |kz| = j0 + j
            zcs[u] = zr & 1;
            zq[u] = 8 * (zi & 1);
        }
        for (int ts = 0; ts < nstage && !err; ts++) {
            const int tb = ts % TC_NST;
            err |= (uint32_t)umma::mbar_wait(&mfull[tb], (uint32_t)((ts / TC_NST) & 1), TC_WAIT);
            const unsigned char *tab = sm + tb * L.stage;
            const float *muz = reinterpret_cast<const float *>(tab + L.muz);
            for (int ks = half; ks < (xm == 2 ? half + 1 : TC_SS / TC_KS) && !err; ks++) {
                const int sub = ts * (TC_SS / TC_KS) + ks, ab = sub % nab, use = sub / nab;
                if (use > 0) err |= (uint32_t)umma::mbar_wait(&aempty[ab], (uint32_t)((use - 1) & 1), TC_WAIT);
                unsigned char *Bf = sm + L.buf + ab * L.bufstride;
                const int so = ks * TC_KS;
                uint4 *xb = xm ? xc + (size_t)sub * (a.xblock / 16) : nullptr;  // this block in the cache
                if (xm == 2 && bt == zbase) {
                    mbar_expect_tx(&xfull[ab], 2u * (uint32_t)xbytes);
                    bulk_load_stream(Bf + L.xoff, xb, (uint32_t)xbytes, &xfull[ab], a.xkeep);
                    bulk_load_stream(Bf + L.xoff + xlo, xb + xbytes / 16, (uint32_t)xbytes, &xfull[ab], a.xkeep);
                }
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    if (u >= it_n) break;
                    const int sq = so + 8 * it_o[u];
                    const float ys = it_ys[u];
                    float re[8], im[8];
#pragma unroll
                    for (int h = 0; h < 4; h++) {
                        const float4 xx = *tab_chunk(tab, L.boxb, it_xr[u], sq + 2 * h);
                        const float4 yy = *tab_chunk(tab, L.boxb, it_yr[u], sq + 2 * h);
                        // ewald.f90:30-31: coskxky = cx cy - sx sy, sinkxky = sx cy + cx sy
                        re[2 * h] = xx.x * yy.x - xx.y * (ys * yy.y);
                        im[2 * h] = xx.y * yy.x + xx.x * (ys * yy.y);
                        re[2 * h + 1] = xx.z * yy.z - xx.w * (ys * yy.w);
                        im[2 * h + 1] = xx.w * yy.z + xx.z * (ys * yy.w);
                    }
                    uint4 rh, rl, ih, il;
                    split8_h(re, rh, rl);
                    split8_h(im, ih, il);
                    unsigned char *xp = Bf + L.xoff + it_off[u];
                    *reinterpret_cast<uint4 *>(xp) = rh;
                    *reinterpret_cast<uint4 *>(xp + 16) = ih;
                    *reinterpret_cast<uint4 *>(xp + xlo) = rl;
                    *reinterpret_cast<uint4 *>(xp + xlo + 16) = il;
                    if (xm == 1) {
                        uint4 *g = xb + it_off[u] / 16;
                        g[0] = rh;
                        g[1] = ih;
                        g[xbytes / 16] = rl;
                        g[xbytes / 16 + 1] = il;
                    }
                }
#pragma unroll
                for (int u = 0; u < TC_ZMAX; u++) {
                    if (u >= zn) break;
                    const int sq = so + zq[u];
                    const float4 m0 = *reinterpret_cast<const float4 *>(muz + zmo[u] + so);
                    const float4 m1 = *reinterpret_cast<const float4 *>(muz + zmo[u] + so + 4);
                    const float mc[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
                    float v[8];
#pragma unroll
                    for (int h = 0; h < 4; h++) {
                        const float4 zz = *tab_chunk(tab, L.boxb, zer[u], sq + 2 * h);
                        v[2 * h] = mc[2 * h] * (zcs[u] ? zz.y : zz.x);
                        v[2 * h + 1] = mc[2 * h + 1] * (zcs[u] ? zz.w : zz.z);
                    }
                    uint4 hi, lo;
                    split8_h(v, hi, lo);
                    *reinterpret_cast<uint4 *>(Bf + zoff[u]) = hi;
                    *reinterpret_cast<uint4 *>(Bf + 128 * 32 + zoff[u]) = lo;
                }
                umma::fence_smem_to_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&afull[ab]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[tb]);
        }
    } else if (warp == TC_MMA_WARP) {
        // ---------------- MMA issue (one thread): D[128][ncol] += Z X^T, two N halves
        if (lane == 0) {
            const uint32_t idesc_base = umma::idesc_f16(128, 16) & ~(0x3Fu << 17);
            for (int sub = 0; sub < nsub && !err; sub++) {
                const int ab = sub % nab, use = sub / nab;
                err |= (uint32_t)umma::mbar_wait(&afull[ab], (uint32_t)(use & 1), TC_WAIT);
                if (xm == 2) err |= (uint32_t)umma::mbar_wait(&xfull[ab], (uint32_t)(use & 1), TC_WAIT);
                if (err) break;
                umma::fence_after_sync();
                const uint32_t zH = umma::smem_u32(sm + L.buf + ab * L.bufstride), zL = zH + 128 * 32;
                const uint32_t xH = zH + L.xoff, xL = xH + xlo;
                const uint64_t dz_h = umma::sdesc(zH, 128, 256), dz_l = umma::sdesc(zL, 128, 256);
                for (int nt = 0; nt * 256 < G.ncol; nt++) {
                    const int N = min(256, G.ncol - nt * 256);
                    const uint32_t id = idesc_base | ((uint32_t)(N >> 3) << 17);
                    const uint32_t d = tm + (uint32_t)(nt * 256);
                    // rows 256 nt.. of X: 32 row groups of 256 bytes per half
                    const uint64_t dx_h = umma::sdesc(xH + nt * 8192, 128, 256), dx_l = umma::sdesc(xL + nt * 8192, 128, 256);
                    umma::mma_f16(d, dz_h, dx_h, id, sub > 0);
                    umma::mma_f16(d, dz_h, dx_l, id, 1);
                    umma::mma_f16(d, dz_l, dx_h, id, 1);
                }
                umma::commit(&aempty[ab]);
            }
        }
    } else {
        // ---------------- producer: as each table stage lands, the dipoles as 3 component rows
        // (2^6 mu_c, zero outside [s_lo, g1)) for the builders; stages beyond the first TC_NST are
        // copied into a buffer once all builder warps are done with its previous stage
        int issued = min(nstage, TC_NST), landed = 0;
        for (int ts = 0; ts < nstage && !err; ts++) {
            const int tb = ts % TC_NST;
            err |= (uint32_t)umma::mbar_wait(&tfull[tb], (uint32_t)((ts / TC_NST) & 1), TC_WAIT);
            if (err) break;
            landed = ts + 1;
            unsigned char *dst = sm + tb * L.stage;
            {
                const int s = g0 + ts * TC_SS + lane;
                const float4 m = reinterpret_cast<const float4 *>(dst + L.mu)[lane];
                const bool in = s >= a.s_lo && s < g1;
                float *muz = reinterpret_cast<float *>(dst + L.muz);
                if (OP == TC_OP_Q) {
                    muz[lane] = in ? TC_ZS * m.w : 0.f;
                } else {
                    muz[lane] = in ? TC_ZS * m.x : 0.f;
                    muz[TC_SS + lane] = in ? TC_ZS * m.y : 0.f;
                    muz[2 * TC_SS + lane] = in ? TC_ZS * m.z : 0.f;
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&mfull[tb]);
            const int tr = ts + TC_NST - 1;  // refill the buffer of stage ts - 1
            if (ts >= 1 && tr < nstage) {
                err |= (uint32_t)umma::mbar_wait(&tempty[tr % TC_NST], (uint32_t)(((ts - 1) / TC_NST) & 1), TC_WAIT);
                if (err) break;
                if (lane == 0) issue_stage(tr);
                issued = tr + 1;
                __syncwarp();
            }
        }
        // copies still in flight after a timeout land before the CTA leaves
        for (int w = landed; w < issued && err; w++)
            umma::mbar_wait(&tfull[w % TC_NST], (uint32_t)((w / TC_NST) & 1), TC_WAIT);
    }

    // ---------------- all MMAs done: the last commit tracks every earlier MMA of the issuing thread
    if (nsub > 0) {
        const int last = nsub - 1;
        int to = umma::mbar_wait(&aempty[last % nab], (uint32_t)((last / nab) & 1), TC_WAIT);
        if (to) to = umma::mbar_wait(&aempty[last % nab], (uint32_t)((last / nab) & 1), TC_WAIT);
        err |= (uint32_t)to;
    }
    umma::fence_after_sync();
    const bool bad = __syncthreads_or((int)err) != 0;

    // this CTA's slice of the cluster reduction: k-vectors of the dipole components, else items (run pair, |kz|);
    // the thread's first item is fetched now, under the epilogue
    const int cr = (int)cluster_rank(), cn = gridDim.x;
    const int ni = (OP == TC_OP_DIP) ? G.nkl : G.np * jm;
    const int i0 = (int)((long)cr * ni / cn), i1 = (int)((long)(cr + 1) * ni / cn);
    struct Item {
        int4 vp;
        TcKW kw[4];  // (+ky, +kz), (+ky, -kz), (-ky, +kz), (-ky, -kz); k < 0: none
    };
    auto local_k = [&](const int4 &vp, int j, int u) {  // the k-vector's local index, -1: none
        const int p = (u & 2) ? (vp.x >> 16) & 0xffff : vp.x & 0xffff, kz = (u & 1) ? -j : j;
        if (p == 0xffff || ((u & 1) && j == 0)) return -1;
        const int4 sl = sslot[p];
        return kz >= sl.z && kz < sl.z + sl.w ? sl.y + kz - sl.z : -1;
    };
    auto fetch = [&](int it, Item &x) {
        const int q = it / jm, j = G.j0 + it - q * jm;
        x.vp = a.vp[G.vp0 + q];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int i = local_k(x.vp, j, u);
            x.kw[u] = i >= 0 ? a.kw[G.kgoff + i] : TcKW{-1, 0.f};
        }
    };
    Item first;
    if (OP != TC_OP_DIP && i0 + tid < i1) fetch(i0 + tid, first);
    // epilogue: TMEM -> shared, 64 runs (128 columns) at a time -> partial S of every k of the group
    float *stg = reinterpret_cast<float *>(sm);                       // [128][TC_LD]
    float2 *pt = reinterpret_cast<float2 *>(sm + 128 * TC_LD * 4);    // [nkl][NPT]
    for (int ch = 0; ch * TC_CH < nr && !bad; ch++) {
        if (warp < 16) {
            const int lq = warp & 3, part = warp >> 2;  // 4 lane quarters x 4 column quarters
            const int col = ch * 2 * TC_CH + 32 * part;
            float v[32];
            float *row = stg + (32 * lq + lane) * TC_LD + 32 * part;
            const uint32_t t0 = tm + ((uint32_t)(32 * lq) << 16) + (uint32_t)col;
            if (nsub > 0) {
                umma::tmem_ld16x2(t0, t0 + 16, v);
            } else {
#pragma unroll
                for (int j = 0; j < 32; j++) v[j] = 0.f;
            }
#pragma unroll
            for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4 *>(row + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        }
        __syncthreads();
        for (int i = tid; i < TC_CH * jm; i += TC_NT) {
            const int q = i % TC_CH, jj = i / TC_CH, p = ch * TC_CH + q, j = G.j0 + jj;  // row jj: |kz| = j
            if (p >= nr) continue;
            const int4 sl = sslot[p];  // run, local offset, kzlo, nkz
            const bool plus = j >= sl.z && j < sl.z + sl.w;
            const bool minus = j > 0 && -j >= sl.z && -j < sl.z + sl.w;
            if (!plus && !minus) continue;
            float2 gp[NCZ], gm[NCZ];
#pragma unroll
            for (int c = 0; c < NCZ; c++) {
                const int rc = (c * jm + jj) * 2;
                // (x, y) = (Re exy, Im exy) against mu_c c_j (row rc) and mu_c s_j (row rc + 1)
                const float2 dc = *reinterpret_cast<const float2 *>(stg + rc * TC_LD + 2 * q);
                const float2 ds = *reinterpret_cast<const float2 *>(stg + (rc + 1) * TC_LD + 2 * q);
                gp[c] = make_float2(dc.x - ds.y, ds.x + dc.y);
                gm[c] = make_float2(dc.x + ds.y, dc.y - ds.x);
            }
            const float zs = 1.f / TC_ZS;
            if (OP == TC_OP_MU) {
                const float2 kv = make_float2(sskv[p].x * zs, sskv[p].y * zs);
                if (plus) {
                    const float kz = skz[kp.lmax + j] * zs;
                    pt[sl.y + j - sl.z] = make_float2(fmaf(kz, gp[NCZ - 1].x, fmaf(kv.y, gp[1 % NCZ].x, kv.x * gp[0].x)),
                                                      fmaf(kz, gp[NCZ - 1].y, fmaf(kv.y, gp[1 % NCZ].y, kv.x * gp[0].y)));
                }
                if (minus) {
                    const float kz = skz[kp.lmax - j] * zs;
                    pt[sl.y - j - sl.z] = make_float2(fmaf(kz, gm[NCZ - 1].x, fmaf(kv.y, gm[1 % NCZ].x, kv.x * gm[0].x)),
                                                      fmaf(kz, gm[NCZ - 1].y, fmaf(kv.y, gm[1 % NCZ].y, kv.x * gm[0].y)));
                }
            } else {
                // charges: S itself; dipole components: the three G_c
#pragma unroll
                for (int c = 0; c < NPT; c++) {
                    if (plus) pt[NPT * (sl.y + j - sl.z) + c] = make_float2(zs * gp[c].x, zs * gp[c].y);
                    if (minus) pt[NPT * (sl.y - j - sl.z) + c] = make_float2(zs * gm[c].x, zs * gm[c].y);
                }
            }
        }
        __syncthreads();
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        umma::fence_after_sync();
        umma::tmem_dealloc(tm, 512);
        umma::tmem_relinquish();
    }
    // cluster: add the partials of all site groups over this CTA's slice (groups in order, in FP32: FP64
    // arithmetic is slow on this part, and the partials carry only the split operands' ~2^-21 anyway)
    cluster_sync();
    const uint32_t pbase = umma::smem_u32(pt);
    auto total = [&](int i) {
        float2 v[TC_CLMAX];
#pragma unroll
        for (int c = 0; c < TC_CLMAX; c++)
            if (c < cn) v[c] = ld_cluster_f2(pbase + 8u * (uint32_t)i, (uint32_t)c);
        float sx = 0.f, sy = 0.f;
#pragma unroll
        for (int c = 0; c < TC_CLMAX; c++)
            if (c < cn) {
                sx += v[c].x;
                sy += v[c].y;
            }
        return make_float2(sx, sy);
    };
    if (OP == TC_OP_DIP && !bad) {
        for (int i = i0 + tid; i < i1; i += TC_NT) {
            const TcKW kw = a.kw[G.kgoff + i];
            if (kw.k < 0) continue;  // a k-vector of the run that another (band) group sums
            for (int e = 0; e < NPT; e++) {
                const float2 t = total(NPT * i + e);
                kp.Sdip[((size_t)b * kp.nk + kw.k) * 3 + e] = make_double2((double)t.x, (double)t.y);
            }
        }
    }
    // charges and dipoles: Sq = S or Sm = (-Im, Re), the reference's rQm, iQm (ewald.f90:106-107), the FP32
    // weights 4 pi Ak / V conj(S), and a pair's rows of the field pass's V (k_field_v's job, which took a
    // launch of 5 us an iteration at 512 x 32)
    for (int it = i0 + tid; OP != TC_OP_DIP && it < i1 && !bad; it += TC_NT) {
        Item x = first;
        if (it != i0 + tid) fetch(it, x);
        const int j = G.j0 + it % jm;
        float2 w[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            w[u] = make_float2(0.f, 0.f);
            const TcKW kw = x.kw[u];
            if (kw.k < 0) continue;
            const float2 t = total(local_k(x.vp, j, u));
            if (OP == TC_OP_MU) {
                kp.Sm[(size_t)b * kp.nk + kw.k] = make_double2(-(double)t.y, (double)t.x);
                w[u] = make_float2(-kw.w * t.y, -kw.w * t.x);
            } else {
                kp.Sq[(size_t)b * kp.nk + kw.k] = make_double2((double)t.x, (double)t.y);
                w[u] = make_float2(kw.w * t.x, -kw.w * t.y);
            }
            kp.Wf[((size_t)b * 2 + (OP == TC_OP_MU ? 1 : 0)) * kp.nk + kw.k] = w[u];
        }
        if (!a.V || j >= x.vp.w) continue;
        uint32_t *hi = reinterpret_cast<uint32_t *>(a.V + (size_t)b * a.vstride + x.vp.y) + (j >> 2) * 32 + (j & 3);
        uint32_t *lo = hi + 4 * x.vp.z;
        v_rows(w, skz[kp.lmax + j], [&](int r, float c, float sn) {
            const __half2 h = __floats2half2_rn(c, sn);
            const float2 hf = __half22float2(h);
            const __half2 l = __floats2half2_rn(c - hf.x, sn - hf.y);
            hi[4 * r] = *reinterpret_cast<const uint32_t *>(&h);
            lo[4 * r] = *reinterpret_cast<const uint32_t *>(&l);
        });
    }
    cluster_sync();  // remote reads done before any CTA of the cluster leaves
    if (bad && tid == 0) atomicOr(kp.err, 8u);
    if (a.pdl == 2) pdl_wait();  // this grid's end is the band groups' end too
}

// ---------------------------------------------------------------------------------------
// Tensor-core field passes of the mixed engine (the per-iteration k_field_f<F_D> sum,
// ewald.f90:114-117, and the charge field and the force pass): at every site s of a bead,
//   E_x,y(s) = sum_run k_x,y Im(exy(s) T0(s)),   E_z(s) = sum_run Im(exy(s) T1(s)),
//   T0(s) = sum_kz W(kz) ez(s, kz),   T1(s) = sum_kz k_z W(kz) ez(s, kz),
// with W the FP32 weights 4 pi Ak / V conj(S) of the run's k-vectors. Folding +-j as in the
// structure factor (W+ = W(+j), W- = W(-j), Wp = W+ + W-, Wm = W+ - W-):
//   T0 = sum_j (Wp.x c_j - Wm.y s_j) + i (Wp.y c_j + Wm.x s_j)
//   T1 = sum_j k_z(j) [(Wm.x c_j - Wp.y s_j) + i (Wm.y c_j + Wp.x s_j)]
// so T0, T1 of every run at every site are one GEMM per bead,
//   D[s][(run, comp)] = sum_q Q[s][q] V[(run, comp)][q],  comp = T0re|T0im|T1re|T1im,  q = (j, cos|sin),
// with the sites on M (128 per CTA), runs x components on N and only 2 (max |kz| + 1) terms on K (FP16
// hi + lo split, three MMAs per 16-term K step); each TMEM row is then contracted with exy(s, run).
//
// V is formed from the weights once a pass, by the structure factor that makes them or by k_field_v (every CTA
// of a bead formed it before, and V, MMAs and contraction followed one another: 492 us a pass at 4096 x 32
// against 188), and the runs are taken in pairs (kx, +ky), (kx, -ky). With T+, T- the pair's sums, Ts = T+ + T-, Td = T+ - T- and
// e(kx x +- ky y) = ex (cy +- i sy),
//   e+ T+ + e- T- = ex U,  U = cy Ts + i sy Td;   e+ T+ - e- T- = ex V,  V = cy Td + i sy Ts,
// so a pair's contraction is U0, V0 (T0) and U1 (T1) and three products with ex: 20 FMAs and one load
// each of ex and ey for two runs, where one run took 15 and both loads. The rows of V are Ts, Td of T0 and T1
// (8 a pair) and, for the dipole force, of T2 and with V1 (12 a pair: the force is -G mu with
// G = (kx^2 S0, kx ky D0, ky^2 S0, kx S1, ky D1, S2), S and D the real parts of ex U and ex V).
//
// A chunk is the pairs of one accumulator (256 columns at most, half of TMEM), sorted by their largest |kz| so
// that later chunks have fewer K steps. The control warp copies chunk c + 1 of V (one bulk copy) while the MMAs
// of chunk c run into one half of TMEM and 16 warps contract chunk c - 1 from the other.
constexpr int TF_NT = 512;
constexpr int TF_SITES = 128;             // sites per CTA (M)
// byte offset of the 16-byte chunk jc (halves 8 jc .. 8 jc + 7) of row n in a K-major operand
// with kcm core matrices along K
PIMD_D int rowchunk_k(int n, int jc, int kcm) { return (((n >> 3) * kcm + jc) << 7) + ((n & 7) << 4); }

// What a field pass does with the field e (and potential, e[3]) of its sites: thread tid < 128 of the
// block holds site s_own (own: in the pass's range and its sums are good; bad: the block gave up).
template <int MODE, int NT>
PIMD_D void field_out(const KP &kp, int b, int t, int s_own, bool own, bool bad, const float (&e)[4], const DdSite &din, int iter) {
    if (MODE == TF_Q && (kp.fx_mode & 1)) {  // into the scratch (this pass runs beside the pair kernels)
        if (own)
            kp.Fx[(size_t)b * kp.S + s_own] =
                make_double4_32a((double)e[0], (double)e[1], (double)e[2], s_own >= kp.fq ? (double)e[3] : 0.0);
        return;
    }
    if ((MODE == TF_QG || MODE == TF_DG) && (kp.fx_mode & 2)) {
        if (own) {
            const size_t gs = (size_t)b * kp.S + s_own;
            if (MODE == TF_QG) {
                const double q = kp.pos[gs].w;
                kp.Fx[gs] = make_double4_32a(-q * (double)e[0], -q * (double)e[1], -q * (double)e[2],
                                             s_own >= kp.fq ? (double)e[3] : 0.0);
            } else {
                double4_32a f = kp.Fx[gs];
                f.x += (double)e[0];
                f.y += (double)e[1];
                f.z += (double)e[2];
                kp.Fx[gs] = f;
            }
        }
        return;
    }
    if (MODE == TF_Q) {
        // ewald.f90:45-49 as k_field_finish<F_Q>: Efq += E, phi += (charged sites)
        if (own) {
            const size_t gs = (size_t)b * kp.S + s_own;
            double4_32a f = kp.F[gs];
            f.x += (double)e[0];
            f.y += (double)e[1];
            f.z += (double)e[2];
            if (s_own >= kp.fq) f.w += (double)e[3];
            kp.F[gs] = f;
        }
        return;
    }
    if (MODE == TF_QG || MODE == TF_DG) {
        // as k_field_finish<F_QD>: dR += -q E (charge part) or the dipole force; phi of the
        // dipole structure factor at the charged sites
        if (own) {
            const size_t gs = (size_t)b * kp.S + s_own;
            const double q = MODE == TF_QG ? kp.pos[gs].w : -1.0;
            kp.dR[3 * gs + 0] -= q * (double)e[0];
            kp.dR[3 * gs + 1] -= q * (double)e[1];
            kp.dR[3 * gs + 2] -= q * (double)e[2];
            if (MODE == TF_QG && s_own >= kp.fq) kp.F[gs].w += (double)e[3];
        }
        return;
    }
    if (kp.dd_async) {
        // the real-space field runs beside this pass: store the reciprocal field, arrive, and
        // run the unit's SOR update if the real-space blocks of its molecules are done
        if (own) kp.Erec[(size_t)b * kp.S + s_own] = make_float4(e[0], e[1], e[2], 0.f);
        const float er[3] = {e[0], e[1], e[2]};
        if (dd_unit_arrive(kp, b, t)) dd_unit_sor<NT>(kp, b, t, own, er);
        return;
    }
    // the iteration's FP64 SOR update at the CTA's dipole sites, then the block's end
    double av[2] = {0.0, 0.0};
    if (own) {
        const double E[3] = {(double)e[0], (double)e[1], (double)e[2]};
        dd_sor_apply(kp, b, s_own, din, E, iter, av);
    }
    dd_block_end<NT, TF_SITES / 32>(kp, b, av, !bad);  // own sites: threads < TF_SITES
}

constexpr int TP_NT = TF_NT + 32;         // 16 contracting warps, one for copies and MMAs
constexpr int TP_VT = 128;                // threads of a k_field_v block
constexpr int TP_RP = 32;                 // pairs a chunk at most (8 rows each)
constexpr int TP_RPD = 20;                // the same with 12 rows each
constexpr int TP_RING = 8;                // pair tables in shared memory

struct TpArgs {
    const int4 *pair;    // [chunk][rp] ex row offset + 65536 key, ey row offset + 65536 key, k_x, k_y (float bits)
    const int2 *chunk;   // K row blocks (4 |kz| each, even) of the chunk, its offset in a bead's V (16-byte words)
    const int4 *kidx;    // [chunk rp + pair][4 TP jmax blocks] k-vectors of (+ky, +kz), (+ky, -kz), (-ky, +kz), (-ky, -kz)
    const float *kzv;    // k_z by kz + lmax
    uint4 *V;            // [P][vstride] per chunk: hi rows, lo rows
    int vstride, nchunk, rp, kcm;  // kcm: K row blocks of Q (the longest)
    int sbase, s_lo, s_hi;
    int skipconv, pdl;
};

template <bool DG>
__global__ void __launch_bounds__(TP_VT) k_field_v(KP kp, TpArgs a, int slot) {
    constexpr int NC = DG ? 12 : 8;
    const int c = blockIdx.x, b = blockIdx.y;
    const int2 ch = a.chunk[c];
    const int kc = ch.x;
    // the field pass may set up; it waits for this grid, which waits for the structure factor here
    pdl_launch_dependents();
    if (a.pdl) pdl_wait();
    if (a.skipconv && bead_converged(kp, b)) return;
    uint4 *Vh = a.V + (size_t)b * a.vstride + ch.y, *Vl = Vh + NC * a.rp * kc;
    const float2 *W = kp.Wf + ((size_t)b * 2 + slot) * kp.nk;
    for (int it = threadIdx.x; it < a.rp * kc; it += blockDim.x) {
        const int pl = it / kc, jc = it - pl * kc;
        const int4 *ki = a.kidx + (size_t)(c * a.rp + pl) * 4 * a.kcm + 4 * jc;
        float v[NC][8];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int4 k = ki[e];
            auto weight = [&](int i) {
                if (i < 0) return make_float2(0.f, 0.f);
                float2 x = W[i];
                if (DG) {  // both weight slots
                    const float2 y = W[kp.nk + i];
                    x = make_float2(x.x + y.x, x.y + y.y);
                }
                return x;
            };
            const float2 w[4] = {weight(k.x), weight(k.y), weight(k.z), weight(k.w)};
            const int j = 4 * jc + e;
            v_rows<DG>(w, j <= kp.lmax ? a.kzv[kp.lmax + j] : 0.f, [&](int r, float c, float sn) {
                v[r][2 * e] = c;
                v[r][2 * e + 1] = sn;
            });
        }
#pragma unroll
        for (int r = 0; r < NC; r++) {
            uint4 hi, lo;
            split8_h(v[r], hi, lo);
            const int n = NC * pl + r, o = ((n >> 3) * kc + jc) * 8 + (n & 7);
            Vh[o] = hi;
            Vl[o] = lo;
        }
    }
}

// Shared memory (from a 1024-aligned base): ex and ey tables of 128 sites (8 TMA boxes), Q hi and lo, two V
// buffers; the ez tables, read for Q before the second buffer is filled, lie in that one.
struct TpSmem {
    int boxxy, boxz, Q, V, vbuf, total;
    __host__ __device__ TpSmem(int rowsxy, int rowsz, int kcm, int rows) {
        boxxy = ((rowsxy * 128 + 1023) / 1024) * 1024;
        boxz = ((rowsz * 128 + 1023) / 1024) * 1024;
        Q = 8 * boxxy;
        V = Q + 2 * TF_SITES * kcm * 16;
        vbuf = ((2 * rows * kcm * 16 + 1023) / 1024) * 1024;
        total = V + vbuf + (vbuf > 8 * boxz ? vbuf : 8 * boxz) + 1024;
    }
};

template <int MODE>
__global__ void __launch_bounds__(TP_NT, 1)
    k_field_p(const __grid_constant__ CUtensorMap mapxy, const __grid_constant__ CUtensorMap mapz, KP kp, TpArgs a) {
    constexpr bool DG = MODE == TF_DG || MODE == TF_DE;
    constexpr int NC = DG ? 12 : 8, EP = (DG ? TP_RPD : TP_RP) / 4;  // pairs a warp at most
    const int t = blockIdx.x, b = blockIdx.y;
    if (MODE == TF_D) pdl_launch_dependents();
    if (MODE == TF_D && bead_converged(kp, b)) {
        if (a.pdl) pdl_wait();
        const double zero[2] = {0.0, 0.0};
        if (kp.dd_async) {
            const float z[3] = {0.f, 0.f, 0.f};
            if (dd_unit_arrive(kp, b, t)) dd_unit_sor<TP_NT>(kp, b, t, false, z);
            return;
        }
        dd_block_end<TP_NT>(kp, b, zero, false);
        return;
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rowsxy = kp.hmax + kp.kmax + 2, rp = a.rp, kcm = a.kcm, nch = a.nchunk;
    const TpSmem L(rowsxy, kp.lmax + 1, kcm, NC * rp);
    extern __shared__ __align__(1024) unsigned char sm_raw[];
    unsigned char *sm = sm_raw + ((1024u - (umma::smem_u32(sm_raw) & 1023u)) & 1023u);
    __shared__ uint64_t tbar, vfull[2], mdone[2], tfree[2], pfull[TP_RING];
    __shared__ uint32_t tslot;
    // the chunks' pairs, a ring: the copy of chunk c + 5 follows the MMAs of c + 3, which follow every warp's
    // TMEM load of c + 1 and with it the warp's contraction of c
    __shared__ __align__(16) int4 sp[TP_RING][TP_RP];
    const int sb = a.sbase + t * TF_SITES;
    const uint4 *Vb = a.V + (size_t)b * a.vstride;
    unsigned char *zt = sm + L.V + L.vbuf;
    auto copy_chunk = [&](int c) {
        const int2 ch = a.chunk[c];
        const uint32_t vb = (uint32_t)(2 * NC * rp * ch.x * 16);
        mbar_expect_tx(&vfull[c & 1], vb);
        bulk_load(sm + L.V + (c & 1) * L.vbuf, Vb + ch.y, vb, &vfull[c & 1]);
        mbar_expect_tx(&pfull[c % TP_RING], (uint32_t)rp * 16u);
        bulk_load(sp[c % TP_RING], a.pair + (size_t)c * rp, (uint32_t)rp * 16u, &pfull[c % TP_RING]);
    };
    if (tid == TF_NT) {
        umma::mbar_init(&tbar, 1);
        for (int i = 0; i < 2; i++) {
            umma::mbar_init(&vfull[i], 1);
            umma::mbar_init(&mdone[i], 1);
            umma::mbar_init(&tfree[i], TF_NT / 32);
        }
        for (int i = 0; i < TP_RING; i++) umma::mbar_init(&pfull[i], 1);
        mbar_expect_tx(&tbar, 8u * (uint32_t)((rowsxy + kp.lmax + 1) * 128));
        for (int i = 0; i < 8; i++) {
            tma_load_2d(zt + i * L.boxz, &mapz, 2 * (sb + 16 * i), b * kp.ntab + rowsxy, &tbar);
            tma_load_2d(sm + i * L.boxxy, &mapxy, 2 * (sb + 16 * i), b * kp.ntab, &tbar);
        }
    }
    if (warp == 0) umma::tmem_alloc(&tslot, 512);
    const int iter = dd_done(kp) + 1;
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tm = tslot;
    uint32_t err = 0;
    int issued = 0;
    if (tid == TF_NT) {  // the first chunk, beside Q
        if (a.pdl) pdl_wait();
        copy_chunk(0);
        issued = 1;
    }
    __syncwarp();
    unsigned char *Qh = sm + L.Q, *Ql = Qh + TF_SITES * kcm * 16;
    if (warp < TF_NT / 32) {
        err |= (uint32_t)umma::mbar_wait(&tbar, 0, TC_WAIT);
        for (int it = tid; it < TF_SITES * kcm; it += TF_NT) {
            const int s = it % TF_SITES, jc = it / TF_SITES;
            float v[8];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int j = 4 * jc + e;
                const float2 z = j <= kp.lmax ? tab_elem(zt, L.boxz, j, s) : make_float2(0.f, 0.f);
                v[2 * e] = z.x;
                v[2 * e + 1] = z.y;
            }
            uint4 hi, lo;
            split8_h(v, hi, lo);
            const int o = rowchunk_k(s, jc, kcm);
            *reinterpret_cast<uint4 *>(Qh + o) = hi;
            *reinterpret_cast<uint4 *>(Ql + o) = lo;
        }
    }
    // everything above reads only the positions; from here on V and the iteration's fields (a programmatic
    // launch waits for them here); the SOR inputs of the CTA's dipole sites
    if (a.pdl) pdl_wait();
    const int s_own = sb + tid;
    const bool own = tid < TF_SITES && s_own >= a.s_lo && s_own < a.s_hi;
    DdSite din;
    if (MODE == TF_D && own && !kp.dd_async) dd_sor_load(kp, b, s_own, din);
    umma::fence_smem_to_async();
    umma::fence_before_sync();
    bool bad = __syncthreads_or((int)err) != 0;
    umma::fence_after_sync();
    constexpr int NA = MODE == TF_DE ? 9 : DG ? 6 : 4;
    float acc[NA];
#pragma unroll
    for (int i = 0; i < NA; i++) acc[i] = 0.f;
    const int lq = warp & 3, part = warp >> 2, sl = 32 * lq + lane;
    err = 0;
    if (warp == TF_NT / 32) {
        if (lane == 0 && !bad) {
            const uint32_t idesc = (umma::idesc_f16(128, 16) & ~(0x3Fu << 17)) | ((uint32_t)(NC * rp >> 3) << 17);
            const uint32_t qh = umma::smem_u32(Qh), ql = umma::smem_u32(Ql);
            int mma = 0;  // chunks whose MMAs are issued
            for (int c = 0; c < nch; c++) {
                const int h = c & 1;
                // the next chunk's copy goes out once the MMAs that read its buffer are done
                if (c + 1 < nch) {
                    if (c >= 1) err |= (uint32_t)umma::mbar_wait(&mdone[h ^ 1], (uint32_t)(((c - 1) >> 1) & 1), TC_WAIT);
                    if (err) break;
                    copy_chunk(c + 1);
                    issued = c + 2;
                }
                err |= (uint32_t)umma::mbar_wait(&vfull[h], (uint32_t)((c >> 1) & 1), TC_WAIT);
                if (c >= 2) err |= (uint32_t)umma::mbar_wait(&tfree[h], (uint32_t)(((c - 2) >> 1) & 1), TC_WAIT);
                if (err) break;
                umma::fence_after_sync();
                const int kc = a.chunk[c].x;
                const uint32_t vh = umma::smem_u32(sm + L.V + h * L.vbuf), vl = vh + (uint32_t)(NC * rp * kc * 16);
                const uint32_t d = tm + (uint32_t)(256 * h);
                for (int ks = 0; ks < kc / 2; ks++) {
                    const uint64_t dq_h = umma::sdesc(qh + ks * 256, 128, kcm * 128), dq_l = umma::sdesc(ql + ks * 256, 128, kcm * 128);
                    const uint64_t dv_h = umma::sdesc(vh + ks * 256, 128, kc * 128), dv_l = umma::sdesc(vl + ks * 256, 128, kc * 128);
                    umma::mma_f16(d, dq_h, dv_h, idesc, ks > 0);
                    umma::mma_f16(d, dq_h, dv_l, idesc, 1);
                    umma::mma_f16(d, dq_l, dv_h, idesc, 1);
                }
                umma::commit(&mdone[h]);
                mma = c + 1;
            }
            // MMAs and copies still in flight end before the CTA leaves
            for (int c = max(0, mma - 2); c < mma; c++) err |= (uint32_t)umma::mbar_wait(&mdone[c & 1], (uint32_t)((c >> 1) & 1), TC_WAIT);
            for (int c = mma; c < issued; c++) umma::mbar_wait(&vfull[c & 1], (uint32_t)((c >> 1) & 1), TC_WAIT);
            for (int c = max(0, issued - TP_RING); c < issued; c++) umma::mbar_wait(&pfull[c % TP_RING], (uint32_t)((c / TP_RING) & 1), TC_WAIT);
        } else if (lane == 0 && issued) {
            umma::mbar_wait(&vfull[0], 0, TC_WAIT);
            umma::mbar_wait(&pfull[0], 0, TC_WAIT);
        }
        __syncwarp();
    } else if (!bad) {
        const int q4 = rp / 4;
        // the lane's site in the staged tables: its box and float2 slot, and its 16-byte chunk (before the swizzle) times 16
        const unsigned char *tsite = sm + (sl >> 4) * L.boxxy + (sl & 1) * 8;
        const int cs4 = ((sl & 15) >> 1) << 4;
        const uint32_t tl = tm + ((uint32_t)(32 * lq) << 16) + (uint32_t)(part * q4 * NC);
        for (int c = 0; c < nch; c++) {
            const int h = c & 1;
            err |= (uint32_t)umma::mbar_wait(&pfull[c % TP_RING], (uint32_t)((c / TP_RING) & 1), TC_WAIT);
            err |= (uint32_t)umma::mbar_wait(&mdone[h], (uint32_t)((c >> 1) & 1), TC_WAIT);
            if (__any_sync(0xffffffffu, err != 0)) break;
            umma::fence_after_sync();
            float v[64];
            const uint32_t tc = tl + (uint32_t)(256 * h);
            umma::tmem_ld16x4(tc, tc + 16, tc + 32, tc + 48, v);
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tfree[h]);  // chunk c + 2's MMAs may overwrite it
            const int4 *pp = sp[c % TP_RING] + part * q4;
#pragma unroll
            for (int e = 0; e < EP; e++) {
                if (e >= q4) break;
                const int4 P = pp[e];
                const float kx = __int_as_float(P.z), ky = __int_as_float(P.w);
                const float2 ex = *reinterpret_cast<const float2 *>(tsite + (P.x & 0xffff) + (cs4 ^ (P.x >> 16)));
                const float2 ey = *reinterpret_cast<const float2 *>(tsite + (P.y & 0xffff) + (cs4 ^ (P.y >> 16)));
                const float *w = v + NC * e;  // Ts, Td of T0, of T1 (, of T2): re, im
                const float u0r = fmaf(ey.x, w[0], -ey.y * w[3]), u0i = fmaf(ey.x, w[1], ey.y * w[2]);
                const float v0r = fmaf(ey.x, w[2], -ey.y * w[1]), v0i = fmaf(ey.x, w[3], ey.y * w[0]);
                const float u1r = fmaf(ey.x, w[4], -ey.y * w[7]), u1i = fmaf(ey.x, w[5], ey.y * w[6]);
                if constexpr (DG) {
                    const float v1r = fmaf(ey.x, w[6], -ey.y * w[5]), v1i = fmaf(ey.x, w[7], ey.y * w[4]);
                    const float u2r = fmaf(ey.x, w[8], -ey.y * w[11]), u2i = fmaf(ey.x, w[9], ey.y * w[10]);
                    const float S0 = kx * fmaf(ex.x, u0r, -ex.y * u0i), D0 = ky * fmaf(ex.x, v0r, -ex.y * v0i);
                    acc[0] = fmaf(kx, S0, acc[0]);
                    acc[1] = fmaf(kx, D0, acc[1]);
                    acc[2] = fmaf(ky * ky, fmaf(ex.x, u0r, -ex.y * u0i), acc[2]);
                    acc[3] = fmaf(kx, fmaf(ex.x, u1r, -ex.y * u1i), acc[3]);
                    acc[4] = fmaf(ky, fmaf(ex.x, v1r, -ex.y * v1i), acc[4]);
                    acc[5] += fmaf(ex.x, u2r, -ex.y * u2i);
                    if constexpr (MODE == TF_DE) {
                        acc[6] = fmaf(kx, fmaf(ex.x, u0i, ex.y * u0r), acc[6]);
                        acc[7] = fmaf(ky, fmaf(ex.x, v0i, ex.y * v0r), acc[7]);
                        acc[8] += fmaf(ex.x, u1i, ex.y * u1r);
                    }
                } else {
                    acc[0] = fmaf(kx, fmaf(ex.x, u0i, ex.y * u0r), acc[0]);
                    acc[1] = fmaf(ky, fmaf(ex.x, v0i, ex.y * v0r), acc[1]);
                    acc[2] += fmaf(ex.x, u1i, ex.y * u1r);
                    if (MODE == TF_Q || MODE == TF_QG) acc[3] += fmaf(ex.x, u0r, -ex.y * u0i);
                }
            }
        }
    }
    float e[4] = {0.f, 0.f, 0.f, 0.f};
    if constexpr (DG) {  // the dipole of the lane's site, zero outside the range
        float mx = 0.f, my = 0.f, mz = 0.f;
        if (warp < TF_NT / 32 && sb + sl >= a.s_lo && sb + sl < a.s_hi) {
            const float4 m = kp.dipf[(size_t)b * kp.S + sb + sl];
            mx = m.x, my = m.y, mz = m.z;
        }
        e[0] = -fmaf(acc[0], mx, fmaf(acc[1], my, acc[3] * mz));
        e[1] = -fmaf(acc[1], mx, fmaf(acc[2], my, acc[4] * mz));
        e[2] = -fmaf(acc[3], mx, fmaf(acc[4], my, acc[5] * mz));
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) e[i] = acc[i];
    }
    bad = __syncthreads_or((int)(bad || err)) != 0;  // (every MMA is done: Q may be written)
    float *red = reinterpret_cast<float *>(Qh);      // the four pair quarters of each site, in order
    if (warp < TF_NT / 32) {
#pragma unroll
        for (int i = 0; i < 4; i++) red[(part * TF_SITES + sl) * 4 + i] = e[i] * (1.f / TP_WS);
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        umma::fence_after_sync();
        umma::tmem_dealloc(tm, 512);
        umma::tmem_relinquish();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) e[i] = 0.f;
    if (own && !bad) {
#pragma unroll
        for (int rq = 0; rq < 4; rq++)
#pragma unroll
            for (int i = 0; i < 4; i++) e[i] += red[(rq * TF_SITES + tid) * 4 + i];
    }
    if (bad && tid == 0) atomicOr(kp.err, 8u);
    if constexpr (MODE == TF_DE) {
        __syncthreads();
        if (warp < TF_NT / 32) {
#pragma unroll
            for (int i = 0; i < 3; i++) red[(part * TF_SITES + sl) * 4 + i] = acc[6 + i] * (1.f / TP_WS);
        }
        __syncthreads();
        if (own && !bad) {
            float f[3] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int rq = 0; rq < 4; rq++)
#pragma unroll
                for (int i = 0; i < 3; i++) f[i] += red[(rq * TF_SITES + tid) * 4 + i];
            kp.Fx[(size_t)b * kp.S + s_own] = make_double4_32a((double)f[0], (double)f[1], (double)f[2], 0.0);
        }
    }
    field_out<DG ? (int)TF_DG : MODE, TP_NT>(kp, b, t, s_own, own && !bad, bad, e, din, iter);
}

// ---------------------------------------------------------------------------------------
// host side

static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

// Pairs, chunks, k-vector indices and V of the prepared passes: which 0 the 8-row form, 1 the 12-row one.
static bool tp_init(Engine &E, int which, const std::vector<int> &jr, int dmax, std::vector<int4> *place) {
    KP &kp = E.kp;
    Engine::TpSet &T = E.tp[which];
    const int NC = which ? 12 : 8, rowsxy = kp.hmax + kp.kmax + 2, jmax = kp.lmax + 1;
    const int kcm = ((2 * jmax + 15) / 16) * 2;  // K row blocks of Q: 8 halves (4 |kz|: cos, sin) each, an even number
    if (rowsxy > 256 || rowsxy * 128 > 0xffff || jmax > 256) return false;
    int rp = which ? TP_RPD : TP_RP;
    while (rp >= 4 && TpSmem(rowsxy, jmax, kcm, NC * rp).total > dmax) rp -= 4;
    if (rp < 4) return false;
    struct Pair {
        int kx, ky, r[2], jm;
    };
    std::vector<Pair> pairs;
    std::map<std::pair<int, int>, int> at;
    for (int r = 0; r < kp.nrun; r++) {
        const KRun &run = E.h_runs[r];
        const std::pair<int, int> key(run.kx, std::abs(run.ky));
        if (!at.count(key)) {
            at[key] = (int)pairs.size();
            pairs.push_back(Pair{run.kx, key.second, {-1, -1}, 0});
        }
        Pair &p = pairs[at[key]];
        int &slot = p.r[run.ky < 0 ? 1 : 0];
        if (run.kx < 0 || slot >= 0 || (p.jm && p.jm != jr[r])) return false;  // (the structure factor keeps a pair together)
        slot = r;
        p.jm = jr[r];
    }
    std::stable_sort(pairs.begin(), pairs.end(), [](const Pair &x, const Pair &y) { return x.jm > y.jm; });
    const int np = (int)pairs.size(), nch = (np + rp - 1) / rp;
    std::vector<int4> pr((size_t)nch * rp, make_int4(0, 0, 0, 0)), ki((size_t)nch * rp * 4 * kcm, make_int4(-1, -1, -1, -1));
    std::vector<int2> chunk(nch);
    std::vector<int4> where(kp.nrun);
    int words = 0;
    auto bits = [](float f) {
        int i;
        std::memcpy(&i, &f, 4);
        return i;
    };
    for (int c = 0; c < nch; c++) {
        const int kc = ((2 * pairs[c * rp].jm + 15) / 16) * 2;
        chunk[c] = make_int2(kc, words);
        for (int q = 0; q < rp; q++) {
            // the last chunk's missing pairs: zero rows of V against the (0, 0) tables
            const int ry0 = kp.hmax + 1;
            if (c * rp + q >= np) {
                pr[c * rp + q] = make_int4(0, ry0 * 128 | ((ry0 & 7) << 4) << 16, 0, 0);
                continue;
            }
            const Pair &p = pairs[c * rp + q];
            for (int r : p.r)
                if (r >= 0) where[r] = make_int4(words + NC * q * kc, NC * rp * kc, p.jm, 0);
            const int ry = ry0 + p.ky, r0 = p.r[0] >= 0 ? p.r[0] : p.r[1];
            const float kx = (float)E.h_kvec[3 * E.h_runs[r0].kbeg], ky = std::fabs((float)E.h_kvec[3 * E.h_runs[r0].kbeg + 1]);
            pr[c * rp + q] = make_int4(p.kx * 128 | ((p.kx & 7) << 4) << 16, ry * 128 | ((ry & 7) << 4) << 16, bits(kx), bits(ky));
            for (int j = 0; j < p.jm; j++) {
                int k[4] = {-1, -1, -1, -1};
                for (int s = 0; s < 2; s++) {
                    if (p.r[s] < 0) continue;
                    const KRun &run = E.h_runs[p.r[s]];
                    if (j >= run.kzlo && j < run.kzlo + run.nkz) k[2 * s] = run.kbeg + j - run.kzlo;
                    if (j > 0 && -j >= run.kzlo && -j < run.kzlo + run.nkz) k[2 * s + 1] = run.kbeg - j - run.kzlo;
                }
                ki[((size_t)c * rp + q) * 4 * kcm + j] = make_int4(k[0], k[1], k[2], k[3]);
            }
        }
        words += 2 * NC * rp * kc;
    }
    const size_t n[4] = {sizeof(int4) * pr.size(), sizeof(int2) * chunk.size(), sizeof(int4) * ki.size(), 16 * (size_t)words * kp.P};
    const void *src[3] = {pr.data(), chunk.data(), ki.data()};
    void *d[4] = {nullptr, nullptr, nullptr, nullptr};
    for (int i = 0; i < 4; i++) {
        if (cudaMalloc(&d[i], n[i]) != cudaSuccess) {
            cudaGetLastError();
            for (int q = 0; q < i; q++) cudaFree(d[q]);
            return false;
        }
    }
    for (int i = 0; i < 4; i++) {
        E.allocs.push_back(d[i]);
        if (i < 3) cudaMemcpy(d[i], src[i], n[i], cudaMemcpyHostToDevice);
    }
    cudaMemset(d[3], 0, n[3]);  // (rows past a pair's |kz| stay zero)
    if (place) *place = where;
    T.pair = reinterpret_cast<const int4 *>(d[0]);
    T.chunk = reinterpret_cast<const int2 *>(d[1]);
    T.kidx = reinterpret_cast<const int4 *>(d[2]);
    T.V = d[3];
    T.vstride = words;
    T.nchunk = nch;
    T.rp = rp;
    T.kcm = kcm;
    return true;
}

// Which boxes take the tensor-core passes. Their operands hold 22 bits and an accumulator cuts off what is below
// its last place; the FP32-pipe passes round, and add the sums of a tile in FP64. So the tensor-core passes are the
// faster ones and not the more accurate ones, and they take the boxes where groups of TC_BOXRUN runs (256 of at
// most 10 |kz|), the epilogue over them, and for the field the tables of 128 sites (128 rows at most), Q and the rows of 8
// runs, leave room in a CTA's shared memory: cubes of |n| from 4 to 41 (but 30), up to 85 A at a 9 A cutoff.
// Smaller groups and the tables in two parts would reach further, but there the FP32 passes stay. RMS error of the
// gradient and the induced dipoles against the FP64 engine, and a force call (tensor cores; FP32): 512 x 2,
// |n| <= 45: 1.5e-6 1.9e-5 7.5 ms; 3.5e-7 4.7e-6 19.9 ms. 512 x 8, 25 x 25 x 199 A: 4.7e-7 1.3e-5 19.9 ms; 1.6e-7
// 3.9e-6 38.6 ms. 8 x 1, |n| <= 30: 1.9e-6 1.7e-6 2.1 ms; 1.3e-6 1.7e-6 4.6 ms.
constexpr int TC_BOXRUN = 224;
static bool sfac_box(const KP &kp, const std::vector<int2> &src, const std::vector<int> &jr, const std::vector<KRun> &runs, int dmax,
                     int band, int parts) {  // parts: partial sums a k-vector
    int ncol = 16, nkl = 0;
    const int n = (int)src.size();
    for (int p0 = 0; p0 < n;) {
        const int most = std::min(band, jr[src[p0].x] - src[p0].y) <= 10 ? TC_MAXRUN : TC_BOXRUN;
        int nr = 0, k = 0;
        for (; p0 + nr < n && nr < most && src[p0 + nr].y == src[p0].y; nr++) k += runs[src[p0 + nr].x].nkz;
        ncol = std::max(ncol, (2 * nr + 15) / 16 * 16);
        nkl = std::max(nkl, k);
        p0 += nr;
    }
    int nabuf = TC_NABUF_MAX;
    while (nabuf > 2 && TcSmem(kp.ntab, ncol, nabuf).total > dmax) nabuf--;
    const int total = TcSmem(kp.ntab, ncol, nabuf).total;
    return total <= dmax && 128 * TC_LD * 4 + 8 * parts * nkl <= total - 1024;
}
static bool field_box(const KP &kp, int nc) {  // nc: rows of a run pair
    const int boxb = (kp.ntab * 128 + 1023) / 1024 * 1024, kq = (2 * kp.lmax + 17) / 16 * 16;
    return kp.ntab <= 128 && 8 * boxb + 4 * TF_SITES * kq + 16 * nc * kq + 1024 <= 220 * 1024;
}

static void tp_setup(Engine &E, PFN_cuTensorMapEncodeTiled_v12000 enc, const std::vector<int> &jr, std::vector<int4> *place) {
    KP &kp = E.kp;
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, E.device);
    const void *fk[5] = {(const void *)k_field_p<TF_Q>, (const void *)k_field_p<TF_D>, (const void *)k_field_p<TF_QG>,
                         (const void *)k_field_p<TF_DG>, (const void *)k_field_p<TF_DE>};
    size_t fstat = 0;
    for (const void *f : fk) {
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, f) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        fstat = std::max(fstat, fa.sharedSizeBytes);
    }
    const int dmax = optin - (int)fstat;
    for (const void *f : fk)
        if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, dmax) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
    // the ex and ey rows, and the ez rows, of 16 sites
    const cuuint64_t dims[2] = {(cuuint64_t)2 * kp.S, (cuuint64_t)kp.P * kp.ntab};
    const cuuint64_t strides[1] = {(cuuint64_t)kp.S * 8};
    const cuuint32_t es[2] = {1, 1};
    for (int z = 0; z < 2; z++) {
        const cuuint32_t box[2] = {32, (cuuint32_t)(z ? kp.lmax + 1 : kp.hmax + kp.kmax + 2)};
        if (box[1] > 256 || enc(reinterpret_cast<CUtensorMap *>(z ? E.tp_mapz : E.tp_mapxy), CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, kp.tabf,
                                dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return;
    }
    if (field_box(kp, 8) && tp_init(E, 0, jr, dmax, place) && field_box(kp, 12)) tp_init(E, 1, jr, dmax, nullptr);
}

void tc_init(Engine &E) {
    E.tc_ready = false;
    KP &kp = E.kp;
    if (E.precision != PIMD_MIXED || kp.ld <= kp.fd || !kp.tabf || !kp.dipf || !kp.Wf) return;
    // TMA rules: row pitch S x 8 bytes a multiple of 16, box rows <= 256; kz table <= 256
    if ((kp.S & 1) || kp.ntab > 256 || 2 * kp.lmax + 1 > 256) return;
    int major = 0;
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, E.device);
    if (major != 10) return;
    PFN_cuTensorMapEncodeTiled_v12000 enc = encode_fn();
    if (!enc) return;
    // the FP32 k_z of a k-vector depends on kz alone
    std::vector<float> kzv(2 * kp.lmax + 1, 0.f);
    std::vector<int> kzseen(2 * kp.lmax + 1, 0);
    for (int r = 0; r < kp.nrun; r++) {
        const KRun &run = E.h_runs[r];
        for (int j = 0; j < run.nkz; j++) {
            const int kz = run.kzlo + j, k = run.kbeg + j;
            const float v = (float)E.h_kvec[3 * k + 2];
            if (kzseen[kz + kp.lmax] && kzv[kz + kp.lmax] != v) return;
            kzseen[kz + kp.lmax] = 1;
            kzv[kz + kp.lmax] = v;
        }
    }
    // runs sorted by their largest |kz| (longest first), groups of <= 256 runs, 6 (max |kz| + 1)
    // Z rows per group <= 128
    std::vector<int> order(kp.nrun), jr(kp.nrun);
    for (int r = 0; r < kp.nrun; r++) {
        const KRun &run = E.h_runs[r];
        jr[r] = std::max(std::abs(run.kzlo), std::abs(run.kzlo + run.nkz - 1)) + 1;
        order[r] = r;
    }
    // ... the runs (kx, +-ky) of a pair side by side
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
        const KRun &a = E.h_runs[x], &c = E.h_runs[y];
        return std::make_tuple(-jr[x], a.kx, std::abs(a.ky)) < std::make_tuple(-jr[y], c.kx, std::abs(c.ky));
    });
    auto paired = [&](int x, int y) {
        const KRun &a = E.h_runs[x], &c = E.h_runs[y];
        return a.kx == c.kx && a.ky == -c.ky;
    };
    // slots: every run once with its |kz| rows below TC_JB, then the runs reaching beyond once
    // per further band of TC_JB rows (j0 = TC_JB, 2 TC_JB, ...), each band in groups of <= 256
    // slots; a slot's k-vectors outside its group's rows are local entries with k = -1
    constexpr int TC_JB = 21;  // 6 TC_JB <= 128 Z rows
    std::vector<int2> src;     // (run, j0)
    for (int q = 0; q < kp.nrun; q++) src.push_back(make_int2(order[q], 0));
    for (int j0 = TC_JB;; j0 += TC_JB) {
        const size_t n0 = src.size();
        for (int q = 0; q < kp.nrun; q++)
            if (jr[order[q]] > j0) src.push_back(make_int2(order[q], j0));
        if (src.size() == n0) break;
    }
    const int nslot = (int)src.size();
    // dynamic shared memory available: the opt-in limit minus the kernel's static part
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, E.device);
    cudaFuncAttributes fa, fq, fd;
    if (cudaFuncGetAttributes(&fa, k_sfac_tc<TC_OP_MU>) != cudaSuccess ||
        cudaFuncGetAttributes(&fq, k_sfac_tc<TC_OP_Q>) != cudaSuccess ||
        cudaFuncGetAttributes(&fd, k_sfac_tc<TC_OP_DIP>) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    const int dmax = optin - (int)std::max(fa.sharedSizeBytes, std::max(fq.sharedSizeBytes, fd.sharedSizeBytes));
    if (!sfac_box(kp, src, jr, E.h_runs, dmax, TC_JB, 1)) return;
    // the dipole-component sums of the virial (three partials a k-vector) likewise, cubes of |n| from 5 to 15. One
    // component after the other would fit the larger ones and take 481 us instead of 2945 at 4096 x 32, but its
    // sums over all sites of a bead are off by 2.5e-6 (rms, 700 sites) where the FP32 pass is within 4e-7, and the
    // virial of 4096 x 32 by 6.02e-6 instead of 5.95e-6
    E.tc_dip_ok = sfac_box(kp, src, jr, E.h_runs, dmax, TC_JB, 3);
    // the field passes' tables, and where their V has the rows of each run's pair (its offset, to the lo rows, |kz| rows)
    std::vector<int4> place;
    tp_setup(E, enc, jr, &place);
    E.tc_nsplit = 0;
    for (int p0 = 0; p0 < nslot;) {
        int n = 0;
        while (p0 + n < nslot && src[p0 + n].y == src[p0].y) n++;
        E.tc_nsplit += (n + TC_BOXRUN - 1) / TC_BOXRUN;
        p0 += n;
    }
    std::vector<int4> slots(nslot);
    std::vector<float2> skv(nslot);
    std::vector<TcGroup> groups;
    std::vector<TcKW> kloc;
    std::vector<int4> vp;
    std::vector<float2> runkf(kp.nrun);
    for (int r = 0; r < kp.nrun; r++)
        runkf[r] = make_float2((float)E.h_kvec[3 * E.h_runs[r].kbeg], (float)E.h_kvec[3 * E.h_runs[r].kbeg + 1]);
    // groups of at most 256 runs, or of fewer until the operand buffers (four to two) and the epilogue's staging
    // tile and partial S, which reuse the table and operand regions, fit
    int ncolmax = 0, nklmax = 0, nvalid = 0, nabuf = 0;
    auto build = [&](int maxrun) {  // false: does not fit
        groups.clear();
        kloc.clear();
        vp.clear();
        ncolmax = 16, nklmax = nvalid = 0;
        // groups of one band hold equally many runs: the bead's CTAs of all groups run side by side, and a last
        // group of one run (897 runs in groups of 224) would take a CTA's time for it
        for (int p0 = 0; p0 < nslot;) {
            const int j0 = src[p0].y, jmg = std::min(TC_JB, jr[src[p0].x] - j0);
            int left = 0;
            while (p0 + left < nslot && src[p0 + left].y == j0) left++;
            // (a pair stays in one group)
            const int ng = (left + maxrun - 2) / (maxrun - 1);
            int nr = (left + ng - 1) / ng;
            if (nr < left && paired(src[p0 + nr - 1].x, src[p0 + nr].x)) nr++;
            TcGroup g{p0, nr, 0, jmg, 0, (int)kloc.size(), j0, 0, (int)vp.size()};
            g.ncol = ((2 * g.nr + 15) / 16) * 16;
            for (int p = p0; p < p0 + g.nr; p++) {
                const int r = src[p].x;
                const KRun &run = E.h_runs[r];
                slots[p] = make_int4(run.kx + 256 * (run.ky + 128), g.nkl, run.kzlo, run.nkz);
                skv[p] = runkf[r];
                for (int j = 0; j < run.nkz; j++) {
                    const int akz = std::abs(run.kzlo + j);
                    const bool mine = akz >= j0 && akz < j0 + g.jm;
                    nvalid += mine;
                    kloc.push_back(TcKW{mine ? run.kbeg + j : -1, (float)(FOURPI * E.h_Ak[run.kbeg + j] / kp.volume)});
                }
                g.nkl += run.nkz;
                const int4 at = place.empty() ? make_int4(0, 0, 0, 0) : place[r];
                const int q = p - p0, ip = run.ky < 0 ? 0xffff : q, im = run.ky < 0 ? q : 0xffff;
                if (q > 0 && paired(src[p - 1].x, r) && run.ky != 0) {  // the pair's second run
                    int4 &v = vp.back();
                    v.x = run.ky < 0 ? (v.x & 0xffff) | im << 16 : ip | (v.x & ~0xffff);
                } else {
                    vp.push_back(make_int4(ip | im << 16, at.x, at.y, at.z));
                }
            }
            g.np = (int)vp.size() - g.vp0;
            groups.push_back(g);
            ncolmax = std::max(ncolmax, g.ncol);
            nklmax = std::max(nklmax, g.nkl);
            p0 += nr;
        }
        nabuf = TC_NABUF_MAX;
        while (nabuf > 2 && TcSmem(kp.ntab, ncolmax, nabuf).total > dmax) nabuf--;
        const int total = TcSmem(kp.ntab, ncolmax, nabuf).total;
        return total <= dmax && 128 * TC_LD * 4 + 8 * (E.tc_dip_ok ? 3 : 1) * nklmax <= total - 1024;
    };
    int maxrun = TC_MAXRUN;
    while (maxrun >= 32 && !build(maxrun)) maxrun -= 32;
    if (maxrun < 32) return;
    if (nvalid != kp.nk) return;  // every k-vector in exactly one group
    const TcSmem L(kp.ntab, ncolmax, nabuf);
    if (cudaFuncSetAttribute(k_sfac_tc<TC_OP_MU>, cudaFuncAttributeMaxDynamicSharedMemorySize, dmax) != cudaSuccess ||
        cudaFuncSetAttribute(k_sfac_tc<TC_OP_Q>, cudaFuncAttributeMaxDynamicSharedMemorySize, dmax) != cudaSuccess ||
        cudaFuncSetAttribute(k_sfac_tc<TC_OP_DIP>, cudaFuncAttributeMaxDynamicSharedMemorySize, dmax) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    int4 *d_slots = nullptr;
    float2 *d_skv = nullptr;
    TcGroup *d_groups = nullptr;
    TcKW *d_kloc = nullptr;
    float *d_kzv = nullptr;
    int4 *d_vp = nullptr;
    if (cudaMalloc((void **)&d_slots, sizeof(int4) * slots.size()) != cudaSuccess ||
        cudaMalloc((void **)&d_skv, sizeof(float2) * skv.size()) != cudaSuccess ||
        cudaMalloc((void **)&d_groups, sizeof(TcGroup) * groups.size()) != cudaSuccess ||
        cudaMalloc((void **)&d_kloc, sizeof(TcKW) * kloc.size()) != cudaSuccess ||
        cudaMalloc((void **)&d_vp, sizeof(int4) * vp.size()) != cudaSuccess ||
        cudaMalloc((void **)&d_kzv, sizeof(float) * kzv.size()) != cudaSuccess) {
        cudaGetLastError();
        for (void *p : {(void *)d_slots, (void *)d_skv, (void *)d_groups, (void *)d_kloc, (void *)d_kzv, (void *)d_vp})
            if (p) cudaFree(p);
        return;
    }
    for (void *p : {(void *)d_slots, (void *)d_skv, (void *)d_groups, (void *)d_kloc, (void *)d_kzv, (void *)d_vp}) E.allocs.push_back(p);
    cudaMemcpy(d_slots, slots.data(), sizeof(int4) * slots.size(), cudaMemcpyHostToDevice);
    cudaMemcpy(d_skv, skv.data(), sizeof(float2) * skv.size(), cudaMemcpyHostToDevice);
    cudaMemcpy(d_groups, groups.data(), sizeof(TcGroup) * groups.size(), cudaMemcpyHostToDevice);
    cudaMemcpy(d_kloc, kloc.data(), sizeof(TcKW) * kloc.size(), cudaMemcpyHostToDevice);
    cudaMemcpy(d_kzv, kzv.data(), sizeof(float) * kzv.size(), cudaMemcpyHostToDevice);
    cudaMemcpy(d_vp, vp.data(), sizeof(int4) * vp.size(), cudaMemcpyHostToDevice);
    // tables [P][ntab][S] float2 as a 2-D FP32 tensor (x = 2 S values, y = P ntab rows); a box
    // is 16 sites (128 bytes) x ntab rows, written to shared memory with the 128-byte swizzle
    CUtensorMap *map = reinterpret_cast<CUtensorMap *>(E.tc_map);
    const cuuint64_t dims[2] = {(cuuint64_t)2 * kp.S, (cuuint64_t)kp.P * kp.ntab};
    const cuuint64_t strides[1] = {(cuuint64_t)kp.S * 8};
    const cuuint32_t box[2] = {32, (cuuint32_t)kp.ntab};
    const cuuint32_t es[2] = {1, 1};
    if (enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, kp.tabf, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return;
    E.d_tcslot = d_slots;
    E.d_tcskv = d_skv;
    E.d_tcgrp = d_groups;
    E.d_tckloc = d_kloc;
    E.d_tckzv = d_kzv;
    E.d_tcvp = d_vp;
    // X-operand cache of the dipole sites (k_sfac_tc, TC_OP_MU): per bead and run group, one
    // block per 16 sites from the first site group's base, hi and lo rows [0, 2 nr) rounded to
    // 8-row groups; zero-filled once (the padding rows are never written)
    E.d_tcx = nullptr;
    if (kp.ld > kp.fd) {
        int xb = 0;
        for (const TcGroup &g : groups) xb = std::max(xb, ((2 * g.nr + 7) / 8) * 256);
        const int sbase = kp.fd & ~(TC_SS - 1);
        const int xsub = (kp.ld - sbase + TC_SS - 1) / TC_SS * (TC_SS / TC_KS);  // whole table stages
        const size_t bytes = (size_t)kp.P * groups.size() * xsub * 2 * xb;
        void *d_x = nullptr;
        if (cudaMalloc(&d_x, bytes) == cudaSuccess) {
            E.allocs.push_back(d_x);
            cudaMemset(d_x, 0, bytes);
            E.d_tcx = d_x;
            E.tc_xsub = xsub;
            E.tc_xblock = 2 * xb;
        } else {
            cudaGetLastError();
        }
    }
    E.tc_ntg = (int)groups.size();
    E.tc_nband = (int)std::count_if(groups.begin(), groups.end(), [](const TcGroup &g) { return g.j0 > 0; });
    E.tc_ncolmax = ncolmax;
    E.tc_nabuf = nabuf;
    E.tc_ready = true;
    E.tf_ready = E.tp[0].V != nullptr;
    E.tf_qd_ready = E.tf_ready && E.tp[1].V != nullptr;
}

// whether the iterations' field pass is launched as a programmatic dependent (griddepcontrol.wait
// before it reads the iteration's fields)
bool field_pdl_ok(const Engine &E) {
    return E.tc_ready && E.tf_ready && E.ff_tc && E.tc_pdl && E.sf_tc;
}

// One of the prepared passes (k_field_v, then k_field_p).
template <int MODE>
static void launch_field_p(Engine &E, int s0, int s1) {
    const KP &kp = E.kp;
    constexpr bool DG = MODE == TF_DG || MODE == TF_DE;
    const Engine::TpSet &T = E.tp[DG ? 1 : 0];
    TpArgs a;
    a.pair = T.pair;
    a.chunk = T.chunk;
    a.kidx = T.kidx;
    a.kzv = E.d_tckzv;
    a.V = reinterpret_cast<uint4 *>(T.V);
    a.vstride = T.vstride;
    a.nchunk = T.nchunk;
    a.rp = T.rp;
    a.kcm = T.kcm;
    a.sbase = s0 & ~(TC_SS - 1);  // TMA x coordinates 2 (sbase + 16 i): 128-byte aligned
    a.s_lo = s0;
    a.s_hi = s1;
    a.skipconv = MODE == TF_D ? 1 : 0;
    a.pdl = E.tc_pdl ? 1 : 0;
    const int slot = (MODE == TF_D || MODE == TF_QG) ? 1 : 0;
    const TpSmem L(kp.hmax + kp.kmax + 2, kp.lmax + 1, T.kcm, (DG ? 12 : 8) * T.rp);
    const CUtensorMap *xy = reinterpret_cast<const CUtensorMap *>(E.tp_mapxy), *z = reinterpret_cast<const CUtensorMap *>(E.tp_mapz);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cv = {}, cf = {};
    cv.gridDim = dim3(T.nchunk, kp.P);
    cv.blockDim = dim3(TP_VT);
    cf.gridDim = dim3((s1 - a.sbase + TF_SITES - 1) / TF_SITES, kp.P);
    cf.blockDim = dim3(TP_NT);
    cf.dynamicSmemBytes = L.total;
    // V where the structure factor has not written it, and the field pass, each as a programmatic dependent of
    // the kernel before it
    auto run = [&](cudaLaunchConfig_t &cfg, auto &&launch) {
        cfg.stream = E.stream;
        cfg.attrs = at;
        cfg.numAttrs = a.pdl;
        if (launch() == cudaSuccess || !a.pdl) return;
        cudaGetLastError();
        a.pdl = 0;
        cfg.numAttrs = 0;
        E.tc_pdl = false;  // not available: plain launches from now on
        if (E.field_needs_join) cudaStreamWaitEvent(E.stream, E.loop_join, 0);
        launch();
    };
    if (DG || E.tp_vslot != slot) {
        run(cv, [&] { return cudaLaunchKernelEx(&cv, k_field_v<DG>, kp, a, slot); });
        if (!DG) E.tp_vslot = slot;
        ++E.nlaunch;
    }
    run(cf, [&] { return cudaLaunchKernelEx(&cf, k_field_p<MODE>, *xy, *z, kp, a); });
    ++E.nlaunch;
}

// mode TF_D: dipole field, SOR update and convergence test of one iteration at the dipole sites
// [s0, s1) (k_field_f<F_D> + k_field_finish<F_D>); TF_Q: charge field and potential added to F at
// [s0, s1) (k_field_f<F_Q> + k_field_finish<F_Q>); TF_QG, TF_DG: the halves of the force pass
// (launch_field_qd_tc). 1 when launched, else 0.
int launch_field_tc(Engine &E, int mode, int s0, int s1) {
    if (!E.tc_ready || !E.tf_ready || !E.ff_tc || s1 <= s0 || (mode >= TF_DG && !E.tf_qd_ready)) return 0;
    if (mode == TF_D)
        launch_field_p<TF_D>(E, s0, s1);
    else if (mode == TF_Q)
        launch_field_p<TF_Q>(E, s0, s1);
    else if (mode == TF_QG)
        launch_field_p<TF_QG>(E, s0, s1);
    else if (mode == TF_DG)
        launch_field_p<TF_DG>(E, s0, s1);
    else
        launch_field_p<TF_DE>(E, s0, s1);
    return 1;
}

// The differentiation form's reverse sweep on the mixed engine: the dipole force of kp.dipf from the two weight
// slots (TF_DG: into kp.dR, or kp.Fx with fx_mode 2) at [fd, ld); with field, also the field of those weights
// into kp.Fx (TF_DE; a pass of its own took 13 us a sweep at 512 x 32). 1 when launched, else 0.
int launch_adj_dforce_tc(Engine &E, bool field) {
    if (!E.tf_qd_ready || E.kp.ld <= E.kp.fd) return 0;
    return launch_field_tc(E, field ? TF_DE : TF_DG, E.kp.fd, E.kp.ld);
}
// the charge half of the force pass (TF_QG: -q E and phi of the dipole slot's weights) at the
// charged sites from N on (TTM3-F: H1, H2, M), into kp.Fx with fx_mode 2
int launch_adj_qforce_tc(Engine &E) {
    if (!E.tf_qd_ready) return 0;
    return launch_field_tc(E, TF_QG, E.kp.N, E.kp.S);
}

// ewald_std_qd's force pass (k_field_f<F_QD> + k_field_finish<F_QD>) as two tensor-core passes:
// the charge force -q E and potential from the dipole structure factor at [s0, s1), then the
// dipole force at the dipole sites from the total structure factor. 1 when launched, else 0.
int launch_field_qd_tc(Engine &E, int s0, int s1) {
    if (!E.tc_ready || !E.tf_ready || !E.tf_qd_ready || !E.ff_tc || s1 <= s0) return 0;
    launch_field_tc(E, TF_QG, s0, s1);
    if (E.kp.ld > E.kp.fd) launch_field_tc(E, TF_DG, E.kp.fd, E.kp.ld);
    return 1;
}

// Returns 1 when the launch wrote the structure factor of `op` (Sq and the charge weights, Sm
// and the dipole weights, or Sdip; no k_sreduce needed), else 0.
int launch_sfac_tc(Engine &E, int op, int s0, int nsites, int skipconv) {
    if (!E.tc_ready || !E.sf_tc || nsites <= 0 || (op == TC_OP_DIP && !E.tc_dip_ok)) return 0;
    const KP &kp = E.kp;
    TcArgs a;
    a.slot = E.d_tcslot;
    a.skv = E.d_tcskv;
    a.grp = reinterpret_cast<const TcGroup *>(E.d_tcgrp);
    a.kw = reinterpret_cast<const TcKW *>(E.d_tckloc);
    a.kzv = E.d_tckzv;
    a.sbase = s0 & ~(TC_SS - 1);  // TMA x coordinate 2 sbase: 256-byte aligned
    a.s_lo = s0;
    a.s_hi = s0 + nsites;
    a.ncolmax = E.tc_ncolmax;
    a.nabuf = E.tc_nabuf;
    a.skipconv = skipconv;
    // the iterations' dipole structure factor caches X (its site range is the cached one)
    const bool xok = op == TC_OP_MU && E.d_tcx && E.tc_xcache && s0 == kp.fd && nsites == kp.ld - kp.fd;
    a.xcache = xok ? reinterpret_cast<uint4 *>(E.d_tcx) : nullptr;
    a.xsub = E.tc_xsub;
    a.xblock = E.tc_xblock;
    a.xkeep = E.l2_keep ? 1 : 0;
    a.vp = E.d_tcvp;
    a.V = reinterpret_cast<uint4 *>(E.tp[0].V);
    a.vstride = E.tp[0].vstride;
    // the iterations' structure factor follows the previous iteration's field pass on the stream
    // (or the charge passes, which need no overlap): its CTAs are scheduled as that grid drains
    a.pdl = (op == TC_OP_MU && skipconv && E.tc_pdl && E.tf_ready && E.ff_tc) ? 1 : 0;
    // one CTA per SM (shared memory); site groups (= cluster size) so that one wave fills the GPU if the runs were in
    // groups of TC_BOXRUN. The launch's own groups may be larger; the site groups stay those, since their number sets
    // how many sites an accumulator, which cuts off, adds up, and with it the result: 4096 x 32 has one group, and its
    // dipoles are off by 4.4e-5 (rms, against the FP64 engine); in four groups, by the waves of the launch's own run
    // groups, they move by 4e-5
    const int nst = (a.s_hi - a.sbase + TC_SS - 1) / TC_SS;
    int ng = std::max(1, std::min((int)std::max(1L, E.nsm / ((long)E.tc_nsplit * kp.P)), std::min(nst, TC_CLMAX)));
    const int spg = (nst + ng - 1) / ng;
    ng = (nst + spg - 1) / spg;
    a.ntg = E.tc_ntg;
    // the highest stream priority: the mixed engine's real-space dipole field runs beside this
    // kernel on a second stream and must not hold the SMs its clusters wait for
    static int prio_cache[64] = {0}, prio_set[64] = {0};
    if (!prio_set[E.device & 63]) {
        int least = 0, greatest = 0;
        if (cudaDeviceGetStreamPriorityRange(&least, &greatest) == cudaSuccess) prio_cache[E.device & 63] = greatest;
        prio_set[E.device & 63] = 1;
    }
    const TcSmem L(kp.ntab, a.ncolmax, a.nabuf);
    const CUtensorMap *map = reinterpret_cast<const CUtensorMap *>(E.tc_map);
    // run groups [tg0, tg1) with clusters of n site groups of sp stages; pdl as in TcArgs
    auto launch = [&](int tg0, int tg1, int n, int sp, int pdl, bool pev) {
        a.tg0 = tg0;
        a.tsg = sp * TC_SS;
        a.pdl = pdl;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(n, tg1 - tg0, kp.P);
        cfg.blockDim = dim3(TC_NT);
        cfg.dynamicSmemBytes = L.total;
        cfg.stream = E.stream;
        cudaLaunchAttribute at[4];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = n;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        at[1].id = cudaLaunchAttributePriority;
        at[1].val.priority = prio_cache[E.device & 63];
        int na = 2;
        if (pdl) {
            at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at[na].val.programmaticStreamSerializationAllowed = 1;
            na++;
        }
        // the caller's programmatic event: recorded once every CTA has passed its set-up
        // (griddepcontrol.launch_dependents) or left
        if (pev) {
            at[na].id = cudaLaunchAttributeProgrammaticEvent;
            at[na].val.programmaticEvent.event = E.loop_pev;
            at[na].val.programmaticEvent.flags = 0;
            at[na].val.programmaticEvent.triggerAtBlockStart = 0;
            na++;
        }
        cfg.attrs = at;
        cfg.numAttrs = na;
        auto run = [&] {
            return op == TC_OP_MU ? cudaLaunchKernelEx(&cfg, k_sfac_tc<TC_OP_MU>, *map, kp, a)
                   : op == TC_OP_Q ? cudaLaunchKernelEx(&cfg, k_sfac_tc<TC_OP_Q>, *map, kp, a)
                                   : cudaLaunchKernelEx(&cfg, k_sfac_tc<TC_OP_DIP>, *map, kp, a);
        };
        cudaError_t e = run();
        if (e == cudaSuccess && pev) E.sfac_pev_armed = true;
        if (e != cudaSuccess && na > 2) {  // an attribute refused: a plain cluster launch
            cudaGetLastError();
            a.pdl = 0;
            cfg.numAttrs = 2;
            e = run();
        }
        if (e == cudaSuccess) ++E.nlaunch;
        return e;
    };
    // Boxes whose CTAs are more than one wave: the band groups (a quarter of the Z rows or less, but a CTA's whole
    // time) go first, in clusters of four site groups, and the others start beside them, so that the last wave is
    // not one of a few whole CTAs (4096 x 32: 160 on 152 SMs, 398 us an iteration; 275 so). Their k-vectors have |kz| > 20 and weights of 1e-6
    // of the largest, so that their shorter sums leave the dipoles as they are.
    const int main_groups = E.tc_ntg - E.tc_nband;
    const bool split = E.tc_nband > 0 && main_groups > 0 && E.tc_pdl && (long)E.tc_ntg * kp.P > E.nsm;
    const bool pev = E.sfac_pev_req && op == TC_OP_MU && E.loop_pev;
    const int first = a.pdl;
    cudaError_t e = cudaSuccess;
    if (split) {
        const int nb4 = std::min(4, nst), sp4 = (nst + nb4 - 1) / nb4;
        e = launch(main_groups, E.tc_ntg, (nst + sp4 - 1) / sp4, sp4, first, false);
    }
    if (e == cudaSuccess) e = launch(0, split ? main_groups : E.tc_ntg, ng, spg, split ? 2 : first, pev);
    if (e != cudaSuccess) {
        cudaGetLastError();
        E.sf_tc = false;  // e.g. no room for the cluster: the FP32-pipe kernel from now on
        return 0;
    }
    if (op != TC_OP_DIP && a.V) E.tp_vslot = op == TC_OP_MU ? 1 : 0;
    return 1;
}

}  // namespace pimd
