// Rate coefficients and species source terms, FP64 (the drop-in form).
//
// One CTA of 16 warps works on tiles of 32 cells (lane = cell), looping over
// tiles persistently; the rate coefficients of a tile stay in shared memory and
// go to HBM only where the species update asks for them:
//   phase 0  Y[52][32], T, rho, soot of the tile (coalesced rows; the next tile's rows
//            are loaded while this one's rates are formed)
//   phase 1  G_k = exp(Gibbs) and 1 / G_k; the third bodies as weighted sums of Y
//            (src/lib/ckrates.f:103-115, 643-731)
//   phase 2  per reaction pair: k_f, k_r = k_f/Kc, fall-off blend, RC
//            (warp-uniform pair -> no divergence); soot sources
//            (ckrates.f:95-101, 116-642, 740-1352)
//   phase 3  the species' gain and loss sums, straight-line code per warp (generated/omega_program.cuh)
//   phase 4  per species: QDSP, d(omega)/dY, heat release; QDOT (src/lib/solveh.f:116-1142)
// The tables of the pairs (Arrhenius, fall-off, Kc formula, RC assembly) are staged into
// shared memory once per CTA by a bulk (TMA) copy, prepared so that a pair has no division
// (one exponential and about 25 multiplications for most) and nothing is decoded per cell: the
// factors of 1/Kc and of the assembly are rows of the tile's shared memory.
//
// What bounds it: the FP64 pipe and the latency of short phases between barriers. Measured at 1,048,576
// cells with RC written: 32.2 ms before the tables were prepared this way and the sums were generated code
// (88 % of 433,000 warp instructions per tile were table look-ups and divisions), 6.7 ms now (the RC plane
// and the outputs alone take 0.9 ms of HBM time); one tile alone 150 and 33 us.
#pragma once
#include "uc_device.cuh"
#include "generated/omega_program.cuh"

namespace uc {

// per-cell scalar rows of the tile (shared memory); row 0 also stands for "none" in the pair table
enum { SC_TK = 0, SC_TKD, SC_LNT, SC_RHO, SC_RUT, SC_DMOLEA, SC_TB0, SC_STMF = SC_TB0 + 11, SC_STND,
       SC_IT, SC_RHO2, SC_RHO3, SC_IRUT, SC_N };

struct ChemArgs {
    const DevParams *P;
    const PairTab *tab;          // [NPAIR] in global memory
    const double *tk, *rho, *y, *stmf, *stnd;   // y: [52][npad]
    double *rc;                  // [544][npad] or null
    double *sour;                // [6][npad] or null
    double *qdsp, *qdot, *dwdy;  // outputs (any may be null)
    int n, npad, ntile;
    int *status;
    const int *tile_list;        // optional: only these tiles ([*tile_count] entries)
    const int *tile_count;
    // optional ISKIP class per cell (0: computed; 1: 3 <= ISKIP < 10; 2: ISKIP >= 10). Classes 1 and 2
    // keep their RC and SOUR (ckrates.f:94); class 2 keeps its omega, QDOT and d(omega)/dY too
    // (solveh.f:119), class 1 takes them from its kept RC (rc_stale, zero when null).
    const int8_t *skip;
    const double *rc_stale;
};

constexpr int CHEM_POLY = LSP * 14;               // the NASA coefficients, staged into shared memory
constexpr size_t CHEM_SMEM = PAIRTAB_BYTES + sizeof(double) * (size_t)(LRX * TILE + 3 * LSP * TILE + SC_N * TILE +
                                                                      CHEM_POLY + CHEM_WARPS * TILE) + 64;
static_assert(CHEM_SMEM <= 232448, "a tile of the rate kernel does not fit in shared memory");
static_assert(UC_OM_WARPS == CHEM_WARPS, "the generated sums are shared out over the kernel's warps");

// The scalar rows of a tile (one warp).
__device__ __forceinline__ void tile_scalars(const DevParams &P, double *sC, int lane, double tk, double rho,
                                             double stmf, double stnd)
{
    const double TKD = tk * P.TSTR, RUT = (double)82.06f * TKD;
    sC[SC_TK * TILE + lane] = tk;
    sC[SC_TKD * TILE + lane] = TKD;
    sC[SC_LNT * TILE + lane] = log(TKD);
    sC[SC_IT * TILE + lane] = 1.0 / TKD;
    sC[SC_RUT * TILE + lane] = RUT;
    sC[SC_IRUT * TILE + lane] = 1.0 / RUT;
    sC[SC_RHO * TILE + lane] = rho;
    sC[SC_RHO2 * TILE + lane] = rho * rho;
    sC[SC_RHO3 * TILE + lane] = rho * rho * rho;
    sC[SC_DMOLEA * TILE + lane] = rho * P.RSTR / P.WMSTR * 1.0e-06;
    sC[SC_STMF * TILE + lane] = stmf;
    sC[SC_STND * TILE + lane] = stnd;
}

// The soot sources (ckrates.f:1337-1352).
__device__ __forceinline__ void soot_sources(const DevParams &P, const double *sC, double *sour, size_t sstride,
                                             size_t soff, int lane)
{
    const double C1ST = P.C1ST;
    const double PI = 3.1415927e+00, RSOOT = 1.9000e+03, SIGB = 1.38e-23, AVNO = 6.0232e+23;
    const double CMIN = (double)100.0f, CAGL = (double)9.0f;
    const double TKD = sC[SC_TKD * TILE + lane], rho = sC[SC_RHO * TILE + lane];
    const double stmf = sC[SC_STMF * TILE + lane], stnd = sC[SC_STND * TILE + lane];
    const double TBODY = sC[SC_TB0 * TILE + lane];
    double DPST = 0.0;
    if (stnd >= 1.0) DPST = pow(6.0 * stmf / (PI * RSOOT * stnd), (double)0.333333f);
    const double ASST = PI * DPST * DPST * P.RSTR * rho * stnd;
    const double SOURNU = C1ST * rho * 1.000e+04 * exp(-(2.0632e+04 / TKD)) / P.WM[21];
    sour[soff] = SOURNU + C1ST * rho * ASST * 3.468e+03 * exp(-(1.2077e+04 / TKD)) / P.WM[21];
    sour[sstride + soff] = 2.0 * SOURNU * AVNO / CMIN / P.WMSTR;
    sour[2 * sstride + soff] = C1ST * rho * ASST * 1.000e+04 * pow(TKD, (double)0.5f) * exp(-(1.9626e+04 / TKD)) / P.WM[1];
    sour[3 * sstride + soff] = (double)0.13f * C1ST * ASST * 1.060e+02 * pow(TKD, (double)-0.5f) * exp(-(0.0 / TKD)) / P.WM[4] / TBODY;
    sour[4 * sstride + soff] = (double)0.5f * C1ST * ASST * 5.54e+00 * pow(TKD, (double)-0.5f) * exp(-(0.0 / TKD)) / P.WM[3] / TBODY;
    sour[5 * sstride + soff] = 2.0 * C1ST * P.RSTR * CAGL * sqrt(DPST * 6.0 * SIGB * TKD / RSOOT) * rho * rho * stnd;
}

// exp of the Gibbs function of a species, ckrates.f:103-115:
// exp(a1(lnT-1) + a2 T/2 + a3 T^2/6 + a4 T^3/12 + a5 T^4/20 - a6/T + a7)
__device__ __forceinline__ double gibbs_exp(const double *a, double ELOGT, double TKD, double IT)
{
    const double TKD1 = TKD * 0.5;
    const double TKD2 = TKD * TKD / 6.0;
    const double TKD3 = TKD1 * TKD2;
    const double TKD4 = (double)1.2f * TKD1 * TKD3;
    const double g0 = CO_FMA(a[4], TKD4, CO_FMA(a[3], TKD3, CO_FMA(a[2], TKD2, CO_FMA(a[1], TKD1, CO_MUL(a[0], ELOGT - 1.0)))));
    return exp(g0 - over_t(a[5], TKD, IT) + a[6]);
}

// Third bodies of the mixed form (tile_rates_mixed): TBODY from the Y/W rows left in sRC, the
// third-body groups TB001..TB010 and the soot sources (ckrates.f:643-731,
// 1337-1352). Ends with the barrier that publishes them.
template <int NW>
__device__ __forceinline__ void tile_tb_soot(const DevParams &P, const double *sRC, const double *sY, double *sC,
                                             double *sour, size_t sstride, size_t soff, int lane, int warp,
                                             bool keep_sour)
{
    // ---------------- phase 1b: TBODY (ordered sum)
    if (warp == 0) {
        double tb = sRC[lane];
        for (int k = 1; k < LSP; ++k) tb = tb + sRC[k * TILE + lane];
        sC[SC_TB0 * TILE + lane] = tb;
    }
    __syncthreads();
    // ---------------- phase 1c: third-body groups TB001..TB010; soot sources
    for (int j = (warp == 0 ? NW : warp); j <= 11; j += NW) {
        if (j <= 10) {
            const int g = j;
            double acc = sC[SC_TB0 * TILE + lane];
            const int o = P.tb_off[g];
            for (int t = 0; t < P.tb_len[g]; ++t) {
                const int k = P.tb_sp[o + t];
                const double yk = sY[k * TILE + lane];
                const double term = P.tb_hascoef[o + t] ? (P.tb_coef[o + t] * yk) / P.WM[k] : yk / P.WM[k];
                acc = P.tb_sign[o + t] > 0 ? acc + term : acc - term;
            }
            sC[(SC_TB0 + g) * TILE + lane] = acc;
        } else if (sour && !keep_sour) {
            // (skipped cells, ISKIP >= 3, keep theirs: ckrates.f:94)
            soot_sources(P, sC, sour, sstride, soff, lane);
        }
    }
    __syncthreads();
}

// The fall-off blend of a pair (ckrates.f:740-794; AKLOW < 0, the Tseng form, is not used by this data).
__device__ __forceinline__ double fall_off(const FallTab &T, const double *sC, int lane, double TKD, double IT,
                                           double ELOGT, double kf)
{
    const double DMOLE = CO_MUL(sC[T.dmole * TILE + lane], sC[SC_DMOLEA * TILE + lane]);
    const double AK0M = T.aklow * exp(CO_FMA(T.allow, ELOGT, -over_t(T.ealow, TKD, IT))) * DMOLE / (kf + 1.0e-20);
    double RFACT;
    if (T.troe[0] > 0.0) {
        double FCLOG;
        if (T.troe[1] == 0.0) FCLOG = log10(T.troe[0]);
        else FCLOG = log10(CO_FMA(T.troe[0], exp(-(TKD / T.troe[2])), CO_MUL(1.0 - T.troe[0], exp(-(TKD / T.troe[1])))) +
                           exp(-over_t(T.troe[3], TKD, IT)));
        const double CPLOG = log10(AK0M) - CO_FMA((double)0.67f, FCLOG, (double)0.4f);
        const double z = CPLOG / CO_FMA(-(double)0.14f, CPLOG, CO_FMA(-(double)1.27f, FCLOG, (double)0.75f));
        RFACT = pow(10.0, FCLOG / CO_FMA(z, z, 1.0));
    } else if (T.troe[0] == 0.0) {
        RFACT = 1.0;
    } else {
        const double l = log10(AK0M);
        const double XFACT = 1.0 / CO_FMA(l, l, 1.0);
        RFACT = pow(CO_FMA(-T.troe[0], exp(-over_t(T.troe[1], TKD, IT)), exp(-(TKD / T.troe[2]))), XFACT);
    }
    return (AK0M / (1.0 + AK0M)) * RFACT;
}

// Phases 1-2 of a tile: Gibbs functions, third bodies, soot sources and the rate coefficients, with NW warps
// (NW divides 16: a warp takes the pair lists of the virtual warps w, w+NW, ...). Expects the tile's Y rows in
// sY and its scalar rows in sC; writes the third bodies to sC, G_k and 1 / G_k to sG ([104][32]), the six soot
// sources to sour[m*sstride + soff] when sour is not null, and hands the two coefficients of pair p to
// out(p, rc0, rc1). Ends before the barrier that publishes what out stores. Rounded as written, so that the
// kernels that use it give a cell the same coefficients.
template <int NW, class Out>
__device__ __forceinline__ void tile_rates_fp64(const DevParams &P, const PairTab *sTab, const double *sPoly,
                                                const double *sY, double *sG, double *sC, double *sour,
                                                size_t sstride, size_t soff, int lane, int warp, bool keep_sour,
                                                Out out)
{
    const double TKD = sC[SC_TKD * TILE + lane], ELOGT = sC[SC_LNT * TILE + lane], IT = sC[SC_IT * TILE + lane];
    // ---------------- phase 1: Gibbs functions (52 items), third bodies (11 items)
    {
        const double *poly = sPoly + (TKD > UC_TPOL1 ? 7 : 0);
#pragma unroll 1
        for (int j = warp; j < LSP + 11; j += NW) {
            if (j < LSP) {
                const double g = gibbs_exp(poly + j * 14, ELOGT, TKD, IT);
                sG[j * TILE + lane] = g;
                sG[(LSP + j) * TILE + lane] = 1.0 / g;
            } else {
                const double *w = P.tbw + (j - LSP) * LSP;
                double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
                for (int k = 0; k < LSP; k += 4) {
                    s0 = CO_FMA(__ldg(w + k), sY[k * TILE + lane], s0);
                    s1 = CO_FMA(__ldg(w + k + 1), sY[(k + 1) * TILE + lane], s1);
                    s2 = CO_FMA(__ldg(w + k + 2), sY[(k + 2) * TILE + lane], s2);
                    s3 = CO_FMA(__ldg(w + k + 3), sY[(k + 3) * TILE + lane], s3);
                }
                sC[(SC_TB0 + j - LSP) * TILE + lane] = (s0 + s1) + (s2 + s3);
            }
        }
    }
    __syncthreads();
    // ---------------- phase 2: reaction pairs
    const FallTab *fall = reinterpret_cast<const FallTab *>(sTab + NPAIR);
#pragma unroll 1
    for (int vw = warp; vw < CHEM_WARPS; vw += NW) {
        if (vw == P.soot_warp && sour && !keep_sour) soot_sources(P, sC, sour, sstride, soff, lane);
        const int np = P.npair_of_warp[vw];
#pragma unroll 2
        for (int i = 0; i < np; ++i) {
            const int p = P.pair_of_warp[vw][i];
            const PairTab &T = sTab[p];
            double kf = CO_MUL(T.akf, exp(CO_FMA(T.alf, ELOGT, -over_t(T.exaf, TKD, IT))));
            double kr = 0.0;
            if (T.ng) {
                // 1/q, the factors of q and of its divisor in turn (every partial product is a normal number from 138 K
                // on; below 120 K the quotient in the source's order is none for other pairs)
                double iq = CO_MUL(CO_MUL(sG[T.g[0] * TILE + lane], sG[T.g[1] * TILE + lane]), sG[T.g[2] * TILE + lane]);
                for (int t = 3; t < T.ng; ++t) iq = CO_MUL(iq, sG[T.g[t] * TILE + lane]);
                kr = T.rut ? CO_MUL(CO_MUL(kf, sC[T.rut * TILE + lane]), iq) : CO_MUL(kf, iq);
            }
            if (T.fall) {
                const double AFP = fall_off(fall[T.fall - 1], sC, lane, TKD, IT, ELOGT, kf);
                kf = CO_MUL(AFP, kf);
                kr = CO_MUL(AFP, kr);
            }
            // RC assembly, ckrates.f:796-1333
            double rc0 = 0.0, rc1 = 0.0;
            if (T.r0) {
                rc0 = CO_MUL(CO_MUL(T.c0, sC[T.r0 * TILE + lane]), kf);
                if (T.t0) rc0 = CO_MUL(rc0, sC[T.t0 * TILE + lane]);
                if (T.y0 < LSP) rc0 = CO_MUL(rc0, sY[T.y0 * TILE + lane]);
            }
            if (T.r1) {
                rc1 = CO_MUL(CO_MUL(T.c1, sC[T.r1 * TILE + lane]), kr);
                if (T.t1) rc1 = CO_MUL(rc1, sC[T.t1 * TILE + lane]);
                if (T.y1 < LSP) rc1 = CO_MUL(rc1, sY[T.y1 * TILE + lane]);
            }
            out(p, rc0, rc1);
        }
    }
}

// The gain and loss sums of a warp's species (generated): P_k to row k and L_k to row 52 + k of sPL.
__device__ __forceinline__ void tile_omega_sums(const double2 *pr, const double *sY, double *sPL, int lane, int warp)
{
#define RCP(p) pr[(p) * TILE + lane]
#define YO(k) sY[(k) * TILE + lane]
#define OM_PUT(k, v) sPL[(k) * TILE + lane] = v
    switch (warp) {
    case 0: UC_OMEGA_0(); break;
    case 1: UC_OMEGA_1(); break;
    case 2: UC_OMEGA_2(); break;
    case 3: UC_OMEGA_3(); break;
    case 4: UC_OMEGA_4(); break;
    case 5: UC_OMEGA_5(); break;
    case 6: UC_OMEGA_6(); break;
    case 7: UC_OMEGA_7(); break;
    case 8: UC_OMEGA_8(); break;
    case 9: UC_OMEGA_9(); break;
    case 10: UC_OMEGA_10(); break;
    case 11: UC_OMEGA_11(); break;
    case 12: UC_OMEGA_12(); break;
    case 13: UC_OMEGA_13(); break;
    case 14: UC_OMEGA_14(); break;
    case 15: UC_OMEGA_15(); break;
    }
#undef RCP
#undef YO
#undef OM_PUT
}

__global__ void __launch_bounds__(CHEM_THREADS, 1) chem_fp64_kernel(const ChemArgs a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    PairTab *sTab = reinterpret_cast<PairTab *>(smem);
    double *sRC = reinterpret_cast<double *>(smem + PAIRTAB_BYTES);   // [272][32] pairs
    double *sY = sRC + LRX * TILE;                                    // [52][32]
    double *sG = sY + LSP * TILE;                                     // [104][32] G and 1/G, then P and L
    double *sC = sG + 2 * LSP * TILE;                                 // [SC_N][32]
    double *sPoly = sC + SC_N * TILE;                                 // [52][14]
    double *sH = sPoly + CHEM_POLY;                                   // [16][32] heat release by warp
    uint64_t *bar = reinterpret_cast<uint64_t *>(sH + CHEM_WARPS * TILE);
    double2 *pr = reinterpret_cast<double2 *>(sRC);
    const DevParams &P = *a.P;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    // ---- stage the reaction-pair table (bulk copy, bounded wait)
    if (tid == 0) mbar_init(bar, 1);
    __syncthreads();
    if (tid == 0) {
        mbar_expect_tx(bar, PAIRTAB_BYTES);
        constexpr int CH = 8192;
        for (int off = 0; off < PAIRTAB_BYTES; off += CH) {
            int bytes = PAIRTAB_BYTES - off < CH ? PAIRTAB_BYTES - off : CH;
            bulk_g2s(reinterpret_cast<unsigned char *>(sTab) + off,
                     reinterpret_cast<const unsigned char *>(a.tab) + off, bytes, bar);
        }
    }
    if (!mbar_wait_bounded(bar, 0, 1 << 20)) {
        if (tid == 0) atomicExch(a.status, ST_TMA_TIMEOUT);
        mbar_wait_bounded(bar, 0, 1 << 20);   // let the copy in flight land before exiting
        return;
    }

    for (int i = tid; i < CHEM_POLY; i += CHEM_THREADS) sPoly[i] = P.poly[i];
    const double RCONV = P.RCONV;
    const bool want_omega = a.qdsp || a.qdot || a.dwdy;
    const int nwork = a.tile_list ? *a.tile_count : a.ntile;
    constexpr int NROW = (LSP + CHEM_WARPS - 1) / CHEM_WARPS;
    // the rows of a tile that this warp loads: Y of species warp, warp + 16, ..., and the scalars (the last warp)
    double ynext[NROW], snext[4];
    auto load = [&](int w) {
        const size_t cell = (size_t)(a.tile_list ? a.tile_list[w] : w) * TILE + lane;
#pragma unroll
        for (int i = 0; i < NROW; ++i)
            if (warp + i * CHEM_WARPS < LSP) ynext[i] = a.y[(size_t)(warp + i * CHEM_WARPS) * a.npad + cell];
        if (warp == CHEM_WARPS - 1) {
            snext[0] = a.tk[cell];
            snext[1] = a.rho[cell];
            snext[2] = a.stmf ? a.stmf[cell] : 0.0;
            snext[3] = a.stnd ? a.stnd[cell] : 0.0;
        }
    };
    if ((int)blockIdx.x < nwork) load(blockIdx.x);
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const int tile = a.tile_list ? a.tile_list[w] : w;
        const size_t cell = (size_t)tile * TILE + lane;
        const int cls = a.skip ? a.skip[cell] : 0;
        const bool tile_skips = a.skip && __syncthreads_or(cls != 0);
        // ---------------- phase 0
#pragma unroll
        for (int i = 0; i < NROW; ++i)
            if (warp + i * CHEM_WARPS < LSP) sY[(warp + i * CHEM_WARPS) * TILE + lane] = ynext[i];
        if (warp == CHEM_WARPS - 1) tile_scalars(P, sC, lane, snext[0], snext[1], snext[2], snext[3]);
        __syncthreads();
        if (w + (int)gridDim.x < nwork) load(w + gridDim.x);
        // ---------------- phases 1-2
        double *rc = a.rc && cls == 0 ? a.rc + cell : nullptr;
        tile_rates_fp64<CHEM_WARPS>(P, sTab, sPoly, sY, sG, sC, a.sour, a.npad, cell, lane, warp, cls != 0,
                                    [&](int p, double rc0, double rc1) {
                                        if (want_omega) pr[p * TILE + lane] = make_double2(rc0, rc1);
                                        if (rc) {
                                            double *d = rc + (size_t)(2 * p) * a.npad;
                                            d[0] = rc0;
                                            d[a.npad] = rc1;
                                        }
                                    });
        __syncthreads();
        if (!want_omega) continue;                        // RC and SOUR only: no species sums (uniform branch)
        if (tile_skips) {
            // a skipped cell's omega comes from the RC it kept (solveh.f:116-1145 reads RC as it is)
            if (cls == 1)
                for (int p = warp; p < NPAIR; p += CHEM_WARPS)
                    pr[p * TILE + lane] = a.rc_stale ? make_double2(a.rc_stale[(size_t)(2 * p) * a.npad + cell],
                                                                   a.rc_stale[(size_t)(2 * p + 1) * a.npad + cell])
                                                     : make_double2(0.0, 0.0);
            __syncthreads();
        }
        // ---------------- phase 3: gain and loss sums
        tile_omega_sums(pr, sY, sG, lane, warp);
        __syncthreads();
        // ---------------- phase 4: the species' outputs
        const bool put = cls < 2;
        {
            const double TKD = sC[SC_TKD * TILE + lane];
            const double *hc = P.hc + (TKD > UC_TPOL1 ? 6 : 0);
            double hrr = 0.0;
#pragma unroll
            for (int i = 0; i < NROW; ++i) {
                const int k = warp + i * CHEM_WARPS;
                if (k >= LSP) break;
                const double L = sG[(LSP + k) * TILE + lane];
                const double q = -(RCONV * (P.WM[k] * fma(-sY[k * TILE + lane], L, sG[k * TILE + lane])));
                if (a.qdsp && put) a.qdsp[(size_t)k * a.npad + cell] = q;
                if (a.dwdy && put) a.dwdy[(size_t)k * a.npad + cell] = -(RCONV * P.WM[k] * L);
                // species enthalpy (solveh.f:39-57) for the heat release
                const double *e = hc + k * 12;
                const double H = fma(TKD, fma(TKD, fma(TKD, fma(TKD, fma(TKD, e[4], e[3]), e[2]), e[1]), e[0]), e[5]);
                hrr = fma(q, H, hrr);
            }
            sH[warp * TILE + lane] = hrr;
        }
        __syncthreads();
        if (warp == 0 && a.qdot && put) {
            double hrr = 0.0;
            for (int i = 0; i < CHEM_WARPS; ++i) hrr = hrr + sH[i * TILE + lane];
            a.qdot[cell] = hrr;
        }
        // the next tile's barriers order these reads before sH is written again
    }
}

}  // namespace uc

namespace uc {
// List of the tiles whose flag is set (one CTA; order of the tile index).
__global__ void compact_tiles_kernel(const int *flag, int ntile, int *list, int *count)
{
    __shared__ int s_base;
    if (threadIdx.x == 0) s_base = 0;
    __syncthreads();
    for (int t0 = 0; t0 < ntile; t0 += blockDim.x) {
        const int t = t0 + threadIdx.x;
        const int f = (t < ntile) ? flag[t] : 0;
        const unsigned m = __ballot_sync(0xffffffffu, f);
        __shared__ int s_warp[32];
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        if (lane == 0) s_warp[w] = __popc(m);
        __syncthreads();
        if (threadIdx.x == 0) {
            int acc = s_base;
            for (int i = 0; i < (int)(blockDim.x >> 5); ++i) { const int c = s_warp[i]; s_warp[i] = acc; acc += c; }
            s_base = acc;
        }
        __syncthreads();
        if (f) list[s_warp[w] + __popc(m & ((1u << lane) - 1))] = t;
        __syncthreads();
    }
    if (threadIdx.x == 0) *count = s_base;
}
}  // namespace uc
