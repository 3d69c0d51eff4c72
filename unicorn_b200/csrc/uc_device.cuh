// Device-side data structures shared by the unichem kernels (sm_100a).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "generated/mech_tables.h"
#include "rate_limits.h"

namespace uc {

constexpr int LSP = UC_LSP;
constexpr int LRX = UC_LRX;
constexpr int NPAIR = UC_NPAIR;
constexpr int TILE = 32;                 // cells per tile = lanes of a warp
constexpr int CHEM_WARPS = RATE_WARPS;   // warps of the rate/omega kernel
constexpr int CHEM_THREADS = CHEM_WARPS * 32;
constexpr int MAX_SPEC_PER_WARP = 8;
constexpr int PROP_ROWS = 24;            // see DevParams::prow

// status words written by kernels (device side; the host maps them to UC_E*)
constexpr int ST_OK = 0;
constexpr int ST_TMA_TIMEOUT = 1;
constexpr int ST_NEWTON_NOCONV = 2;
constexpr int ST_BAD_ORDER = 3;
constexpr int ST_MMA_TIMEOUT = 4;
constexpr int ST_RELAX_TIMEOUT = 5;

// One reaction pair of the mechanism as the reference's sources give it: forward slot 2p and reverse slot
// 2p + 1 (0-based). Host side: the device tables are made from it.
struct PairSrc {
    double akf, alf, exaf, akf_r;          // Arrhenius of the forward slot; AKF of the reverse slot
    double aklow, allow, ealow;            // fall-off low-pressure limit (aklow = 0: none)
    double troe[4];                        // TROE(IR,1..4)
    int8_t has_rev, rut, qlen, dmole;      // reverse formula present; RUT power; q length; TB group of DMOLE
    int8_t rc_order0, rc_order1, rc_tb0, rc_tb1;   // RC assembly (order 0 = slot never written)
    int8_t rc_len0, rc_len1;
    int8_t qsp[8], qdiv[8];                // q = G[qsp0] (*|/) G[qsp1] ...
    int8_t rc_kind0[4], rc_idx0[4];        // post factors: kind 1 = *Y[idx], 0 = /WM[idx]
    int8_t rc_kind1[4], rc_idx1[4];
};

// The pair as the FP64 rate kernels evaluate it: k_f = akf T^alf exp(-exaf / T); k_r = k_f * (RUT power) * 1/q
// with 1/q a product of rows of the table of G and 1/G; RC = c * rho^order * [third body] * k [* Y]. Rows name
// scalar rows (SC_*, 0: none) of the tile, so nothing is decoded or divided per cell.
struct __align__(16) PairTab {
    double akf, alf, exaf, c0, c1, pad0;
    uint8_t g[KC_MAX], ng, rut;            // rows of the G table (k: G_k, 52 + k: 1 / G_k); ng = 0: no reverse
    uint8_t r0, t0, r1, t1;                // rows of rho^order (0: the slot is never written) and of the third body
    uint8_t y0, y1, fall, pad1;            // species whose Y is a factor (255: none); 1 + fall-off entry (0: none)
};
static_assert(sizeof(PairTab) == 64, "PairTab layout");
struct __align__(16) FallTab {
    double aklow, allow, ealow, troe[4];
    int dmole, pad;                        // scalar row of the third body
};
static_assert(sizeof(FallTab) == 64, "FallTab layout");
// both tables lie one after the other, staged into shared memory by bulk (TMA) copies at kernel start
constexpr int PAIRTAB_BYTES = NPAIR * (int)sizeof(PairTab) + FALL_MAX * (int)sizeof(FallTab);
static_assert(PAIRTAB_BYTES % 16 == 0, "bulk copy size must be a multiple of 16 bytes");

// Constants of one context: scales, tables prepared at set-up, and the
// static work split of the species phase.
struct DevParams {
    double TSTR, RSTR, WMSTR, ALSTR, VSTR, HSTR, GASC, PBACK, CONVRC, CONVRM, CONVRD;
    double C1ST, C2ND, C3RD, RCONV, HCONVR, TKDMIN, RSTR_WMSTR, BETA1, BETA3, REI;
    double WM[LSP], HFO[LSP];
    int8_t elem[LSP * 3];                 // atoms of C, H, O per species
    double poly[LSP * 14];
    double om22[LSP * 12];
    double cdia[LSP];
    double ci11[20];
    double WMIK[LSP * LSP], DWMIK[LSP * LSP], WMCD[LSP * LSP];
    double ETLJ1[LSP * LSP], ETLJ2[LSP * LSP], ETLJ3[LSP * LSP], ETLJ4[LSP * LSP];
    double RETLJ1[LSP * LSP];             // 1 / ETLJ1 (the mixed form's collision-integral argument)
    // cp/R / W and h of every species as polynomials in T for Horner evaluation, per temperature range
    // (0: T <= TPOL1, 1: above): cp_k / W_k = sum_i cpc[i] T^i, h_k = T (sum_i hc[i] T^i) + hc[5]
    double cpc[LSP * 2 * 5], hc[LSP * 2 * 6];
    // the FP64 property kernel's tables, species fastest (lane = species): per temperature range rows 0-4
    // the Eucken factor's polynomial (0.115 + 0.354 cp/R), 5-10 cdia^2 times the Omega(2,2) fit, 11 CONVRC / W_kk,
    // 12 CONVRM W_kk (W_kk = WMIK of the species with itself), 13-17 cpc, 18-23 hc; and for the pair
    // (b, k) at b * LSP + k: 1 / WMCD, WMIK(k, b), 1 / DWMIK(k, b) (RETLJ1 is symmetric)
    double prow[2][PROP_ROWS][LSP];
    double piw[LSP * LSP], pw[LSP * LSP], pid[LSP * LSP];
    // per temperature range and species the coefficients of A1..A6 of the T Newton: p_i / W_k / (i + 1), and p_6 / W_k
    alignas(16) double tco[2][LSP][6];
    // third bodies as weights of Y: row 0 TBODY (1 / W_k), rows 1..10 the groups
    double tbw[11 * LSP];
    // third-body groups 1..10 (TBODY + sum sign*coef*Y/W)
    int16_t tb_off[11], tb_len[11];
    int8_t tb_sp[64], tb_sign[64], tb_hascoef[64];
    double tb_coef[64];
    // omega phase
    int16_t prd_off[LSP], prd_len[LSP], loss_off[LSP], loss_len[LSP];
    uint16_t prd_term[UC_NPRD_TERMS];
    double prd_coef[UC_NPRD_TERMS];
    uint16_t loss_term[UC_NLOSS_TERMS];
    int8_t ra_len[LRX], ra_sp[LRX * 3];
    // species assigned to each warp of the rate/omega kernel (balanced by terms)
    int8_t spec_of_warp[CHEM_WARPS][MAX_SPEC_PER_WARP];
    int8_t nspec_of_warp[CHEM_WARPS];
    // reaction pairs assigned to each warp (balanced by cost)
    int16_t pair_of_warp[CHEM_WARPS][WARP_ITEMS];
    int8_t npair_of_warp[CHEM_WARPS];
    int soot_warp;                        // the warp (of 16) that forms the soot sources
};

// Rounded as written (no contraction of a product into a neighbouring sum, which the compiler may do one way or
// the other): for code that several kernels run and that has to give a cell the same bits in each.
#define CO_FMA(a, b, c) __fma_rn(a, b, c)
#define CO_MUL(a, b) __dmul_rn(a, b)
#define CO_ADD(a, b) __dadd_rn(a, b)

// n / d without the branch of the compiler's division, which would end the scheduling of the statements around
// it and is three times the instructions: the hardware's reciprocal approximation r, one step of third order for
// the quotient (with e = 1 - d r, 1 / d = r (1 + e + e^2 + ...)), and the residual correction of Markstein (IBM J.
// Res. Dev. 34, 1990). For 2^-1022 <= |d| <= 2^1022 and a quotient in the normal range up to 2^1023 it is within
// one unit in the last place of the division (no difference in 1.8 million random quotients). Where the residual is
// not finite, because d is zero or infinite, n is infinite, an operand is NaN or the quotient overflows, n r is what
// the division gives. A subnormal d is taken as zero, a finite one above 2^1022 as infinite.
__device__ __forceinline__ double co_quot(double n, double d)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = __fma_rn(-d, r, 1.0), q0 = __dmul_rn(n, r);
    const double q = __fma_rn(q0, __fma_rn(e, e, e), q0), m = __fma_rn(-d, q, n);
    return (__double2hiint(m) & 0x7ff00000) != 0x7ff00000 ? __fma_rn(m, r, q) : q0;
}

// x / T with 1 / T at hand: the quotient corrected by its residual (within one unit in the last place of the division
// for finite x and T in the range of temperatures; no difference in a million), for the exponents, where an error
// is multiplied by the exponent's size.
__device__ __forceinline__ double over_t(double x, double TKD, double IT)
{
    const double q = CO_MUL(x, IT);
    return CO_FMA(CO_FMA(-q, TKD, x), IT, q);
}

// ------------------------------------------------------------------ TMA / mbarrier

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// 1-D bulk copy global -> shared (no multicast), completion on the mbarrier.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// Bounded wait on phase `parity` of the mbarrier: returns false if it gave up.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, int max_tries)
{
    for (int i = 0; i < max_tries; ++i) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

}  // namespace uc
