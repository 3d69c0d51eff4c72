// Property kernels: Y clip + mixture-averaged transport (FP64: a warp takes a cell; mixed
// form, with the pair terms in FP32: a thread takes one), cp/h (FP64: a thread takes a cell,
// or in small fields a block 32 cells) and temperature from enthalpy (FP64, a thread a cell).
#pragma once
#include "uc_device.cuh"

namespace uc {

struct PropArgs {
    const DevParams *P;
    const double *tk;
    double *y;                       // [52][npad], clipped in place (main:821-828)
    double *vmu, *vtc, *vdf;         // outputs (vdf [52][npad])
    int n, npad;
};

__device__ __forceinline__ int ci_range(double TKDS)
{
    int K = 0;
    if (TKDS >= 2.0) K = 1;
    if (TKDS > 5.0) K = 2;
    if (TKDS > 70.0) K = 3;
    return K;
}

// src/unicornd-mild-sd-5.f:821-1006, FP64. A warp takes a cell. The cell's sub-mixture (species with Y >= 1e-3,
// and N2; about five) is a list in shared memory: one lane per entry forms the entry's own values and its Wilke
// sums, then lanes are species (k = lane and lane + 32) and sum 1 / D_kb over the list, so the pair
// tables are read in rows and no lane waits for another cell's list. The Y rows of a block's cells come in
// and D_k goes out through shared memory, in rows of cells. The divisions and square roots of each pair are
// divisions and square roots of each species: X_b / D_kb is X_b CI / (WMCD TKBP) from a table of
// reciprocals, sqrt(ATC_k / ATC_b) a product of the two species' roots.
//
// The roots are taken per species, so ATC and AMU have to be positive: the fits give that from 20 to 6,000 K.
//
// What bounds it: FP64 latency (a cell is one chain of sums; four blocks per SM hide part of it). A thread per
// cell, as before (a chain of about 300 pairs per thread, its lists in local memory), took 150 us for
// 101 cells, 420 us for 180,901 and 1.53 ms for 1,048,576; this form 13.5 us, 253 us and 1.41 ms.
// CELLS: cells of a block's tile, 16 for whole cache lines of the rows, 8 where that leaves SMs without
// a block (fields below PROP_SMALL cells per SM).
constexpr int PROP_THREADS = 256;
constexpr int PROP_SMALL = 32;

template <int CELLS>
__global__ void __launch_bounds__(PROP_THREADS, 4) props_fp64_kernel(const PropArgs a)
{
    __shared__ double sY[LSP][CELLS + 1], sD[LSP][CELLS + 1];
    __shared__ double sN2[CELLS], sMu[CELLS], sTc[CELLS], sCi[20];
    enum { L_X, L_ATC, L_AMU, L_RA, L_RM, L_IA, L_IM, L_N };
    __shared__ double sL[PROP_THREADS / 32][L_N][LSP];     // per warp: the sub-mixture's values
    __shared__ int sK[PROP_THREADS / 32][LSP];             // ... and its species
    const DevParams &P = *a.P;
    const size_t np = a.npad;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < 20) sCi[tid] = P.ci11[tid];
    const int k1 = min(lane + 32, LSP - 1);        // the second species of the lane (lanes 20..31: none)
    const bool two = lane + 32 < LSP;
    const int ntile = (a.n + CELLS - 1) / CELLS;
    for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const int c0 = tile * CELLS, nc = min(CELLS, a.n - c0);
        for (int i = tid; i < LSP * CELLS; i += PROP_THREADS) {
            const int k = i / CELLS, j = i % CELLS;
            if (j >= nc) continue;
            double v = a.y[(size_t)k * np + c0 + j];
            if (k < LSP - 1 && v < 0.0) {          // Y clip (main:821-828)
                v = 0.0;
                a.y[(size_t)k * np + c0 + j] = 0.0;
            }
            sY[k][j] = v;
        }
        __syncthreads();
        if (warp == PROP_THREADS / 32 - 1 && lane < nc) {
            double mass = 0.0;                     // N2 closure (main:827-828), summed in the reference's order
#pragma unroll
            for (int k = 0; k < LSP - 1; ++k) mass = mass + sY[k][lane];
            sN2[lane] = 1.0 - mass;
        }
        for (int j = warp; j < nc; j += PROP_THREADS / 32) {
            const double y0 = sY[lane][j];
            const double y1 = two && lane + 32 < LSP - 1 ? sY[k1][j] : 0.0;
            // sub-mixture: all species but those with Y < 1e-3 (a NaN stays in and shows in the results), plus N2
            // (main:842-915)
            const bool in0 = !(y0 < 1.0e-03), in1 = !(y1 < 1.0e-03), isn2 = lane + 32 == LSP - 1;
            const double iw0 = P.tbw[lane], iw1 = P.tbw[k1];
            double x0 = in0 ? y0 * iw0 : 0.0, x1 = in1 ? y1 * iw1 : 0.0;
            double mass = (in0 ? y0 : 0.0) + (in1 ? y1 : 0.0), TMOLE = x0 + x1;
            for (int o = 16; o > 0; o >>= 1) {
                mass += __shfl_xor_sync(0xffffffffu, mass, o);
                TMOLE += __shfl_xor_sync(0xffffffffu, TMOLE, o);
            }
            const double xn2 = (1.0 - mass) * P.tbw[LSP - 1];
            TMOLE += xn2;
            if (isn2) x1 = xn2;
            // the list, in species order (N2 last)
            const unsigned m0 = __ballot_sync(0xffffffffu, in0), m1 = __ballot_sync(0xffffffffu, in1 || isn2);
            const unsigned below = (1u << lane) - 1;
            const int nl = __popc(m0) + __popc(m1);
            double(*L)[LSP] = sL[warp];
            int *K = sK[warp];
            if (in0) {
                K[__popc(m0 & below)] = lane;
                L[L_X][__popc(m0 & below)] = x0;
            }
            if (in1 || isn2) {
                K[__popc(m0) + __popc(m1 & below)] = lane + 32;
                L[L_X][__popc(m0) + __popc(m1 & below)] = x1;
            }
            __syncwarp();
            // the entries' own values (main:929-939)
            const double tk = a.tk[c0 + j], TKRT = sqrt(tk), T = tk * P.TSTR;
            const double(*row)[LSP] = P.prow[T >= UC_TPOL1 ? 1 : 0];
            const double TKBP = tk * TKRT / P.PBACK;
            for (int l = lane; l < nl; l += 32) {
                const int k = K[l];
                const double eu = fma(fma(fma(fma(row[4][k], T, row[3][k]), T, row[2][k]), T, row[1][k]), T, row[0][k]);
                const double si = fma(fma(fma(fma(fma(row[10][k], T, row[9][k]), T, row[8][k]), T, row[7][k]), T, row[6][k]), T, row[5][k]);
                const double is = TKRT / si, atc = row[11][k] * eu * is, amu = row[12][k] * is;
                const double ra = sqrt(atc), rm = sqrt(amu);
                L[L_ATC][l] = atc;
                L[L_AMU][l] = amu;
                L[L_RA][l] = ra;
                L[L_RM][l] = rm;
                L[L_IA][l] = 1.0 / ra;
                L[L_IM][l] = 1.0 / rm;
            }
            __syncwarp();
            // Wilke sums (main:957-979)
            double tc = 0.0, mu = 0.0;
            for (int l = lane; l < nl; l += 32) {
                const int k = K[l];
                const double ra = L[L_RA][l], rm = L[L_RM][l], x = L[L_X][l];
                double phi = 0.0, psi = 0.0;
                for (int b = 0; b < nl; ++b) {
                    const int ij = K[b] * LSP + k;
                    const double w = P.pw[ij], id = L[L_X][b] * P.pid[ij];
                    const double t1 = fma(ra * L[L_IA][b], w, 1.0), t2 = fma(rm * L[L_IM][b], w, 1.0);
                    if (b != l) {
                        phi = fma(id, t1 * t1, phi);
                        psi = fma(id, t2 * t2, psi);
                    }
                }
                tc += L[L_ATC][l] * x / (x + (double)1.065f * phi);
                mu += L[L_AMU][l] * x / (x + psi);
            }
            for (int o = 16; o > 0; o >>= 1) {
                tc += __shfl_xor_sync(0xffffffffu, tc, o);
                mu += __shfl_xor_sync(0xffffffffu, mu, o);
            }
            // 1 / D_kb (main:940-953, 981-1003)
            double efd[2] = {0.0, 0.0}, ilast[2] = {0.0, 0.0};
            for (int l = 0; l < nl; ++l) {
                const int b = K[l];
                const double xb = L[L_X][l];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int k = h ? k1 : lane, ij = b * LSP + k;
                    const double t = T * P.RETLJ1[ij];
                    const double *c = sCi + ci_range(t) * 5;
                    ilast[h] = fma(fma(fma(fma(c[4], t, c[3]), t, c[2]), t, c[1]), t, c[0]) * P.piw[ij];   // TKBP / D_kb
                    // (the reference gives N2 its own term: ISPQ(LSP) is never assigned)
                    if (b != k || b == LSP - 1) efd[h] = fma(xb, ilast[h], efd[h]);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const bool in = h ? in1 : in0;
                const double aa = in ? TMOLE - (h ? x1 : x0) : TMOLE;
                // a species alone: its D with N2, the last of the list
                const double d = in && aa <= 1.0e-10 ? TKBP / ilast[h] : aa * TKBP / efd[h];
                if (h == 0 || two) sD[h ? k1 : lane][j] = P.CONVRD * d;
            }
            __syncwarp();
            if (lane == 0) {
                sMu[j] = mu;
                sTc[j] = tc;
            }
        }
        __syncthreads();
        for (int i = tid; i < LSP * CELLS; i += PROP_THREADS) {
            const int k = i / CELLS, j = i % CELLS;
            if (j < nc) a.vdf[(size_t)k * np + c0 + j] = sD[k][j];
        }
        if (tid < nc) {
            a.y[(size_t)(LSP - 1) * np + c0 + tid] = sN2[tid];
            a.vmu[c0 + tid] = sMu[tid];
            a.vtc[c0 + tid] = sTc[tid];
        }
        __syncthreads();
    }
}

// The collision integral CI11 of the pair (i, j) in Horner form with the
// argument t = T / ETLJ1 from the reciprocal table: FP64, no division
// (the quartic in T* has alternating-sign coefficients and cancels).
__device__ __forceinline__ double ci11_horner(const DevParams &P, int ij, double TKD1)
{
    const double t = TKD1 * P.RETLJ1[ij];
    const double *c = P.ci11 + ci_range(t) * 5;
    return fma(fma(fma(fma(c[4], t, c[3]), t, c[2]), t, c[1]), t, c[0]);
}

// The mixed form of src/unicornd-mild-sd-5.f:821-1006: the per-pair work of
// the Wilke sums and of the binary diffusion sums (square roots, divisions,
// the products of each term) runs in FP32; what cancels or accumulates stays
// FP64 -- the polynomials in T (cp/R of the Eucken factor, the Omega(2,2) fit
// to T^5, the CI11 quartic, all in Horner form), the sums over species, the
// mole numbers and TMOLE - X_i, and the per-species values ATC, AMU. Every
// pair term then carries a few FP32 roundings and nothing adds them up, so
// mu, lambda and D_k stay within a few 1e-7 of the FP64 form.
__global__ void __launch_bounds__(128) props_mixed_kernel(const PropArgs a)
{
    const DevParams &P = *a.P;
    const size_t np = a.npad;
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < (size_t)a.n; c += (size_t)gridDim.x * blockDim.x) {
        double TMASS = 0.0;
        for (int k = 0; k < LSP - 1; ++k) {
            double yk = a.y[k * np + c];
            if (yk < 0.0) { yk = 0.0; a.y[k * np + c] = 0.0; }
            TMASS = TMASS + yk;
        }
        a.y[(LSP - 1) * np + c] = 1.0 - TMASS;
        int8_t sub[LSP];
        double X[LSP];
        int IA = 0;
        double TMASSD = 0.0, TMOLE = 0.0;
        for (int k = 0; k < LSP - 1; ++k) {
            const double yk = a.y[k * np + c];
            if (yk < 1.0e-03) continue;
            sub[IA] = (int8_t)k;
            TMASSD = TMASSD + yk;
            X[IA] = yk / P.WM[k];
            TMOLE = TMOLE + X[IA];
            ++IA;
        }
        int LSPT = IA + 1;
        if (LSPT >= LSP) LSPT = LSP;
        sub[LSPT - 1] = LSP - 1;
        X[LSPT - 1] = (1.0 - TMASSD) / P.WM[LSP - 1];
        TMOLE = TMOLE + X[LSPT - 1];
        const double tk = a.tk[c];
        const double TKRT = sqrt(tk);
        const double TKD1 = tk * P.TSTR;
        const int IPL1 = TKD1 >= UC_TPOL1 ? 7 : 0, IPL2 = TKD1 >= UC_TPOL1 ? 6 : 0;
        const float TKBP = (float)(tk * TKRT / P.PBACK);
        double ATC[LSP], AMU[LSP];
        float ATCf[LSP], AMUf[LSP], Xf[LSP];
        for (int i = 0; i < LSPT; ++i) {
            const int k = sub[i];
            const double *p = P.poly + k * 14 + IPL1;
            const double *q = P.om22 + k * 12 + IPL2;
            const double cpr = fma(fma(fma(fma(p[4], TKD1, p[3]), TKD1, p[2]), TKD1, p[1]), TKD1, p[0]);
            const double EUKEN = (double)0.115f + (double)0.354f * cpr;
            const double om = fma(fma(fma(fma(fma(q[5], TKD1, q[4]), TKD1, q[3]), TKD1, q[2]), TKD1, q[1]), TKD1, q[0]);
            const double SIOME = P.cdia[k] * P.cdia[k] * om;
            ATC[i] = P.CONVRC * EUKEN * TKRT / P.WMIK[k * LSP + k] / SIOME;
            AMU[i] = P.CONVRM * TKRT * P.WMIK[k * LSP + k] / SIOME;
            ATCf[i] = (float)ATC[i];
            AMUf[i] = (float)AMU[i];
            Xf[i] = (float)X[i];
        }
        double VTC = 0.0, VMU = 0.0;
        double VDFQ[LSP];
        for (int i = 0; i < LSPT; ++i) {
            const int k = sub[i];
            double PHIK = 0.0, PHDIK = 0.0, EFDIK = 0.0;
            for (int j = 0; j < LSPT; ++j) {
                if (j == i) continue;
                const int kb = sub[j];
                const int ij = k * LSP + kb;
                const float w = (float)P.WMIK[ij], dw = (float)P.DWMIK[ij];
                const float t1 = 1.0f + sqrtf(ATCf[i] / ATCf[j]) * w;
                const float t2 = 1.0f + sqrtf(AMUf[i] / AMUf[j]) * w;
                PHIK += (double)(Xf[j] * (t1 * t1) / dw);
                PHDIK += (double)(Xf[j] * (t2 * t2) / dw);
                const float CI = (float)ci11_horner(P, i < j ? k * LSP + kb : kb * LSP + k, TKD1);
                EFDIK += (double)(Xf[j] * CI / ((float)P.WMCD[ij] * TKBP));
            }
            VTC = VTC + ATC[i] * X[i] / (X[i] + (double)1.065f * PHIK);
            VMU = VMU + AMU[i] * X[i] / (X[i] + PHDIK);
            const double AA = TMOLE - X[i];
            if (AA <= 1.0e-10) {
                double d = 0.0;
                if (i != LSPT - 1) {
                    const int kl = sub[LSPT - 1];
                    d = P.WMCD[k * LSP + kl] * (double)TKBP / ci11_horner(P, k * LSP + kl, TKD1);
                }
                VDFQ[i] = P.CONVRD * d;
            } else {
                VDFQ[i] = P.CONVRD * AA / EFDIK;
            }
        }
        a.vtc[c] = VTC;
        a.vmu[c] = VMU;
        int pos = 0;
        for (int k = 0; k < LSP; ++k) {
            double v;
            if (k < LSP - 1 && pos < LSPT - 1 && sub[pos] == k) {
                v = VDFQ[pos];
                ++pos;
            } else {
                double EFD = 0.0;
                for (int b = 0; b < LSPT; ++b) {
                    const int nb = sub[b];
                    const float CI = (float)ci11_horner(P, k * LSP + nb, TKD1);
                    EFD += (double)(Xf[b] * CI / ((float)P.WMCD[k * LSP + nb] * TKBP));
                }
                v = P.CONVRD * TMOLE / EFD;
            }
            a.vdf[k * np + c] = v;
        }
    }
}

// Mixture cp (spgsolv.f:102-173) and h = sum_k Y_k h_k (h_k: solveh.f:39-57).
struct CpHArgs {
    const DevParams *P;
    const double *tk, *y;
    double *cp, *h;
    int n, npad;
};

// cp and h of each cell from the coefficient tables of DevParams (the polynomials of
// spgsolv.f:102-173 and solveh.f:39-57 with the divisions by W_k, by the powers' orders and
// the scale factors folded in at set-up), in Horner form: a few fused multiply-adds per
// species, so the kernel is bound by reading the 52 Y rows (the table form rounds differently
// from the reference's expression by a few units in the last place). Below CPH_SMALL cells per SM a block
// takes 32 cells (lane = cell) and deals the species over its warps, so that a small field's rows are all read at
// once: 12 us for 101 cells against 28 for a thread per cell; above, a thread takes a cell, which keeps as many
// bytes in flight without the barriers: 172 us for 1,048,576 cells against 344, 48 against 60 for 180,901.
constexpr int CPH_SMALL = 512;
__global__ void __launch_bounds__(256) cp_h_kernel(const CpHArgs a)
{
    const DevParams &P = *a.P;
    const size_t np = a.npad;
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < (size_t)a.n; c += (size_t)gridDim.x * blockDim.x) {
        const double T = a.tk[c] * P.TSTR;
        const int r = T > UC_TPOL1 ? 1 : 0;
        double TCP = 0.0, hs = 0.0;
#pragma unroll 4
        for (int k = 0; k < LSP; ++k) {
            const double yk = a.y[k * np + c];
            const double *q = P.cpc + (k * 2 + r) * 5;
            const double *e = P.hc + (k * 2 + r) * 6;
            const double cpk = fma(fma(fma(fma(q[4], T, q[3]), T, q[2]), T, q[1]), T, q[0]);
            const double hk = fma(T * fma(fma(fma(fma(e[4], T, e[3]), T, e[2]), T, e[1]), T, e[0]), 1.0, e[5]);
            TCP = TCP + cpk * yk;
            hs = hs + yk * hk;
        }
        if (a.cp) a.cp[c] = TCP / P.WMSTR * P.GASC * P.TSTR / P.HSTR;
        if (a.h) a.h[c] = hs;
    }
}

constexpr int CPH_WARPS = 8;
__global__ void __launch_bounds__(CPH_WARPS * 32) cp_h_small_kernel(const CpHArgs a)
{
    constexpr int NK = (LSP + CPH_WARPS - 1) / CPH_WARPS;
    __shared__ double sCp[CPH_WARPS][32], sHs[CPH_WARPS][32];
    const DevParams &P = *a.P;
    const size_t np = a.npad;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double scale = P.GASC * P.TSTR / P.HSTR / P.WMSTR;
    // (rows end at npad, a multiple of 32: every lane has a cell to read)
    for (size_t c0 = (size_t)blockIdx.x * 32; c0 < (size_t)a.n; c0 += (size_t)gridDim.x * 32) {
        const size_t c = c0 + lane;
        const double T = a.tk[c] * P.TSTR;
        double y[NK], cp = 0.0, hs = 0.0;
#pragma unroll
        for (int i = 0; i < NK; ++i) y[i] = warp + i * CPH_WARPS < LSP ? a.y[(warp + i * CPH_WARPS) * np + c] : 0.0;
        const double(*row)[LSP] = P.prow[T > UC_TPOL1 ? 1 : 0];
#pragma unroll
        for (int i = 0; i < NK; ++i) {
            const int k = min(warp + i * CPH_WARPS, LSP - 1);
            const double cpk = fma(fma(fma(fma(row[17][k], T, row[16][k]), T, row[15][k]), T, row[14][k]), T, row[13][k]);
            const double hk = fma(T, fma(fma(fma(fma(row[22][k], T, row[21][k]), T, row[20][k]), T, row[19][k]), T, row[18][k]), row[23][k]);
            cp = fma(cpk, y[i], cp);
            hs = fma(hk, y[i], hs);
        }
        sCp[warp][lane] = cp;
        sHs[warp][lane] = hs;
        __syncthreads();
        if (warp < 2 && c < (size_t)a.n) {
            double s = 0.0;
#pragma unroll
            for (int i = 0; i < CPH_WARPS; ++i) s += warp ? sHs[i][lane] : sCp[i][lane];
            if (warp == 0 && a.cp) a.cp[c] = s * scale;
            if (warp == 1 && a.h) a.h[c] = s;
        }
        __syncthreads();
    }
}

// Temperature from the sensible enthalpy by Newton (solveh.f:1170-1234).
struct TempArgs {
    const DevParams *P;
    const double *y, *ht;
    double *tk;
    int *status;
    int n, npad;
    const int8_t *skip;              // optional ISKIP class: skipped cells keep T (solveh.f:1173)
};

__global__ void __launch_bounds__(128) temperature_fp64_kernel(const TempArgs a)
{
    const DevParams &P = *a.P;
    const size_t np = a.npad;
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < (size_t)a.n; c += (size_t)gridDim.x * blockDim.x) {
        if (a.skip && a.skip[c]) continue;
        double ENTH = (a.ht[c] - (double)0.5f * 0.0) * P.HSTR;
        for (int k = 0; k < LSP; ++k) ENTH = ENTH + a.y[k * np + c] * P.HFO[k] * P.HSTR;
        int IPL = 0;
        double TPOLY = UC_TPOL1;
        double TKD = a.tk[c] * P.TSTR;
        double A1, A2, A3, A4, A5, A6;
        for (int guard = 0; guard < 3; ++guard) {
            if (TKD > TPOLY) TKD = TPOLY / 2.0;
            A1 = A2 = A3 = A4 = A5 = A6 = 0.0;
            for (int k = 0; k < LSP; ++k) {
                const double *p = P.poly + k * 14 + IPL;
                const double yk = a.y[k * np + c];
                A1 = A1 + p[0] * yk / P.WM[k];
                A2 = A2 + p[1] * yk / P.WM[k] / 2.0;
                A3 = A3 + p[2] * yk / P.WM[k] / 3.0;
                A4 = A4 + p[3] * yk / P.WM[k] / 4.0;
                A5 = A5 + p[4] * yk / P.WM[k] / 5.0;
                A6 = A6 + p[5] * yk / P.WM[k];
            }
            const double FUNT = ((A1 + (A2 + (A3 + (A4 + A5 * TPOLY) * TPOLY) * TPOLY) * TPOLY) * TPOLY + A6) * P.GASC / P.WMSTR - ENTH;
            if (FUNT >= 1.0e-07) break;
            if (IPL >= 7) break;
            IPL = 7;
            if (TKD <= TPOLY) TKD = UC_TPOL2 / 2.0;
            TPOLY = UC_TPOL2;
        }
        bool conv = false;
        for (int it = 1; it <= 100; ++it) {
            const double DTKD = ((A1 + (A2 + (A3 + (A4 + A5 * TKD) * TKD) * TKD) * TKD) * TKD + A6 - ENTH * P.WMSTR / P.GASC) /
                                (A1 + (2.0 * A2 + (3.0 * A3 + (4.0 * A4 + 5.0 * A5 * TKD) * TKD) * TKD) * TKD);
            if (fabs(DTKD) <= (double)0.001f) { conv = true; break; }
            TKD = TKD - DTKD;
        }
        if (!conv && a.status) atomicCAS(a.status, ST_OK, ST_NEWTON_NOCONV);
        if (TKD > UC_TPOL2) TKD = UC_TPOL2;
        if (TKD < P.TKDMIN) TKD = P.TKDMIN;
        a.tk[c] = TKD / P.TSTR;
    }
}

}  // namespace uc
