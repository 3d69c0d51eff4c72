// Batched stiff point-implicit integration of independent cells (FP64, or FP32 rates with the FP64 update).
//
// Each cell is advanced over dt by n_sub sub-steps of dt/n_sub; every
// sub-step is the reference's own chain for a one-cell field: the rate
// coefficients (src/lib/ckrates.f), the point-implicit species update with
// its closure (src/lib/solvesp.f; the cell converges on its own residual,
// SPNORM = LSP-1, no face terms), T from the cell's constant total enthalpy
// (src/lib/solveh.f:1186-1234) and rho from the ideal gas at the cell's
// pressure (src/unicornd-mild-sd-5.f:1056-1062).
//
// n_sub comes from the cell's chemical time scale (nsub_kernel) and spans
// 1..~200, so the cost per cell is very uneven. The cells are ordered by
// n_sub (a stable counting sort, longest first) and a persistent kernel, one
// CTA per SM, takes 32-cell tiles from an atomic work queue: tiles hold cells
// of equal or neighbouring n_sub, and the longest tiles start first.
//
// Per tile the CTA keeps everything on chip: the reaction-pair table (one
// bulk copy per CTA), the tile's RC plane [544][32], Y, Y at the sub-step
// start and the update's scratch. The rates of a sub-step run on all NW
// warps (the phases of chem_fp64_kernel). The update runs on three of them, with
// the program of the tile-resident update (two form the species' sums, warp 0
// closes them; the two forms of the integration thus compute a cell the same way) and
// RC and Y in shared memory; the closure and the Newton for T run on warp 0 (lane = cell).
#pragma once
#include <cstddef>

#include "chem_kernel.cuh"
#include "chem_mixed_kernel.cuh"
#include "update_tr_kernel.cuh"

namespace uc {

// The rate coefficients of a tile in the mixed form of chem_mixed_kernel (FP64
// Gibbs exponents, ln Kc and exponent assembly; FP32 exponentials, fall-off
// blend and RC products), stored as doubles in sRC so that the FP64 update reads
// them unchanged; third bodies and soot sources as in the FP64 form. Reads the
// scalar rows of sC (SC_*), uses sG as scratch for the Gibbs exponents and the
// mixed pair table in global memory. Returns, uniformly over the block, whether
// a rate of the tile left the FP32 range (the caller then recomputes the tile
// in FP64).
template <int NW>
__device__ bool tile_rates_mixed(const DevParams &P, const PairTabM *tabm, double *sRC, const double *sY, double *sG,
                                 double *sC, double *sour, size_t sstride, size_t soff, int lane, int warp)
{
    {   // phase 1a: Gibbs exponents (FP64) and the Y/W rows
        const double TKD = sC[SC_TKD * TILE + lane], ELOGT = sC[SC_LNT * TILE + lane];
        const double IT = 1.0 / TKD;
        const int ip = TKD > UC_TPOL1 ? 7 : 0;
        const double T1 = TKD * 0.5, T2 = TKD * TKD * (1.0 / 6.0), T3 = T1 * T2, T4 = 1.2 * T1 * T3;
        for (int k = warp; k < LSP; k += NW) {
            const double *c = P.poly + k * 14 + ip;
            sG[k * TILE + lane] = c[0] * (ELOGT - 1.0) + c[1] * T1 + c[2] * T2 + c[3] * T3 + c[4] * T4 - c[5] * IT + c[6];
            sRC[k * TILE + lane] = sY[k * TILE + lane] / P.WM[k];
        }
    }
    __syncthreads();
    tile_tb_soot<NW>(P, sRC, sY, sC, sour, sstride, soff, lane, warp, false);
    bool out = false;
    {   // phase 2: reaction pairs -> RC (FP32 arithmetic, stored as doubles)
        const double TKD = sC[SC_TKD * TILE + lane], ELOGT = sC[SC_LNT * TILE + lane], IT = 1.0 / TKD;
        const double LNRHO = log(sC[SC_RHO * TILE + lane]), LNRUT = log(sC[SC_RUT * TILE + lane]);
        const double LNDMOLEA = log(sC[SC_DMOLEA * TILE + lane]);
        const float TKDf = (float)TKD;
        for (int vw = warp; vw < CHEM_WARPS; vw += NW)
        for (int i = 0; i < P.npair_of_warp[vw]; ++i) {
            const int p = P.pair_of_warp[vw][i];
            const PairTabM &T = tabm[p];
            const double lnkf = T.lnakf + T.alf * ELOGT - T.exaf * IT;
            double lnkr = -1.0e300;
            if (T.has_rev) {
                double lnq = 0.0;
                for (int t = 0; t < T.qlen; ++t) lnq += T.qsgn[t] * sG[T.qsp[t] * TILE + lane];
                lnkr = lnkf + T.rut * LNRUT - lnq;
            }
            double lafp = 0.0;
            if (T.falloff) {
                const double l20 = -46.051701859880914;      // ln 1e-20 (ckrates.f:770)
                const double lden = lnkf > l20 ? lnkf + log1p(exp(l20 - lnkf)) : l20 + log1p(exp(lnkf - l20));
                const double lnk0m = T.lnaklow + T.allow * ELOGT - T.ealow * IT +
                                     log(sC[(SC_TB0 + T.dmole) * TILE + lane]) + LNDMOLEA - lden;
                float RFACT;
                if (T.troe[0] > 0.0f) {
                    float FCLOG;
                    if (T.troe[1] == 0.0f) FCLOG = log10f(T.troe[0]);
                    else FCLOG = log10f((1.0f - T.troe[0]) * expf(-(TKDf / T.troe[1])) +
                                        T.troe[0] * expf(-(TKDf / T.troe[2])) + expf(-(T.troe[3] / TKDf)));
                    const float CPLOG = (float)(lnk0m * 0.43429448190325176) - (0.4f + 0.67f * FCLOG);
                    const float z = CPLOG / (0.75f - 1.27f * FCLOG - 0.14f * CPLOG);
                    RFACT = exp10f(FCLOG / (1.0f + z * z));
                } else if (T.troe[0] == 0.0f) {
                    RFACT = 1.0f;
                } else {
                    const float l = (float)(lnk0m * 0.43429448190325176);
                    const float XFACT = 1.0f / (1.0f + l * l);
                    RFACT = powf(-(T.troe[0] * expf(-(T.troe[1] / TKDf))) + expf(-(TKDf / T.troe[2])), XFACT);
                }
                lafp = (double)logf(RFACT) - (lnk0m > 0.0 ? log1p(exp(-lnk0m)) : log1p(exp(lnk0m)) - lnk0m);
            }
            float rc0 = 0.0f, rc1 = 0.0f;
            const double e0 = lnkf + lafp + T.lnc0 + T.order0 * LNRHO;
            const double e1 = lnkr + lafp + T.lnc1 + T.order1 * LNRHO;
            if ((T.order0 && e0 > 85.0) || (T.order1 && T.has_rev && e1 > 85.0)) out = true;
            if (T.order0) {
                float v = exp_split(e0);
                if (T.tb0 >= 0) v *= (float)sC[(SC_TB0 + T.tb0) * TILE + lane];
                for (int t = 0; t < T.ny0; ++t) v *= (float)sY[T.yk0[t] * TILE + lane];
                rc0 = v;
            }
            if (T.order1 && T.has_rev) {
                float v = exp_split(e1);
                if (T.tb1 >= 0) v *= (float)sC[(SC_TB0 + T.tb1) * TILE + lane];
                for (int t = 0; t < T.ny1; ++t) v *= (float)sY[T.yk1[t] * TILE + lane];
                rc1 = v;
            }
            sRC[(2 * p) * TILE + lane] = (double)rc0;
            sRC[(2 * p + 1) * TILE + lane] = (double)rc1;
        }
    }
    return __syncthreads_or(out) != 0;
}

struct IntArgs {
    const DevParams *P;
    const PairTab *tab;
    const PairTabM *tabm;            // the mixed form's pair table (global memory)
    double *tk, *rho, *y, *soot;     // state, updated in place: [npad], [npad], [52][npad], [2][npad]
    const double *pnd;               // p / PSTR per cell [npad]
    const int *nsub;                 // sub-steps per cell [npad]
    const int *order;                // [npad]: position -> cell (sorted by n_sub), or null (identity)
    int *next_tile;                  // work-queue counter, zero at launch
    int *passes;                     // [npad] out: update passes summed over the sub-steps
    int *status;
    double dt, sor1, tol;
    int isor, n, npad, ntile;
};

constexpr size_t INT_SMEM =
    PAIRTAB_BYTES + sizeof(double) * (size_t)(LRX * TILE + 4 * LSP * TILE + SC_N * TILE + 6 * TILE + CHEM_POLY) + 64;
static_assert(INT_SMEM <= 232448, "integrator tile does not fit in shared memory");

// A1..A6 of solveh.f:1186-1205 for one temperature range: sums over the species of Y_k times tabulated coefficients
// (a fused multiply-add each, where the reference's expression divides twice per term: with those divisions the
// T Newton of 32,768 cells took 112 us, without them 22 us).
__device__ __forceinline__ void newton_sums(const DevParams &P, int range, const double *y, int ys, double (&A)[6])
{
#pragma unroll
    for (int i = 0; i < 6; ++i) A[i] = 0.0;
#pragma unroll
    for (int k = 0; k < LSP; ++k) {
        const double2 *c = reinterpret_cast<const double2 *>(P.tco[range][k]);
        const double yk = y[k * ys];
        const double2 c0 = __ldg(c), c1 = __ldg(c + 1), c2 = __ldg(c + 2);
        A[0] = CO_FMA(c0.x, yk, A[0]);
        A[1] = CO_FMA(c0.y, yk, A[1]);
        A[2] = CO_FMA(c1.x, yk, A[2]);
        A[3] = CO_FMA(c1.y, yk, A[3]);
        A[4] = CO_FMA(c2.x, yk, A[4]);
        A[5] = CO_FMA(c2.y, yk, A[5]);
    }
}
static_assert(offsetof(DevParams, tco) % 16 == 0, "the Newton's coefficients are read two at a time");

// A1 T + A2 T^2 + ... + A6
__device__ __forceinline__ double newton_h(const double (&A)[6], double T)
{
    return CO_FMA(CO_FMA(CO_FMA(CO_FMA(CO_FMA(A[4], T, A[3]), T, A[2]), T, A[1]), T, A[0]), T, A[5]);
}

// Total enthalpy of a cell at its own temperature, in the units of ENTH in
// solveh.f:1186-1205; y has stride ys between species.
__device__ __forceinline__ double enthalpy_total(const DevParams &P, double tk, const double *y, int ys)
{
    const double TKD = tk * P.TSTR;
    double A[6];
    newton_sums(P, TKD > UC_TPOL1 ? 1 : 0, y, ys, A);
    return newton_h(A, TKD) * P.GASC / P.WMSTR;
}

// Newton for T at total enthalpy ENTH (solveh.f:1186-1234). Returns tk;
// sets *conv to false if 100 iterations did not meet the step tolerance. The multiply-adds are written out: a sum
// of two products may be contracted either way, and the two forms of the integration compute a cell alike.
__device__ __forceinline__ double temperature_at(const DevParams &P, double tk, const double *y, int ys, double ENTH,
                                                 bool *conv)
{
    double TPOLY = UC_TPOL1;
    double TKD = tk * P.TSTR;
    double A[6];
#pragma unroll 1
    for (int range = 0;; range = 1) {
        if (TKD > TPOLY) TKD = TPOLY / 2.0;
        newton_sums(P, range, y, ys, A);
        const double FUNT = newton_h(A, TPOLY) * P.GASC / P.WMSTR - ENTH;
        if (FUNT >= 1.0e-07 || range == 1) break;
        if (TKD <= TPOLY) TKD = UC_TPOL2 / 2.0;
        TPOLY = UC_TPOL2;
    }
    const double h0 = ENTH * P.WMSTR / P.GASC;
    *conv = false;
#pragma unroll 1
    for (int it = 1; it <= 100; ++it) {
        const double den = CO_FMA(CO_FMA(CO_FMA(CO_FMA(5.0 * A[4], TKD, 4.0 * A[3]), TKD, 3.0 * A[2]), TKD, 2.0 * A[1]), TKD, A[0]);
        const double DTKD = (newton_h(A, TKD) - h0) / den;
        if (fabs(DTKD) <= (double)0.001f) { *conv = true; break; }
        TKD = TKD - DTKD;
    }
    if (TKD > UC_TPOL2) TKD = UC_TPOL2;
    if (TKD < P.TKDMIN) TKD = P.TKDMIN;
    return TKD / P.TSTR;
}

// rho of an ideal gas at p / PSTR = pnd (main:1056-1062)
__device__ __forceinline__ double gas_density(const DevParams &P, double tk, double pnd, const double *y, int ys)
{
    double r0 = 0.0, r1 = 0.0;
#pragma unroll
    for (int k = 0; k < LSP; k += 2) {
        r0 = CO_FMA(__ldg(P.tbw + k), y[k * ys], r0);
        r1 = CO_FMA(__ldg(P.tbw + k + 1), y[(k + 1) * ys], r1);
    }
    return pnd / (P.BETA1 * tk * (r0 + r1));
}

// Sub-step count per cell from the omega of the start state (QDSP rows):
// x = max over Y_k > y_tau of dt*|QDSP_k|/(RCONV*rho*Y_k), n_sub = clamp(ceil(x/c_tau), 1, nsub_max).
__global__ void nsub_kernel(const DevParams *Pp, const double *rho, const double *y, const double *qdsp, int n, int npad,
                            double dt, double c_tau, double y_tau, int nsub_max, int *nsub)
{
    const DevParams &P = *Pp;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < npad; c += gridDim.x * blockDim.x) {
        double x = 0.0;
        for (int k = 0; k < LSP; ++k) {
            const double yk = y[(size_t)k * npad + c];
            if (yk > y_tau) {
                const double v = dt * fabs(qdsp[(size_t)k * npad + c]) / (P.RCONV * rho[c] * yk);
                if (!(v <= x)) x = v;
            }
        }
        const double m = ceil(x / c_tau);
        nsub[c] = (m != m || m >= (double)nsub_max) ? nsub_max : (m < 1.0 ? 1 : (int)m);
    }
}

// Total enthalpy of each cell of a field (held while the composition changes)
__global__ void hold_enthalpy_kernel(const DevParams *Pp, const double *tk, const double *y, int npad, double *enth)
{
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < npad; c += gridDim.x * blockDim.x)
        enth[c] = enthalpy_total(*Pp, tk[c], y + c, npad);
}

// T from the held total enthalpy and the current Y (solveh.f:1186-1234), then rho
// from the ideal gas at the cell pressure (main:1056-1062); the first *nlive cells when nlive is given,
// else all npad
__global__ void temperature_held_kernel(const DevParams *Pp, const double *enth, const double *y, const double *pnd,
                                        int npad, double *tk, double *rho, int *status, const int *nlive = nullptr)
{
    const DevParams &P = *Pp;
    const int nc = nlive ? *nlive : npad;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += gridDim.x * blockDim.x) {
        bool conv;
        const double t = temperature_at(P, tk[c], y + c, npad, enth[c], &conv);
        if (!conv && status) atomicCAS(status, ST_OK, ST_NEWTON_NOCONV);
        tk[c] = t;
        rho[c] = gas_density(P, t, pnd[c], y + c, npad);
    }
}

// ---- stable counting sort of positions by n_sub, largest first.
// Chunk j of `chunk` cells is owned by CTA j; key = nsub_max - n_sub. A chunk is scattered by one warp, 32 cells
// after 32 (67 us for 4096 cells, 14 us for 512), so small fields have small chunks: up to 256 of them to 1,048,576
// cells, beyond that more of 4096; one CTA scans their counts. The order does not depend on the chunks.
__host__ __device__ constexpr int sort_chunk(int n) { return n <= 256 * 512 ? 512 : n <= 256 * 2048 ? 2048 : 4096; }
constexpr int SORT_MAXBIN = 1024;

__global__ void sort_count_kernel(const int *nsub, int n, int nsub_max, int chunk, int nchunk, int *hist)
{
    __shared__ int h[SORT_MAXBIN + 1];
    const int j = blockIdx.x;
    for (int b = threadIdx.x; b <= nsub_max; b += blockDim.x) h[b] = 0;
    __syncthreads();
    const int c0 = j * chunk, c1 = min(n, c0 + chunk);
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) atomicAdd(&h[nsub_max - nsub[c]], 1);
    __syncthreads();
    for (int b = threadIdx.x; b <= nsub_max; b += blockDim.x) hist[(size_t)b * nchunk + j] = h[b];
}

// Exclusive scan of hist in (bin, chunk) order, in place; one CTA.
__global__ void sort_scan_kernel(int *hist, int total)
{
    __shared__ int s_carry;
    __shared__ int s_warp[32];
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int base = 0; base < total; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const int v = i < total ? hist[i] : 0;
        int incl = v;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) s_warp[w] = incl;
        __syncthreads();
        if (threadIdx.x == 0) {
            int acc = 0;
            for (int q = 0; q < nw; ++q) { const int t = s_warp[q]; s_warp[q] = acc; acc += t; }
        }
        __syncthreads();
        const int excl = s_carry + s_warp[w] + incl - v;
        if (i < total) hist[i] = excl;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) s_carry = excl + v;
        __syncthreads();
    }
}

// Scatter: one warp per chunk walks its cells in index order (stable).
__global__ void sort_scatter_kernel(const int *nsub, int n, int npad, int nsub_max, int chunk, int nchunk, const int *offs,
                                    int *order)
{
    __shared__ int off[SORT_MAXBIN + 1];
    const int j = blockIdx.x, lane = threadIdx.x;
    for (int b = lane; b <= nsub_max; b += 32) off[b] = offs[(size_t)b * nchunk + j];
    __syncwarp();
    const int c0 = j * chunk, c1 = min(n, c0 + chunk);
    for (int base = c0; base < c1; base += 32) {
        const int c = base + lane;
        const bool v = c < c1;
        const int key = v ? nsub_max - nsub[c] : -1;
        const unsigned act = __ballot_sync(0xffffffffu, v);
        const unsigned peers = __match_any_sync(0xffffffffu, key) & act;
        const int rank = __popc(peers & ((1u << lane) - 1));
        int pos = 0;
        if (v) pos = off[key] + rank;
        __syncwarp();
        if (v && rank == 0) off[key] += __popc(peers);
        __syncwarp();
        if (v) order[pos] = c;
    }
    // positions n..npad-1 keep the padding cells
    if (j == 0)
        for (int c = n + lane; c < npad; c += 32) order[c] = c;
}

// ---- rounds form: the cells in n_sub order (longest first) advance one sub-step per round; round r
// (0-based) advances the cells with n_sub > r, a prefix of that order. After the sort's scan, hist[b * nchunk]
// counts the cells whose key nsub_max - n_sub is below b, so round r has hist[(nsub_max - r) * nchunk] cells.
__global__ void round_counts_kernel(const int *hist, int nchunk, int nsub_max, int *cells, int *tiles)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nsub_max; r += gridDim.x * blockDim.x) {
        const int c = hist[(size_t)(nsub_max - r) * nchunk];
        cells[r] = c;
        tiles[r] = (c + TILE - 1) / TILE;
    }
}

__global__ void iota_kernel(int *v, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v[i] = i;
}

// The state of the rounds form, position by position: y [52][npad], tk, rho, pnd, soot [2][npad], enth in
// doubles; nsub, passes (summed over the sub-steps), last (passes of the last sub-step) and ord (the cell at
// the position) in ints. Two such buffers alternate: between rounds the live cells are re-ordered.
struct RoundState {
    double *y, *tk, *rho, *pnd, *soot, *enth;
    int *nsub, *passes, *last, *ord;
};

// The state in n_sub order: position pos holds cell order[pos] (pos < n; the padding cells keep their place)
__global__ void gather_state_kernel(const int *order, int n, int npad, const double *y, const double *tk,
                                    const double *rho, const double *pnd, const double *soot, const int *nsub,
                                    RoundState d)
{
    for (int pos = blockIdx.x * blockDim.x + threadIdx.x; pos < npad; pos += gridDim.x * blockDim.x) {
        const int c = pos < n ? order[pos] : pos;
        for (int k = 0; k < LSP; ++k) d.y[(size_t)k * npad + pos] = y[(size_t)k * npad + c];
        d.tk[pos] = tk[c];
        d.rho[pos] = rho[c];
        d.pnd[pos] = pnd[c];
        d.soot[pos] = soot[c];
        d.soot[npad + pos] = soot[(size_t)npad + c];
        d.nsub[pos] = nsub[c];
        d.passes[pos] = 0;
        d.last[pos] = 0;
        d.ord[pos] = c;
    }
}

// Sort key of the positions of round r for round r + 1: the cells that go on (n_sub > r + 1) by the passes
// their last sub-step took, most first (a cell's pass count changes little from one sub-step to the next,
// so warps then hold cells that stop together), the others after them.
constexpr int ROUND_KEYS = 102;            // 0..99: 100 - min(passes, 100) of a live cell; 101: done
__global__ void round_key_kernel(const int *nsub, const int *last, const int *nlive, int r, int *key)
{
    const int n = *nlive;
    for (int pos = blockIdx.x * blockDim.x + threadIdx.x; pos < n; pos += gridDim.x * blockDim.x)
        key[pos] = nsub[pos] > r + 1 ? 100 - min(max(last[pos], 1), 100) : ROUND_KEYS - 1;
}

// Stable counting sort of the first *nlive keys (chunks of sort_chunk(n); hist [nbins][nchunk], scanned by
// sort_scan_kernel in between): perm[new position] = old position.
__global__ void key_count_kernel(const int *key, const int *nlive, int nbins, int chunk, int nchunk, int *hist)
{
    __shared__ int h[SORT_MAXBIN];
    const int j = blockIdx.x, n = *nlive;
    for (int b = threadIdx.x; b < nbins; b += blockDim.x) h[b] = 0;
    __syncthreads();
    const int c0 = j * chunk, c1 = min(n, c0 + chunk);
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) atomicAdd(&h[key[c]], 1);
    __syncthreads();
    for (int b = threadIdx.x; b < nbins; b += blockDim.x) hist[(size_t)b * nchunk + j] = h[b];
}

__global__ void key_scatter_kernel(const int *key, const int *nlive, int nbins, int chunk, int nchunk, const int *offs,
                                   int *perm)
{
    __shared__ int off[SORT_MAXBIN];
    const int j = blockIdx.x, lane = threadIdx.x, n = *nlive;
    for (int b = lane; b < nbins; b += 32) off[b] = offs[(size_t)b * nchunk + j];
    __syncwarp();
    const int c0 = j * chunk, c1 = min(n, c0 + chunk);
    for (int base = c0; base < c1; base += 32) {
        const int c = base + lane;
        const bool v = c < c1;
        const int k = v ? key[c] : -1;
        const unsigned act = __ballot_sync(0xffffffffu, v);
        const unsigned peers = __match_any_sync(0xffffffffu, k) & act;
        const int rank = __popc(peers & ((1u << lane) - 1));
        int pos = 0;
        if (v) pos = off[k] + rank;
        __syncwarp();
        if (v && rank == 0) off[k] += __popc(peers);
        __syncwarp();
        if (v) perm[pos] = c;
    }
}

// d[pos] = s[perm[pos]] for the first *nlive positions, d[pos] = s[pos] beyond; blockIdx.y: one of the Y rows or,
// last, the other values
constexpr int PERMUTE_ROWS = LSP + 1;
__global__ void permute_state_kernel(const int *perm, const int *nlive, int npad, RoundState s, RoundState d)
{
    const int pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= npad) return;
    const int q = pos < *nlive ? perm[pos] : pos;
    if (blockIdx.y < LSP) {
        d.y[(size_t)blockIdx.y * npad + pos] = s.y[(size_t)blockIdx.y * npad + q];
        return;
    }
    d.tk[pos] = s.tk[q];
    d.rho[pos] = s.rho[q];
    d.pnd[pos] = s.pnd[q];
    d.soot[pos] = s.soot[q];
    d.soot[npad + pos] = s.soot[npad + q];
    d.enth[pos] = s.enth[q];
    d.nsub[pos] = s.nsub[q];
    d.passes[pos] = s.passes[q];
    d.last[pos] = s.last[q];
    d.ord[pos] = s.ord[q];
}

// back to cell order (the first n positions)
__global__ void scatter_state_kernel(int n, int npad, RoundState s, double *y, double *tk, double *rho,
                                     double *soot, int *passes)
{
    for (int pos = blockIdx.x * blockDim.x + threadIdx.x; pos < n; pos += gridDim.x * blockDim.x) {
        const int c = s.ord[pos];
        for (int k = 0; k < LSP; ++k) y[(size_t)k * npad + c] = s.y[(size_t)k * npad + pos];
        tk[c] = s.tk[pos];
        rho[c] = s.rho[pos];
        soot[c] = s.soot[pos];
        soot[(size_t)npad + c] = s.soot[npad + pos];
        passes[c] = s.passes[pos];
    }
}

// A pass of the tile's update with RC and Y in shared memory (the warps of one tile as in update_tr_kernel:
// two sum, one closes; see there). The closing warp writes species k while the others sum species k + 1,
// which reads neither value of k but through the copies YOS.
struct IntTile {
    const double *rc;              // [544][32] at the lane's column, and so the others
    double *y;                     // [52][32]
    const double *ry0;             // [52][32]: rho * Y at the sub-step start
    double *part;                  // [slots][32] pairs
    const double *sour;            // [6][32]
    int *flag;
};
// the kernel's dynamic shared memory, laid out in this order
constexpr size_t INT_OFF_RC = PAIRTAB_BYTES, INT_OFF_Y = INT_OFF_RC + sizeof(double) * LRX * TILE,
                 INT_OFF_G = INT_OFF_Y + sizeof(double) * LSP * TILE, INT_OFF_Y0 = INT_OFF_G + sizeof(double) * 2 * LSP * TILE,
                 INT_OFF_C = INT_OFF_Y0 + sizeof(double) * LSP * TILE, INT_OFF_S = INT_OFF_C + sizeof(double) * SC_N * TILE,
                 INT_OFF_POLY = INT_OFF_S + sizeof(double) * 6 * TILE,
                 INT_OFF_BAR = INT_OFF_POLY + sizeof(double) * CHEM_POLY, INT_OFF_QUIT = INT_OFF_BAR + 8;
static_assert(INT_OFF_QUIT + 8 <= INT_SMEM, "shared memory of the integrator");
static_assert(UC_CO_SLOTS <= LSP, "the partial sums take the place of the Gibbs functions");
// from the shared array itself, so that a function that is not inlined reads it with shared-memory loads
__device__ __forceinline__ IntTile int_tile()
{
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    return {reinterpret_cast<double *>(smem + INT_OFF_RC) + lane, reinterpret_cast<double *>(smem + INT_OFF_Y) + lane,
            reinterpret_cast<double *>(smem + INT_OFF_Y0) + lane, reinterpret_cast<double *>(smem + INT_OFF_G) + 2 * lane,
            reinterpret_cast<double *>(smem + INT_OFF_S) + lane, reinterpret_cast<int *>(smem + INT_OFF_QUIT)};
}
#define CO_WAIT_Y(set) asm volatile("bar.sync %0, 96;" ::"n"(1 + (set)) : "memory")
#define CO_ARRIVE_Y(set) asm volatile("bar.arrive %0, 96;" ::"n"(1 + (set)) : "memory")
#define CO_WAIT_P(set) asm volatile("bar.sync %0, 96;" ::"n"(3 + (set)) : "memory")
#define CO_ARRIVE_P(set) asm volatile("bar.arrive %0, 96;" ::"n"(3 + (set)) : "memory")
#define YO(k) t.y[(k) * TILE]
#define YOS(m) ysh[m]
#define SOUR(m) t.sour[(m) * TILE]
#define RCS2(i) make_double2(t.rc[(UC_CO_NT + 2 * (i)) * TILE], t.rc[(UC_CO_NT + 2 * (i) + 1) * TILE])
#define TM_LD2(b, q, col, p)                                    \
    do {                                                        \
        bank##b[2 * (q)] = t.rc[2 * (p) * TILE];                \
        bank##b[2 * (q) + 1] = t.rc[(2 * (p) + 1) * TILE];      \
    } while (0)
#define TM_LD4(b, q, col, p0, p1)       \
    do {                                \
        TM_LD2(b, q, col, p0);          \
        TM_LD2(b, (q) + 1, col, p1);    \
    } while (0)
#define TM_LD8(b, q, col, p0, p1, p2, p3)     \
    do {                                      \
        TM_LD4(b, q, col, p0, p1);            \
        TM_LD4(b, (q) + 2, col, p2, p3);      \
    } while (0)
#define TM_WAIT(b, n) do { } while (0)
#define RCT(b, i) bank##b[i]
#define CO_PUT(slot, a, b) co_st2(t.part + (slot) * (2 * TILE), a, b)
#define CO_GET(buf, k, mine, now) do { } while (0)
#define CO_CHECK()                                              \
    do {                                                        \
        asm volatile("bar.sync 5, 96;" ::: "memory");          \
        if (co_ldi(t.flag)) return false;                       \
    } while (0)
template <int W>
__device__ __noinline__ bool int_sums()
{
    const IntTile t = int_tile();
    double ysh[UC_CO_NSHADOW], bank0[2 * UC_CO_SEG], bank1[2 * UC_CO_SEG];
    if (W == 0) UC_CO_SUMS_0();
    else UC_CO_SUMS_1();
    return true;
}
#define CO_TAKE(slot, a, b) co_ld2(t.part + (slot) * (2 * TILE), a, b)
#define CO_QUOT(n, d) co_quot(n, d)
#define CO_GIVE(buf, k) do { } while (0)
#define RY0(k) t.ry0[(k) * TILE]
#define DTW(k) (dt * prm.WM[k])
#define CO_PF(s, k) do { } while (0)
#define FSS(s) 0.0
#define FNS(s) 0.0
#define CO_TAIL(k) do { if (fnew < 0.0) fnew = 0.0; if (!done) t.y[(k) * TILE] = fnew; } while (0)
__device__ __noinline__ bool int_close(const DevParams &prm, double rho, double dt, double sor1, double sor2,
                                       bool done, double &rsd)
{
    const IntTile t = int_tile();
    UC_CO_CLOSE();
    return true;
}
// before the first pass: the last run's values stand in shared memory already
__device__ __forceinline__ void int_close_begin() { CO_ARRIVE_Y(UC_CO_LAST_SET); }
#undef CO_WAIT_Y
#undef CO_ARRIVE_Y
#undef CO_WAIT_P
#undef CO_ARRIVE_P
#undef CO_QUOT
#undef YO
#undef YOS
#undef SOUR
#undef RCS2
#undef TM_LD2
#undef TM_LD4
#undef TM_LD8
#undef TM_WAIT
#undef RCT
#undef CO_PUT
#undef CO_GET
#undef CO_CHECK
#undef CO_TAKE
#undef CO_GIVE
#undef RY0
#undef DTW
#undef CO_PF
#undef FSS
#undef FNS
#undef CO_TAIL

// MIXED: the rates of every sub-step in the mixed form (tile_rates_mixed; a tile with a rate beyond the
// FP32 range is recomputed in FP64), the update, closure and Newton in FP64 as in the FP64 form.
template <int NW, bool MIXED>
__global__ void __launch_bounds__(NW * 32, 1) integrate_fp64_kernel(const IntArgs a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    PairTab *sTab = reinterpret_cast<PairTab *>(smem);
    double *sRC = reinterpret_cast<double *>(smem + INT_OFF_RC);      // [544][32]
    double *sY = reinterpret_cast<double *>(smem + INT_OFF_Y);        // [52][32] current Y
    double *sYN = reinterpret_cast<double *>(smem + INT_OFF_G);       // [52][32] Gibbs scratch / partial sums
    double *sY0 = reinterpret_cast<double *>(smem + INT_OFF_Y0);      // [52][32] rho * Y at the sub-step start
    double *sC = reinterpret_cast<double *>(smem + INT_OFF_C);        // [SC_N][32]
    double *sS = reinterpret_cast<double *>(smem + INT_OFF_S);        // [6][32] soot sources
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + INT_OFF_BAR);
    int *s_quit = reinterpret_cast<int *>(smem + INT_OFF_QUIT);       // no more passes of this sub-step
    __shared__ int s_tile, s_smax;
    const DevParams &P = *a.P;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    if (tid == 0) mbar_init(bar, 1);
    __syncthreads();
    if (tid == 0) {
        mbar_expect_tx(bar, PAIRTAB_BYTES);
        constexpr int CH = 8192;
        for (int off = 0; off < PAIRTAB_BYTES; off += CH) {
            const int bytes = PAIRTAB_BYTES - off < CH ? PAIRTAB_BYTES - off : CH;
            bulk_g2s(reinterpret_cast<unsigned char *>(sTab) + off, reinterpret_cast<const unsigned char *>(a.tab) + off,
                     bytes, bar);
        }
    }
    if (!mbar_wait_bounded(bar, 0, 1 << 20)) {
        if (tid == 0) atomicExch(a.status, ST_TMA_TIMEOUT);
        mbar_wait_bounded(bar, 0, 1 << 20);
        return;
    }
    double *sPoly = reinterpret_cast<double *>(smem + INT_OFF_POLY);  // [52][14]
    for (int i = tid; i < CHEM_POLY; i += NW * 32) sPoly[i] = P.poly[i];
    const size_t np = a.npad;
    const double sor1 = a.sor1, sor2 = 1.0 - a.sor1;

    for (;;) {
        if (tid == 0) s_tile = atomicAdd(a.next_tile, 1);
        __syncthreads();
        const int tile = s_tile;
        if (tile >= a.ntile) break;
        const int pos = tile * TILE + lane;
        size_t cell = a.order ? (size_t)a.order[pos] : (size_t)pos;
        if (cell >= (size_t)a.npad) {          // a broken order: keep the access in bounds and report it
            cell = pos;
            atomicExch(a.status, ST_BAD_ORDER);
        }
        // ---- load the tile's state (gathered through the order)
        for (int k = warp; k < LSP; k += NW) sY[k * TILE + lane] = a.y[k * np + cell];
        double tk = 0.0, rho = 0.0, pnd = 0.0, s1 = 0.0, s2 = 0.0, ENTH0 = 0.0;
        int ns = 0, npass = 0;
        bool tconv = true;
        if (warp == 0) {
            tk = a.tk[cell];
            rho = a.rho[cell];
            pnd = a.pnd[cell];
            s1 = a.soot[cell];
            s2 = a.soot[np + cell];
            ns = a.nsub[cell];
        }
        __syncthreads();
        if (warp == 0) {
            ENTH0 = enthalpy_total(P, tk, sY + lane, TILE);
            int m = ns;
            for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (lane == 0) s_smax = m;
        }
        __syncthreads();
        const int smax = s_smax;
        for (int st = 0; st < smax; ++st) {
            if (warp == 0) tile_scalars(P, sC, lane, tk, rho, s1, s2);
            __syncthreads();
            if (!MIXED || tile_rates_mixed<NW>(P, a.tabm, sRC, sY, sYN, sC, sS, TILE, lane, lane, warp))
                tile_rates_fp64<NW>(P, sTab, sPoly, sY, sYN, sC, sS, TILE, lane, lane, warp, false,
                                    [&](int p, double rc0, double rc1) {
                                        sRC[(2 * p) * TILE + lane] = rc0;
                                        sRC[(2 * p + 1) * TILE + lane] = rc1;
                                    });
            __syncthreads();
            if (warp == 1) { while (int_sums<0>()) {} }
            else if (warp == 2) { while (int_sums<1>()) {} }
            else if (warp == 0) {
                const double dt = a.dt / (double)ns;
                double so[6];
#pragma unroll
                for (int m = 0; m < 6; ++m) so[m] = sS[m * TILE + lane];
                for (int k = 0; k < LSP - 1; ++k) sY0[k * TILE + lane] = rho * sY[k * TILE + lane];
                const double s10 = s1, s20 = s2;
                bool done = st >= ns;
                int_close_begin();
                for (int pass = 1;; ++pass) {
                    const int quit = pass > a.isor || __all_sync(0xffffffffu, done);
                    if (lane == 0) *s_quit = quit;
                    double rsd = 0.0;
                    if (!int_close(P, rho, dt, sor1, sor2, done, rsd)) break;
                    double ys[22], n1, n2;
                    ys[1] = sY[1 * TILE + lane]; ys[3] = sY[3 * TILE + lane];
                    ys[4] = sY[4 * TILE + lane]; ys[21] = sY[21 * TILE + lane];
                    co_soot(ys, so, s10, s20, rho, dt, P.WMSTR, sor1, sor2, s1, s2, n1, n2, rsd);
                    if (!done) {
                        s1 = n1;
                        s2 = n2;
                        ++npass;
                        if (rsd / (double)(LSP - 1) <= a.tol) done = true;
                    }
                }
            }
            if (warp == 0 && st < ns) {
                // N2 closure and renormalisation (solvesp.f:2839-2915)
                double ft = sY[lane];
                for (int k = 1; k < LSP - 1; ++k) ft = ft + sY[k * TILE + lane];
                ft = ft + s1;
                double n2 = 1.0 - ft;
                if (ft > 1.0) {
                    for (int k = 0; k < LSP - 1; ++k) sY[k * TILE + lane] = sY[k * TILE + lane] / ft;
                    s1 = s1 / ft;
                    n2 = 0.0;
                }
                sY[(LSP - 1) * TILE + lane] = n2;
                bool conv;
                tk = temperature_at(P, tk, sY + lane, TILE, ENTH0, &conv);
                tconv = tconv && conv;
                rho = gas_density(P, tk, pnd, sY + lane, TILE);
            }
            __syncthreads();
        }
        // ---- store
        for (int k = warp; k < LSP; k += NW) a.y[k * np + cell] = sY[k * TILE + lane];
        if (warp == 0) {
            a.tk[cell] = tk;
            a.rho[cell] = rho;
            a.soot[cell] = s1;
            a.soot[np + cell] = s2;
            a.passes[cell] = npass;
            if (!tconv && a.status) atomicCAS(a.status, ST_OK, ST_NEWTON_NOCONV);
        }
        __syncthreads();
    }
}

}  // namespace uc
