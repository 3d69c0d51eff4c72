// Point-implicit species update (src/lib/solvesp.f:85-2915) with each tile's
// rate coefficients held on chip across passes: the FP64 default.
//
// Within one update call the cells are independent (the transport terms are
// frozen at the start), and only the stopping test couples them: the pass
// loop ends at the first pass whose residual sum|dY| over all cells meets the
// tolerance (solvesp.f:2833). The kernel therefore runs the passes in chunks
// of C: a 32-cell tile's RC block [544][32] is staged on chip once, C passes of
// that tile run back to back, the tile's residual of each pass and, for all but
// the last pass of the chunk, a snapshot of the tile's Y are recorded; then the
// next tile. After a grid barrier every block sums the residual partials of each
// pass of the chunk in the same order and finds the first pass that met the
// tolerance; if it lies inside the chunk, its snapshot becomes the result. The RC
// plane is read from HBM once per chunk instead of once per pass.
//
// Three warps work on one tile, three tiles on an SM (417 KB of RC: 336 rows of each
// tile in tensor memory, 208 in shared memory). Two warps form the sums of
// the species, each from the terms of its own row pairs, and the third
// closes them (UC_CO_SUMS_*, UC_CO_CLOSE of the generated program), in runs of up to
// three species that do not enter one another's sums. While one run is closed, the other warps
// sum the next: what a species of the run multiplies there is summed apart and waits for it in one
// multiply-add. The closing warp hands new values over and goes on (bar.arrive); it
// waits only for the next run's partial sums, the summing warps only for the run before
// the one being closed.
//
// What bounds it: latency, and the fetching of instructions. The species order is sequential
// (Gauss-Seidel), and the program is straight-line code that no cache near the warps holds (108 KB a
// pass). Measured at 1,048,576 cells x 100 passes: one warp per tile running the ungrouped program (9,260
// instructions a pass, 148 KB) 168 ms; the grouped sums alone, still one warp per tile (6,800 instructions)
// 106 ms; this form 90.5 ms, and 7.0 us instead of 21 us for a pass of a tile that has the GPU to itself. A third
// summing warp per tile (7,450 instructions, 119 KB) ran the large field as fast and a field of one tile per SM
// 5 % slower; an even split between the two summing warps took 107 ms (warps 0, 4 and 8 share a scheduler),
// shares of 0.45, 0.35 and 0.30 for the first 99, 91.5 and 90.6; beginning the passes of a block's tiles together
// 99 ms (they then stage together too).
//
// A tensor-memory access reaches the lanes of its warp's quarter only (warp
// index mod 4). Warps 0, 4 and 8, in quarter 0, are the first summing warps of the three tiles (40 pairs
// each); warps 1, 2 and 3, each alone in its quarter, the second ones (128 pairs each); warps 5, 6 and 7
// close and hold no rows. Rows 336..543 lie in shared memory, where every
// warp of the tile reads any of them. Row pairs (the forward and reverse coefficient of
// a reaction, used together) are read by one 16-byte load.
//
// The residual is summed per tile, then per warp in tile order, per block in tile-slot order
// and over the blocks in block order.
#pragma once
#include <cooperative_groups.h>
#include <cuda.h>                       // CUtensorMap (the type only; encoded through the runtime's entry point)

#include "uc_device.cuh"
#include "update_kernel.cuh"
#include "generated/update_program_co.cuh"

namespace uc {

constexpr int TR_TILES = 3;                        // tiles in flight per block
constexpr int TR_TILE_WARPS = UC_CO_SUMS + 1;
constexpr int TR_WARPS = TR_TILES * TR_TILE_WARPS;
constexpr int TR_CHUNK_MAX = 32;
constexpr int TR_SNAP_ROWS = LSP - 1 + 2;          // Y of species 1..51 and the two soot scalars
// shared memory of a tile (doubles): RC rows, rho * Y of the old level, partial sums [slot][32] pairs, new Y
// [2 sets][3][32]
constexpr size_t TR_OFF_RY0 = (size_t)UC_CO_NS * TILE;
constexpr size_t TR_OFF_PART = TR_OFF_RY0 + (size_t)(LSP - 1) * TILE;
constexpr size_t TR_OFF_Y = TR_OFF_PART + UC_CO_SLOTS * TILE * 2;
constexpr size_t TR_TILE_DOUBLES = TR_OFF_Y + 6 * TILE;
constexpr size_t TR_SMEM = TR_TILES * TR_TILE_DOUBLES * sizeof(double);
constexpr uint32_t TR_BOX_T = UC_CO_PIECE, TR_BOX_S = UC_CO_NS;    // rows per box of the tiled bulk copies
static_assert(TR_SMEM + 2048 <= 232448, "shared memory of the tile-resident update");
static_assert(TR_TILE_DOUBLES * sizeof(double) % 128 == 0, "alignment of the bulk copies");
static_assert(UC_CO_NT == 2 * UC_CO_PIECE && UC_CO_PIECE <= UC_CO_NS && UC_CO_NS <= 256 && UC_CO_NS % 16 == 0,
              "the tensor-memory rows pass through the shared-memory rows' place in two pieces");
static_assert(UC_CO_NT + UC_CO_NS == LRX, "every row of the plane is staged");
static_assert(UC_CO_SUMS == 2 && 2 * (UC_CO_PAIRS_0 + UC_CO_PAIRS_1) == UC_CO_PIECE, "each pair of a piece has one owner");
static_assert(UC_CO_PAIRS_0 % 2 == 0, "a warp's columns begin at a multiple of 16");
static_assert(TR_TILES * 8 * UC_CO_PAIRS_0 <= 512 && 8 * UC_CO_PAIRS_1 <= 512, "tensor-memory columns of a quarter");
static_assert(UC_CO_LAST == LSP - 4, "argon, helium and nitrogen follow the last block with terms");

struct TrArgs {
    double *snap;          // [chunk - 1][TR_SNAP_ROWS][npad]
    double *partial;       // [2][TR_CHUNK_MAX][gridDim.x]
    int chunk;             // passes per chunk, 1..TR_CHUNK_MAX
    int *status;
    int adapt;             // longer chunks (up to TR_CHUNK_MAX) while the previous call's count says that
                           // many passes are still to come
};

#ifndef UC_TR_WAIT_TRIES
#define UC_TR_WAIT_TRIES (1 << 22)
#endif

// One tile as its three warps see it; pointers already point at the lane's column.
struct CoTile {
    double *slot;          // RC rows 336..543: [208][32], after staging [104][32] pairs
    double *ry0;           // [51][32]
    double *part;          // [slots][32] pairs
    double *yb;            // [6][32]
    uint64_t *bar;         // staging
    int *flag;             // per-cell form: no more passes
    uint32_t tcol;         // the warp's first tensor-memory column (with its lane quarter)
    int id;                // named barriers: id, id + 1 new Y (id also: all three warps); id + 2, id + 3 partial sums
    int lane, role, tile;  // role 0, 1: summing warp, 2: the closing warp; tile: of the block's three
};

__device__ __forceinline__ CoTile co_tile(double *smem, uint64_t *bars, int *flags, uint32_t tmem)
{
    const int w = threadIdx.x >> 5, q = w & 3;
    CoTile c;
    c.lane = threadIdx.x & 31;
    c.role = q == 0 ? 0 : w < 4 ? 1 : 2;
    // the closing warp shares its scheduler with another tile's second summing warp
    const int t = c.tile = q == 0 ? w >> 2 : w < 4 ? w - 1 : (w - 4) % TR_TILES;
    double *base = smem + (size_t)t * TR_TILE_DOUBLES;
    c.slot = base;
    c.ry0 = base + TR_OFF_RY0 + c.lane;
    c.part = base + TR_OFF_PART + 2 * c.lane;
    c.yb = base + TR_OFF_Y + c.lane;
    c.bar = bars + t;
    c.flag = flags + t;
    c.id = 1 + 4 * t;
    // (from lane 0, so that the compiler knows it to be the same for the whole warp)
    c.tcol = __shfl_sync(0xffffffffu, tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(q == 0 ? 8 * UC_CO_PAIRS_0 * t : 0), 0);
    return c;
}

// Barriers of the tile's three warps. co_sync (between the passes, and where CO_CHECK stands: set 0 of the new Y is
// not in use then), where the staged rows change, has the memory clobber; those of a
// pass need none: only the exchange buffers change there, and those are read and written by volatile asm. Each
// use of a barrier is complete before its next: a warp arrives at set s again only after it has waited for
// what the other side sends once it has passed set s.
__device__ __forceinline__ void co_sync(const CoTile &c) { asm volatile("bar.sync %0, 96;" ::"r"(c.id) : "memory"); }
#define CO_WAIT_Y(set) asm volatile("bar.sync %0, 96;" ::"r"(c.id + (set)))
#define CO_ARRIVE_Y(set) asm volatile("bar.arrive %0, 96;" ::"r"(c.id + (set)))
#define CO_WAIT_P(set) asm volatile("bar.sync %0, 96;" ::"r"(c.id + 2 + (set)))
#define CO_ARRIVE_P(set) asm volatile("bar.arrive %0, 96;" ::"r"(c.id + 2 + (set)))

__device__ __forceinline__ void co_st2(double *p, double a, double b)
{
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(smem_u32(p)), "d"(a), "d"(b));
}
__device__ __forceinline__ void co_ld2(const double *p, double &a, double &b)
{
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(a), "=d"(b) : "r"(smem_u32(p)));
}
__device__ __forceinline__ void co_st1(double *p, double a)
{
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(smem_u32(p)), "d"(a));
}
__device__ __forceinline__ double co_ld1(const double *p)
{
    double a;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(a) : "r"(smem_u32(p)));
    return a;
}
__device__ __forceinline__ int co_ldi(const int *p)
{
    int a;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(a) : "r"(smem_u32(p)));
    return a;
}

__device__ __forceinline__ void tr_tmem_st2(uint32_t taddr, double a, double b)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(__double2loint(a)),
                 "r"(__double2hiint(a)), "r"(__double2loint(b)), "r"(__double2hiint(b))
                 : "memory");
}

// The loads of a bank complete at tcgen05.wait::ld; the registers loaded are operands
// of the wait, so no use of them can be scheduled before it.
#define UC_TR_R4(b, i) "+r"(b[4 * (i)]), "+r"(b[4 * (i) + 1]), "+r"(b[4 * (i) + 2]), "+r"(b[4 * (i) + 3])
#define UC_TR_WAIT(...) asm volatile("tcgen05.wait::ld.sync.aligned;" : __VA_ARGS__)
#define UC_TR_WAIT_1(b) UC_TR_WAIT(UC_TR_R4(b, 0))
#define UC_TR_WAIT_2(b) UC_TR_WAIT(UC_TR_R4(b, 0), UC_TR_R4(b, 1))
#define UC_TR_WAIT_3(b) UC_TR_WAIT(UC_TR_R4(b, 0), UC_TR_R4(b, 1), UC_TR_R4(b, 2))
#define UC_TR_WAIT_4(b) UC_TR_WAIT(UC_TR_R4(b, 0), UC_TR_R4(b, 1), UC_TR_R4(b, 2), UC_TR_R4(b, 3))
#define UC_TR_WAIT_5(b) UC_TR_WAIT(UC_TR_R4(b, 0), UC_TR_R4(b, 1), UC_TR_R4(b, 2), UC_TR_R4(b, 3), UC_TR_R4(b, 4))
#define UC_TR_WAIT_6(b) \
    UC_TR_WAIT(UC_TR_R4(b, 0), UC_TR_R4(b, 1), UC_TR_R4(b, 2), UC_TR_R4(b, 3), UC_TR_R4(b, 4), UC_TR_R4(b, 5))
static_assert(UC_CO_SEG <= 6, "UC_TR_WAIT_n for every number of pairs in a bank");

// rows [y, y + box) of the RC plane for the 32 cells from x, into shared memory as [box][32]: one tiled bulk
// copy through the plane's tensor map (no multicast), completion on the mbarrier
__device__ __forceinline__ void tr_box_load(double *dst, const CUtensorMap *map, int x, int y, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// The RC block of a tile into L2, ahead of its staging (one thread).
__device__ __forceinline__ void co_prefetch(const CUtensorMap *map_t, const CUtensorMap *map_s, int tile)
{
#define CO_PREFETCH(map, y)                                                                             \
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(                \
                     reinterpret_cast<uint64_t>(map)), "r"(tile * TILE), "r"(y) : "memory")
    CO_PREFETCH(map_t, 0);
    CO_PREFETCH(map_t, UC_CO_PIECE);
    CO_PREFETCH(map_s, UC_CO_NT);
#undef CO_PREFETCH
}

// Copy box y0.. of the plane into the tile's slot once its warps are done with what it held.
__device__ __forceinline__ void co_fetch(const CoTile &c, const CUtensorMap *map, int tile, int y0, int rows)
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    co_sync(c);
    if (c.role == UC_CO_SUMS && c.lane == 0) {
        mbar_expect_tx(c.bar, (uint32_t)(rows * TILE * sizeof(double)));
        tr_box_load(c.slot, map, tile * TILE, y0, c.bar);
    }
    __syncwarp();
}

// Wait for it; bounded: on a timeout the status is set and the copy in flight is waited for again.
__device__ __forceinline__ void co_wait(const CoTile &c, uint32_t &phase, int *status)
{
    if (!mbar_wait_bounded(c.bar, phase, UC_TR_WAIT_TRIES)) {
        if (c.lane == 0) atomicExch(status, ST_TMA_TIMEOUT);
        mbar_wait_bounded(c.bar, phase, UC_TR_WAIT_TRIES);   // let the copy in flight land
    }
    phase ^= 1u;
}

// Move a summing warp's pairs of one piece from the slot into its tensor memory.
__device__ __forceinline__ void co_to_tmem(const CoTile &c, const int16_t *pairs, const int16_t *cols, int n, int piece)
{
    const double *row = c.slot + c.lane - (ptrdiff_t)piece * UC_CO_PIECE * TILE;
#pragma unroll 4
    for (int i = piece * n; i < (piece + 1) * n; ++i) {
        const double *r = row + (ptrdiff_t)(2 * pairs[i]) * TILE;
        tr_tmem_st2(c.tcol + (uint32_t)cols[i], r[0], r[TILE]);
    }
}

// Stage one tile's RC block on chip, all rows by bulk copies: the tensor-memory rows in two pieces through
// the slot, each moved on by the warps that own its pairs, then the shared-memory rows, which stay. load() fills the
// tile's other rows, free once the first copy has been issued; the caller has begun to load its cells' Y before.
template <class F>
__device__ __forceinline__ void co_stage(const CoTile &c, const CUtensorMap *map_t, const CUtensorMap *map_s, int tile,
                                         uint32_t &phase, int *status, F load)
{
    for (int piece = 0; piece < 2; ++piece) {
        co_fetch(c, map_t, tile, piece * UC_CO_PIECE, UC_CO_PIECE);
        if (piece == 0) load();          // into the tile's other rows, free from here on
        co_wait(c, phase, status);
        if (c.role == 0) co_to_tmem(c, uc_co_pairs_0, uc_co_cols_0, UC_CO_PAIRS_0, piece);
        else if (c.role == 1) co_to_tmem(c, uc_co_pairs_1, uc_co_cols_1, UC_CO_PAIRS_1, piece);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    co_fetch(c, map_s, tile, UC_CO_NT, UC_CO_NS);
    co_wait(c, phase, status);
    // rows 2p and 2p + 1 become one row of pairs, in place, 16 rows at a time, dealt over the warps
    for (int i0 = 16 * c.role; i0 < UC_CO_NS; i0 += 16 * TR_TILE_WARPS) {
        double v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = c.slot[(size_t)(i0 + q) * TILE + c.lane];
        __syncwarp();
        double2 *pr = reinterpret_cast<double2 *>(c.slot + (size_t)i0 * TILE) + c.lane;
#pragma unroll
        for (int q = 0; q < 8; ++q) pr[q * TILE] = make_double2(v[2 * q], v[2 * q + 1]);
    }
    co_sync(c);
}

#define YO(k) yv[k]
#define YOS(m) ysh[m]
#define RCS2(i) pslot[(i) * TILE]
#define TM_LD2(b, q, col, p)                                                                          \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"                     \
                 : "=r"(bank##b[4 * (q)]), "=r"(bank##b[4 * (q) + 1]), "=r"(bank##b[4 * (q) + 2]),    \
                   "=r"(bank##b[4 * (q) + 3])                                                        \
                 : "r"(c.tcol + (uint32_t)(col)))
#define TM_LD4(b, q, col, p0, p1)                                                                     \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"     \
                 : "=r"(bank##b[4 * (q)]), "=r"(bank##b[4 * (q) + 1]), "=r"(bank##b[4 * (q) + 2]),    \
                   "=r"(bank##b[4 * (q) + 3]), "=r"(bank##b[4 * (q) + 4]), "=r"(bank##b[4 * (q) + 5]), \
                   "=r"(bank##b[4 * (q) + 6]), "=r"(bank##b[4 * (q) + 7])                            \
                 : "r"(c.tcol + (uint32_t)(col)))
#define TM_LD8(b, q, col, p0, p1, p2, p3)                                                             \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, " \
                 "%12, %13, %14, %15}, [%16];"                                                       \
                 : "=r"(bank##b[0]), "=r"(bank##b[1]), "=r"(bank##b[2]), "=r"(bank##b[3]),            \
                   "=r"(bank##b[4]), "=r"(bank##b[5]), "=r"(bank##b[6]), "=r"(bank##b[7]),            \
                   "=r"(bank##b[8]), "=r"(bank##b[9]), "=r"(bank##b[10]), "=r"(bank##b[11]),          \
                   "=r"(bank##b[12]), "=r"(bank##b[13]), "=r"(bank##b[14]), "=r"(bank##b[15])         \
                 : "r"(c.tcol + (uint32_t)(col)))
#define TM_WAIT(b, n) UC_TR_WAIT_##n(bank##b)
#define RCT(b, i) __hiloint2double((int)bank##b[2 * (i) + 1], (int)bank##b[2 * (i)])
#define CO_PUT(slot, a, b) co_st2(c.part + (slot) * (2 * TILE), a, b)
#define CO_GET(buf, k, mine, now)                                   \
    do {                                                            \
        yv[k] = co_ld1(c.yb + (buf) * TILE);                        \
        if (mine) {                                                 \
            if (now ? keep : keep_prev) *dst = yv[k];               \
            dst += step;                                            \
        }                                                           \
        if (!now && (k) == UC_CO_LAST) dst = next;                  \
    } while (0)
#define CO_CHECK()                               \
    do {                                         \
        if (CELLS) {                             \
            co_sync(c);                          \
            if (co_ldi(c.flag)) return false;    \
        }                                        \
    } while (0)

// One pass of summing warp W, which also stores the new Y of every second species (keep): dst is where the next one
// goes, step from one to the next, next where the first one of this pass goes. The last run of the pass before
// arrives in this one (keep_prev).
// Returns false when the closing warp has said that no pass is left (per-cell form).
template <int W, bool CELLS>
__device__ __forceinline__ bool co_sums(const CoTile &c, double (&yv)[LSP], double *&dst, size_t step,
                                        double *next, bool keep, bool keep_prev)
{
    const double2 *pslot = reinterpret_cast<const double2 *>(c.slot) + c.lane;
    double ysh[UC_CO_NSHADOW];
    uint32_t bank0[4 * UC_CO_SEG], bank1[4 * UC_CO_SEG];
    if (W == 0) UC_CO_SUMS_0();
    else UC_CO_SUMS_1();
    return true;
}

// The last run of the last pass: wait for it and store this warp's third.
template <int W>
__device__ __forceinline__ void co_sums_end(const CoTile &c, double *dst, size_t step, bool keep)
{
    CO_WAIT_Y(UC_CO_LAST_SET);
#define CO_LAST_SPECIES(buf, k) \
    if ((k) % UC_CO_SUMS == W) {                                       \
        if (keep) *dst = co_ld1(c.yb + (buf) * TILE);         \
        dst += step;                                          \
    }
    UC_CO_LAST_RUN();
#undef CO_LAST_SPECIES
}
#undef CO_PUT
#undef CO_GET

#define SOUR(m) so[m]
#define CO_TAKE(slot, a, b) co_ld2(c.part + (slot) * (2 * TILE), a, b)
#define CO_GIVE(buf, k) co_st1(c.yb + (buf) * TILE, yv[k])
#define CO_QUOT(n, d) co_quot(n, d)
#define RY0(k) c.ry0[(k) * TILE]
#define DTW(k) (CELLS ? dt * s_w[k] : s_w[k])
#define CO_PF(s, k)                                                                        \
    do {                                                                                   \
        if (FACES) {                                                                       \
            fss[s] = face_sum ? __ldg(face_sum + (size_t)(k) * np) : 0.0;                  \
            fns[s] = face_nbr ? __ldg(face_nbr + (size_t)(k) * np) : 0.0;                  \
        }                                                                                  \
    } while (0)
#define FSS(s) fss[s]
#define FNS(s) fns[s]
#define CO_TAIL(k) do { if (fnew < 0.0) fnew = 0.0; if (!CELLS || !done) yv[k] = fnew; } while (0)

// Before the first pass of a tile: the last run's values, as every pass begins with them.
__device__ __forceinline__ void co_close_begin(const CoTile &c, const double (&yv)[LSP])
{
#define CO_LAST_SPECIES(buf, k) CO_GIVE(buf, k)
    UC_CO_LAST_RUN();
#undef CO_LAST_SPECIES
    CO_ARRIVE_Y(UC_CO_LAST_SET);
}

// One pass of the closing warp; face_sum, face_nbr at the lane's cell (or null). s_w: dt * WM (CELLS: WM); so:
// SOUR 1..6.
template <bool FACES, bool CELLS>
__device__ __forceinline__ bool co_close(const CoTile &c, double (&yv)[LSP], const double (&so)[6], const double *s_w,
                                         double rho, double dt, double sor1, double sor2, const double *face_sum,
                                         const double *face_nbr, size_t np, bool done, double &rsd)
{
    double fss[UC_CO_WINDOW], fns[UC_CO_WINDOW];
#pragma unroll
    for (int i = 0; i < UC_CO_WINDOW; ++i) fss[i] = fns[i] = 0.0;
    UC_CO_CLOSE();
    return true;
}
#undef YO
#undef YOS
#undef SOUR
#undef RCS2
#undef TM_LD2
#undef TM_LD4
#undef TM_LD8
#undef TM_WAIT
#undef RCT
#undef CO_CHECK
#undef CO_TAKE
#undef CO_GIVE
#undef CO_QUOT
#undef RY0
#undef DTW
#undef CO_PF
#undef FSS
#undef FNS
#undef CO_TAIL
#undef CO_WAIT_Y
#undef CO_ARRIVE_Y
#undef CO_WAIT_P
#undef CO_ARRIVE_P

// soot mass fraction and number density (solvesp.f:2807-2832); st1 enters the residual. Rounded as written, like
// the generated program.
template <int N>
__device__ __forceinline__ void co_soot(const double (&yv)[N], const double (&so)[6], double s10, double s20,
                                        double rho, double dt, double wmstr, double sor1, double sor2, double st1,
                                        double st2, double &n1, double &n2, double &rsd)
{
    const double y2 = yv[1], y4 = yv[3], y5 = yv[4], y22 = yv[21];
    const double net = __fma_rn(-so[4], y4, __fma_rn(-so[3], y5, __fma_rn(-so[2], y2, __dmul_rn(2.0 * so[0], y22))));
    double rhs1 = __fma_rn(dt * ((double)0.012011f / wmstr), net, __dmul_rn(rho, s10));
    double fnew = __fma_rn(sor2, st1, rhs1 * sor1 / rho);
    rsd += fabs(st1 - fnew);
    if (fnew < 0.0) fnew = 0.0;
    n1 = fnew;
    rhs1 = __fma_rn(dt * so[1], y22, __dmul_rn(rho, s20));
    fnew = __fma_rn(sor2, st2, rhs1 * sor1 / __fma_rn(dt, so[5], rho));
    if (fnew < 0.0) fnew = 0.0;
    n2 = fnew;
}

// rho * Y of the old level, which every pass reads, into shared memory: dealt over the warps
__device__ __forceinline__ void co_load_cell(const CoTile &c, const UpdArgs &a, size_t cell, double rho)
{
    const size_t np = a.npad;
#pragma unroll
    for (int k0 = 0; k0 < LSP - 1; k0 += TR_TILE_WARPS) {
        const int k = k0 + c.role;
        if (k < LSP - 1) c.ry0[k * TILE] = rho * a.y0[k * np + cell];
    }
}

// The summing warp's part of a chunk of the field update.
template <int W>
__device__ __forceinline__ void co_sum_chunk(const CoTile &c, const UpdArgs &a, const TrArgs &t, const CUtensorMap *map_t,
                                             const CUtensorMap *map_s, int tile, size_t cell, bool live, int C,
                                             uint32_t &phase)
{
    const size_t np = a.npad;
    double yv[LSP];
#pragma unroll
    for (int k = 0; k < LSP; ++k) yv[k] = a.y[k * np + cell];
    const double rho = a.rho[cell];
    co_stage(c, map_t, map_s, tile, phase, t.status, [&] { co_load_cell(c, a, cell, rho); });
    double *dst = nullptr;
    for (int j = 0; j < C; ++j)
        co_sums<W, false>(c, yv, dst, UC_CO_SUMS * np,
                          (j < C - 1 ? t.snap + (size_t)j * TR_SNAP_ROWS * np : a.y) + W * np + cell, live, live && j > 0);
    co_sums_end<W>(c, dst, UC_CO_SUMS * np, live);
}

// FACES: the frozen transport terms are given (else they are zero, as in SOLVESP without faces).
template <bool FACES>
__global__ void __launch_bounds__(TR_WARPS * 32, 1)
update_tr_kernel(const UpdArgs a, const TrArgs t, const __grid_constant__ CUtensorMap map_t,
                 const __grid_constant__ CUtensorMap map_s)
{
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    extern __shared__ __align__(128) double s_rc[];          // [TR_TILES][TR_TILE_DOUBLES]
    __shared__ double s_wm[LSP];
    __shared__ double s_part[TR_TILES][TR_CHUNK_MAX];
    __shared__ __align__(8) uint64_t s_bar[TR_TILES];
    __shared__ uint32_t s_tmem;
    __shared__ int s_stop, s_pred, s_flag[TR_TILES];
    const DevParams &P = *a.P;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const size_t np = a.npad;
    const double sor1 = a.sor1, sor2 = 1.0 - a.sor1, dt = a.dt;

    if (w == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x < TR_TILES) mbar_init(&s_bar[threadIdx.x], 1);
    for (int k = threadIdx.x; k < LSP; k += blockDim.x) s_wm[k] = dt * P.WM[k];
    // the pass count of the previous call (*a.passes, written by block 0 at the end: every block reads it
    // before the first grid barrier). Only the chunk schedule depends on it, not the result: a chunk runs
    // passes beyond the stopping pass at most, whose Y is dropped for the snapshot of the stopping pass.
    if (threadIdx.x == 0) s_pred = t.adapt ? __ldcg(a.passes) : 0;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const CoTile c = co_tile(s_rc, s_bar, s_flag, s_tmem);
    const int slot = c.tile;
    uint32_t phase = 0;
    // tiles over the blocks first, so that a small field uses every SM
    const int stride = gridDim.x * TR_TILES, first = slot * gridDim.x + blockIdx.x;

    int p0 = 0, passes = 0, cpar = 0;
    for (;;) {
        int want = t.chunk;
        if (s_pred > 0) want = max(want, min(TR_CHUNK_MAX, s_pred - p0 - 4));
        const int C = min(want, a.isor - p0);
        if (c.role == UC_CO_SUMS) s_part[slot][lane] = 0.0;
        __syncwarp();
        for (int tile = first; tile < a.ntile; tile += stride) {
            const size_t cell = (size_t)tile * TILE + lane;
            const bool live = cell < (size_t)a.n && !(a.hold && a.hold[cell]);
            if (c.role == 0) co_sum_chunk<0>(c, a, t, &map_t, &map_s, tile, cell, live, C, phase);
            else if (c.role == 1) co_sum_chunk<1>(c, a, t, &map_t, &map_s, tile, cell, live, C, phase);
            else {
                double yv[LSP];
#pragma unroll
                for (int k = 0; k < LSP; ++k) yv[k] = a.y[k * np + cell];
                const double rho = a.rho[cell];
                double st1 = a.soot[cell], st2 = a.soot[np + cell], so[6];
#pragma unroll
                for (int m = 0; m < 6; ++m) so[m] = a.sour[m * np + cell];
                const double s10 = a.soot0[cell], s20 = a.soot0[np + cell];
                co_stage(c, &map_t, &map_s, tile, phase, t.status, [&] { co_load_cell(c, a, cell, rho); });
                if (lane == 0 && tile + stride < a.ntile) co_prefetch(&map_t, &map_s, tile + stride);
                co_close_begin(c, yv);
                for (int j = 0; j < C; ++j) {
                    double rsd = 0.0;
                    co_close<FACES, false>(c, yv, so, s_wm, rho, dt, sor1, sor2, a.face_sum ? a.face_sum + cell : nullptr,
                                           a.face_nbr ? a.face_nbr + cell : nullptr, np, false, rsd);
                    co_soot(yv, so, s10, s20, rho, dt, P.WMSTR, sor1, sor2, st1, st2, st1, st2, rsd);
                    double r = live ? rsd : 0.0;
                    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
                    if (lane == 0) s_part[slot][j] += r;
                    if (live) {           // argon, helium and soot; the summing warps store the others
                        const bool snap = j < C - 1;
                        double *sn = (snap ? t.snap + (size_t)j * TR_SNAP_ROWS * np : a.y) + cell;
                        sn[(LSP - 3) * np] = yv[LSP - 3];
                        sn[(LSP - 2) * np] = yv[LSP - 2];
                        double *ss = snap ? sn + (LSP - 1) * np : a.soot + cell;
                        ss[0] = st1;
                        ss[np] = st2;
                    }
                }
            }
        }
        // ---- residual of each pass of the chunk, and the stopping test (solvesp.f:2833-2838)
        __syncthreads();
        if (threadIdx.x < C) {
            double b = 0.0;
            for (int v = 0; v < TR_TILES; ++v) b += s_part[v][threadIdx.x];
            t.partial[((size_t)cpar * TR_CHUNK_MAX + threadIdx.x) * gridDim.x + blockIdx.x] = b;
        }
        grid.sync();
        if (w == 0) {                     // lane j: pass j of the chunk, over the blocks in order
            double tot = 0.0;
            if (lane < C) {
                const double *pp = t.partial + ((size_t)cpar * TR_CHUNK_MAX + lane) * gridDim.x;
#pragma unroll 8
                for (int b = 0; b < (int)gridDim.x; ++b) tot += __ldcg(pp + b);
            }
            const unsigned met = __ballot_sync(0xffffffffu, lane < C && tot / a.spnorm <= a.tol);
            if (lane == 0) s_stop = met ? __ffs(met) - 1 : -1;
        }
        __syncthreads();
        const int stop = s_stop;
        cpar ^= 1;
        if (stop >= 0) {
            passes = p0 + stop + 1;
            if (stop < C - 1) {
                // the pass that met the tolerance lies inside the chunk: its snapshot is the result
                // (written by other blocks before the grid barrier: read through L2)
                const double *sn = t.snap + (size_t)stop * TR_SNAP_ROWS * np;
                for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < (size_t)a.n;
                     c += (size_t)gridDim.x * blockDim.x) {
                    if (a.hold && a.hold[c]) continue;
                    for (int k = 0; k < LSP - 1; ++k) a.y[k * np + c] = __ldcg(sn + k * np + c);
                    a.soot[c] = __ldcg(sn + (LSP - 1) * np + c);
                    a.soot[np + c] = __ldcg(sn + LSP * np + c);
                }
            }
            break;
        }
        p0 += C;
        if (p0 >= a.isor) {
            passes = a.isor + 1;          // ISOR1 + 1 when the tolerance was not met
            break;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.passes = passes;
    // N2 closure and renormalisation (solvesp.f:2839-2915); the cells this thread copied above
    for (size_t cell = (size_t)blockIdx.x * blockDim.x + threadIdx.x; cell < (size_t)a.n;
         cell += (size_t)gridDim.x * blockDim.x) {
        if (a.hold && a.hold[cell]) continue;
        double ft = __ldcg(a.y + cell);
        for (int k = 1; k < LSP - 1; ++k) ft = ft + __ldcg(a.y + k * np + cell);
        ft = ft + __ldcg(a.soot + cell);
        double n2 = 1.0 - ft;
        if (ft > 1.0) {
            for (int k = 0; k < LSP - 1; ++k) a.y[k * np + cell] = __ldcg(a.y + k * np + cell) / ft;
            a.soot[cell] = __ldcg(a.soot + cell) / ft;
            n2 = 0.0;
        }
        a.y[(LSP - 1) * np + cell] = n2;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (w == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "r"(512));
}

// Per-cell form of the tile-resident update, for the batched integration (uc_integrate, rounds form):
// every cell runs its own pass loop with its own step a.dt / nsub[cell] and stops on its own residual
// (SPNORM = LSP - 1: solvesp.f:2833-2838 for a one-cell field), then the N2 closure and renormalisation
// (solvesp.f:2839-2915), all in the closing warp's registers. Only the first *nlive cells of the arrays are live (the caller
// orders the cells so that the ones still integrating come first); tiles beyond them are not touched.
// The old time level (a.y0, a.soot0) is the state at the sub-step start, and the caller may pass the
// state arrays themselves: a tile's rows are read before they are written. passes[cell] is
// incremented by the passes the cell ran, last[cell] set to them. No grid barrier.
// The arithmetic of a pass is that of update_tr_kernel; a lane that has converged keeps its Y while the
// others of its tile run on (its values are computed and dropped).
template <int W>
__device__ __forceinline__ void co_sum_cells(const CoTile &c, const UpdArgs &a, const CUtensorMap *map_t,
                                             const CUtensorMap *map_s, int tile, size_t cell, uint32_t &phase,
                                             int *status)
{
    const size_t np = a.npad;
    double yv[LSP];
#pragma unroll
    for (int k = 0; k < LSP; ++k) yv[k] = a.y[k * np + cell];
    const double rho = a.rho[cell];
    co_stage(c, map_t, map_s, tile, phase, status, [&] { co_load_cell(c, a, cell, rho); });
    double *dst = nullptr;
    while (co_sums<W, true>(c, yv, dst, 0, nullptr, false, false)) {}
}

__global__ void __launch_bounds__(TR_WARPS * 32, 1)
update_cells_kernel(const UpdArgs a, const int *nlive, const int *nsub, int *passes, int *last, int *status,
                    const __grid_constant__ CUtensorMap map_t, const __grid_constant__ CUtensorMap map_s)
{
    extern __shared__ __align__(128) double s_rc[];          // [TR_TILES][TR_TILE_DOUBLES]
    __shared__ double s_wm[LSP];
    __shared__ __align__(8) uint64_t s_bar[TR_TILES];
    __shared__ uint32_t s_tmem;
    __shared__ int s_flag[TR_TILES];
    const int n = *nlive;
    if (n <= 0) return;                                     // uniform over the grid
    const DevParams &P = *a.P;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const size_t np = a.npad;
    const double sor1 = a.sor1, sor2 = 1.0 - a.sor1;
    const int ntile = (n + TILE - 1) / TILE;

    if (w == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x < TR_TILES) mbar_init(&s_bar[threadIdx.x], 1);
    for (int k = threadIdx.x; k < LSP; k += blockDim.x) s_wm[k] = P.WM[k];
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const CoTile c = co_tile(s_rc, s_bar, s_flag, s_tmem);
    const int slot = c.tile;
    uint32_t phase = 0;

    for (int tile = slot * gridDim.x + blockIdx.x; tile < ntile; tile += gridDim.x * TR_TILES) {
        const size_t cell = (size_t)tile * TILE + lane;
        const bool live = cell < (size_t)n;
        if (c.role == 0) co_sum_cells<0>(c, a, &map_t, &map_s, tile, cell, phase, status);
        else if (c.role == 1) co_sum_cells<1>(c, a, &map_t, &map_s, tile, cell, phase, status);
        else {
            double yv[LSP];
#pragma unroll
            for (int k = 0; k < LSP; ++k) yv[k] = a.y[k * np + cell];
            const double rho = a.rho[cell];
            const double dt = a.dt / (double)max(1, nsub[cell]);
            double st1 = a.soot[cell], st2 = a.soot[np + cell], so[6];
#pragma unroll
            for (int m = 0; m < 6; ++m) so[m] = a.sour[m * np + cell];
            const double s10 = a.soot0[cell], s20 = a.soot0[np + cell];
            co_stage(c, &map_t, &map_s, tile, phase, status, [&] { co_load_cell(c, a, cell, rho); });
            if (lane == 0 && tile + (int)gridDim.x * TR_TILES < ntile)
                co_prefetch(&map_t, &map_s, tile + (int)gridDim.x * TR_TILES);
            co_close_begin(c, yv);
            bool done = !live;
            int npass = 0;
            for (int pass = 1;; ++pass) {
                const int quit = pass > a.isor || __all_sync(0xffffffffu, done);
                if (lane == 0) asm volatile("st.shared.b32 [%0], %1;" ::"r"(smem_u32(c.flag)), "r"(quit));
                double rsd = 0.0;
                if (!co_close<false, true>(c, yv, so, s_wm, rho, dt, sor1, sor2, nullptr, nullptr, np, done, rsd)) break;
                double n1, n2;
                co_soot(yv, so, s10, s20, rho, dt, P.WMSTR, sor1, sor2, st1, st2, n1, n2, rsd);
                if (!done) {
                    st1 = n1;
                    st2 = n2;
                    ++npass;
                    if (rsd / (double)(LSP - 1) <= a.tol) done = true;
                }
            }
            if (live) {
                // N2 closure and renormalisation (solvesp.f:2839-2915)
                double ft = yv[0];
#pragma unroll
                for (int k = 1; k < LSP - 1; ++k) ft = ft + yv[k];
                ft = ft + st1;
                double n2 = 1.0 - ft;
                if (ft > 1.0) {
#pragma unroll
                    for (int k = 0; k < LSP - 1; ++k) yv[k] = yv[k] / ft;
                    st1 = st1 / ft;
                    n2 = 0.0;
                }
                yv[LSP - 1] = n2;
#pragma unroll
                for (int k = 0; k < LSP; ++k) a.y[k * np + cell] = yv[k];
                a.soot[cell] = st1;
                a.soot[np + cell] = st2;
                passes[cell] += npass;
                last[cell] = npass;
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (w == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "r"(512));
}

}  // namespace uc
