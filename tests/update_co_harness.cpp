// Test-only harness: runs the three-warp form of the species-update program
// (unicorn_b200/csrc/generated/update_program_co.cuh) on the host, one thread per warp, with the named
// barriers of the device (bar.arrive / bar.sync over the tile's warps) as counting barriers. A barrier that is
// not complete within two seconds, or that one warp reaches twice in one use, ends the run with -1.
#include <atomic>
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>
#define LSP 52
#define LRX 544
struct double2 { double x, y; };
#include "../unicorn_b200/csrc/generated/update_program_co.cuh"

namespace {
struct Barrier {
    std::mutex m;
    std::condition_variable cv;
    int count = 0;
    long phase = 0;
    bool here[UC_CO_SUMS + 1] = {};
};
struct Cell {
    Barrier bar[4];
    std::atomic<bool> bad{false};
    const double *rc;                    // [544]
    double part[UC_CO_SLOTS][2], yb[6], ry0[LSP], dtw[LSP], sour[6], rho, sor1, sor2;
    double y[LSP];                       // in: the start of the passes; out: the result (each warp writes its rows)
    double rsd;
    int passes;
};

void arrive(Cell &c, int b, int who, bool wait)
{
    Barrier &B = c.bar[b];
    std::unique_lock<std::mutex> l(B.m);
    if (B.here[who]) c.bad = true;
    B.here[who] = true;
    const long p = B.phase;
    if (++B.count == UC_CO_SUMS + 1) {
        B.count = 0;
        std::memset(B.here, 0, sizeof(B.here));
        ++B.phase;
        B.cv.notify_all();
        return;
    }
    if (wait && !B.cv.wait_for(l, std::chrono::seconds(2), [&] { return B.phase != p || c.bad; })) c.bad = true;
}

#define CO_FMA(a, b, c) std::fma(a, b, c)
#define CO_MUL(a, b) ((a) * (b))
#define CO_ADD(a, b) ((a) + (b))
#define YO(k) yv[k]
#define YOS(m) ysh[m]
#define RCS2(i) double2{c.rc[UC_CO_NT + 2 * (i)], c.rc[UC_CO_NT + 2 * (i) + 1]}
// the pair in a tensor-memory column; the register slots of a wide load are consecutive
#define TM_LD2(b, q, col, p)                                                        \
    do {                                                                            \
        if (at[(col) / 4] != (p)) c.bad = true;                                     \
        bank[b][2 * (q)] = c.rc[2 * at[(col) / 4]];                                 \
        bank[b][2 * (q) + 1] = c.rc[2 * at[(col) / 4] + 1];                         \
    } while (0)
#define TM_LD4(b, q, col, p0, p1)                                                   \
    do {                                                                            \
        if ((col) % 8) c.bad = true;                                                \
        TM_LD2(b, q, col, p0);                                                      \
        TM_LD2(b, (q) + 1, (col) + 4, p1);                                          \
    } while (0)
#define TM_LD8(b, q, col, p0, p1, p2, p3)                                           \
    do {                                                                            \
        if ((col) % 16 || (q)) c.bad = true;                                        \
        TM_LD4(b, q, col, p0, p1);                                                  \
        TM_LD4(b, (q) + 2, (col) + 8, p2, p3);                                      \
    } while (0)
#define TM_WAIT(b, n) do { } while (0)
#define RCT(b, i) bank[b][i]
#define CO_PUT(slot, a, b) do { c.part[slot][0] = a; c.part[slot][1] = b; } while (0)
#define CO_GET(buf, k, mine, now) yv[k] = c.yb[buf]
#define CO_CHECK() do { if (c.bad) return; } while (0)
#define CO_WAIT_Y(set) do { arrive(c, set, W, true); if (c.bad) return; } while (0)
#define CO_ARRIVE_P(set) arrive(c, 2 + (set), W, false)

template <int W>
void sums(Cell &c)
{
    const short *pairs = W == 0 ? uc_co_pairs_0 : uc_co_pairs_1;
    const short *cols = W == 0 ? uc_co_cols_0 : uc_co_cols_1;
    const int n = 2 * (W == 0 ? UC_CO_PAIRS_0 : UC_CO_PAIRS_1);
    std::vector<int> at(n, -1);
    for (int i = 0; i < n; ++i) at[cols[i] / 4] = pairs[i];
    double yv[LSP], ysh[UC_CO_NSHADOW], bank[2][2 * UC_CO_SEG];
    std::memcpy(yv, c.y, sizeof(yv));
    for (int j = 0; j < c.passes; ++j) {
        if (W == 0) UC_CO_SUMS_0();
        else UC_CO_SUMS_1();
    }
    CO_WAIT_Y(UC_CO_LAST_SET);
}

#define SOUR(m) c.sour[m]
#define CO_TAKE(slot, a, b) do { a = c.part[slot][0]; b = c.part[slot][1]; } while (0)
#define CO_GIVE(buf, k) c.yb[buf] = yv[k]
#define CO_QUOT(n, d) ((n) / (d))
#define RY0(k) c.ry0[k]
#define DTW(k) c.dtw[k]
#define CO_PF(s, k) do { } while (0)
#define FSS(s) 0.0
#define FNS(s) 0.0
#define CO_TAIL(k) do { if (fnew < 0.0) fnew = 0.0; yv[k] = fnew; } while (0)
#define CO_ARRIVE_Y(set) arrive(c, set, UC_CO_SUMS, false)
#define CO_WAIT_P(set) do { arrive(c, 2 + (set), UC_CO_SUMS, true); if (c.bad) return; } while (0)
#define CO_LAST_SPECIES(buf, k) CO_GIVE(buf, k)

void close(Cell &c, double *out)
{
    const double rho = c.rho, sor1 = c.sor1, sor2 = c.sor2;
    double yv[LSP];
    std::memcpy(yv, c.y, sizeof(yv));
    UC_CO_LAST_RUN();
    CO_ARRIVE_Y(UC_CO_LAST_SET);
    for (int j = 0; j < c.passes; ++j) {
        double rsd = 0.0;
        UC_CO_CLOSE();
        c.rsd = rsd;
    }
    std::memcpy(out, yv, sizeof(yv));
}
}  // namespace

extern "C" int harness_update_co(int n, const double *rho_a, const double *y0_a, double *y_a, const double *rc_a,
                                 const double *sour_a, const double *wm, double dt, int passes, double relx)
{
    for (int i = 0; i < n; ++i) {
        Cell c;
        std::vector<double> rc(LRX);
        for (int r = 0; r < LRX; ++r) rc[r] = rc_a[(size_t)r * n + i];
        c.rc = rc.data();
        c.rho = rho_a[i];
        c.sor1 = relx;
        c.sor2 = 1.0 - relx;
        c.passes = passes;
        for (int k = 0; k < LSP; ++k) {
            c.y[k] = y_a[(size_t)k * n + i];
            c.ry0[k] = c.rho * y0_a[(size_t)k * n + i];
            c.dtw[k] = dt * wm[k];
        }
        for (int m = 0; m < 6; ++m) c.sour[m] = sour_a[(size_t)m * n + i];
        double out[LSP];
        std::thread a(sums<0>, std::ref(c)), b(sums<1>, std::ref(c));
        close(c, out);
        a.join();
        b.join();
        for (Barrier &B : c.bar)
            if (B.count) c.bad = true;       // somebody arrived and nobody waited for it
        if (c.bad) return -1;
        for (int k = 0; k < LSP - 1; ++k) y_a[(size_t)k * n + i] = out[k];
    }
    return 0;
}
