// Generated by unicorn_b200/mech/codegen.py: the species update (src/lib/solvesp.f:85-2806) with three
// warps per 32-cell tile. UC_CO_SUMS_0 and _1 are a pass of the two summing warps, UC_CO_CLOSE one of the
// closing warp. RC slots 0..335 lie in tensor memory, each pair of slots (2p, 2p + 1) with the one
// summing warp that uses it (uc_co_pairs_w: the pairs in row order; uc_co_cols_w: the first of the four
// 32-bit columns of each); the others lie in shared memory as rows of pairs, RCS2(i). Accessors: TM_LD2(bank,
// q, col, p) loads pair p (column col) into slots 2q, 2q + 1 of a register bank, TM_LD4 and TM_LD8 two and four
// pairs in neighbouring columns, TM_WAIT(bank, n) waits for the loads of its n pairs, RCT(bank, i); CO_PUT
// (slot, a, b) publishes two partial sums, CO_TAKE(slot, a, b) reads them; CO_GIVE(buf, k) publishes the
// new Y of species k, CO_GET(buf, k, mine, now) takes it into YO(k) (mine: this warp also stores it; now: of
// this pass, else of the pass before). Even and odd runs use sets 0 and 1 of the buffers and barriers:
// CO_ARRIVE_P(set) by the summing warps, CO_WAIT_P(set) by the closing one, CO_ARRIVE_Y, CO_WAIT_Y the other way;
// CO_CHECK() may leave the program (no more passes). CO_PF(slot, k) fetches the face terms of species k
// (FSS, FNS); RY0(k) is rho times the old level's Y; DTW(k) is dt * WM(k); CO_QUOT(n, d) is the quotient;
// CO_FMA(a, b, c) = a * b + c, CO_MUL and CO_ADD are rounded as they stand, so that every kernel that runs the
// program computes a cell bit for bit the same.
// 32 runs: 0 1 2 3 4 5 6 7 8 9 10 11-12 13 14 15-16 17-18 19-21 22 23-24 25 26 27-28 29-30 31 32-33 34-36 37-38 39-40 41 42-43 44-46 47-48
// Per summing warp: 40 segments, 122 tensor-memory loads, 265 shared-memory pair loads, 1750 operations; 125 segments, 409 tensor-memory loads, 167 shared-memory pair loads, 2582 operations.
#pragma once
#define UC_CO_NT 336
#define UC_CO_NS 208
#define UC_CO_PIECE 168
#define UC_CO_SEG 4
#define UC_CO_SUMS 2
#define UC_CO_NSHADOW 8
#define UC_CO_LAST 48
#define UC_CO_SLOTS 14
#define UC_CO_WINDOW 7
// the last run: its species' buffers hold their values when a pass begins, handed over through the set
#define UC_CO_LAST_SET 1
#define UC_CO_LAST_RUN() do { CO_LAST_SPECIES(3, 47); CO_LAST_SPECIES(4, 48); } while (0)
// operations per cell and pass (a multiply-add is two, a quotient one), the exchange between the warps included
#define UC_UPDATE_FLOPS_PER_CELL_PASS 5123
#define UC_CO_PAIRS_0 20
#define UC_CO_PAIRS_1 64
#define UC_CO_SUMS_0() do { \
    double G0a, G0b, H0, L0, L1, P0, P1, e0a, e0b, e1a, e2a, e30a, e31a, e39a, e40a, e43a, e47a, e48a, e4a, e4b, e6a, e8a, e9a, f10a, f2a, f48a, f8a, g0a, g0b, g1a, g1b, g2a, v0, v1, v2, v3, v4, v5, v6; \
    TM_LD4(0, 0, 96, 58, 76); \
    TM_LD2(0, 2, 44, 130); \
    TM_LD2(0, 3, 92, 37); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 32, 35, 40); \
    TM_LD2(1, 2, 40, 124); \
    TM_LD2(1, 3, 156, 138); \
    const double2 s0 = RCS2(94); \
    e48a = CO_MUL(YO(2), s0.x); \
    const double2 s1 = RCS2(97); \
    e48a = CO_FMA(YO(2), s1.x, e48a); \
    L0 = CO_MUL((YO(16) * YO(38)), s1.y); \
    const double2 s2 = RCS2(98); \
    e48a = CO_FMA(YO(2), s2.x, e48a); \
    L1 = CO_MUL((YO(43) * YO(13)), s2.y); \
    const double2 s3 = RCS2(102); \
    e47a = CO_MUL(YO(2), s3.x); \
    g0a = CO_MUL(YO(29), RCT(0, 4)); \
    L0 = CO_FMA(YO(28), RCT(0, 5), L0); \
    g0b = CO_MUL(YO(12), RCT(0, 6)); \
    L1 = CO_FMA(YO(13), RCT(0, 7), L1); \
    g0a = CO_FMA(YO(14), RCT(0, 0), g0a); \
    L0 = CO_FMA(YO(20), RCT(0, 1), L0); \
    g0b = CO_FMA(YO(19), RCT(0, 2), g0b); \
    L1 = CO_FMA(YO(18), RCT(0, 3), L1); \
    TM_WAIT(1, 4); \
    TM_LD8(0, 0, 16, 23, 49, 6, 118); \
    g0a = CO_FMA(YO(23), RCT(1, 6), g0a); \
    L0 = CO_FMA(YO(25), RCT(1, 7), L0); \
    const double2 s4 = RCS2(32); \
    g0b = CO_FMA(YO(38), s4.x, g0b); \
    L1 = CO_FMA(YO(36), s4.y, L1); \
    const double2 s5 = RCS2(43); \
    g0a = CO_FMA(YO(39), s5.x, g0a); \
    L0 = CO_FMA(YO(38), s5.y, L0); \
    const double2 s6 = RCS2(53); \
    g0b = CO_FMA(YO(40), s6.x, g0b); \
    L1 = CO_FMA(YO(41), s6.y, L1); \
    const double2 s7 = RCS2(54); \
    g0a = CO_FMA(YO(40), s7.x, g0a); \
    L0 = CO_FMA(YO(42), s7.y, L0); \
    const double2 s8 = RCS2(71); \
    g0b = CO_FMA(YO(43), s8.x, g0b); \
    const double2 s9 = RCS2(83); \
    g0a = CO_FMA(YO(46), s9.x, g0a); \
    const double2 s10 = RCS2(86); \
    g0b = CO_FMA(YO(46), s10.x, g0b); \
    P0 = CO_MUL(YO(2), CO_ADD(g0a, g0b)); \
    f48a = CO_MUL(YO(18), s10.y); \
    g1a = CO_MUL(YO(21), s8.y); \
    const double2 s11 = RCS2(94); \
    g1a = CO_FMA(YO(39), s11.y, g1a); \
    const double2 s12 = RCS2(102); \
    g1a = CO_FMA(YO(16), s12.y, g1a); \
    L0 = CO_FMA(YO(22), g1a, L0); \
    CO_WAIT_Y(1); \
    CO_GET(3, 47, 0, 0); \
    CO_GET(4, 48, 1, 0); \
    P0 = CO_FMA(YO(48), e48a, P0); \
    P1 = CO_MUL(YO(47), e47a); \
    L1 = CO_FMA(YO(48), f48a, L1); \
    v0 = CO_ADD(P0, P1); \
    v1 = CO_ADD(L0, L1); \
    CO_PUT(0, v0, v1); \
    CO_ARRIVE_P(0); \
    YOS(0) = YO(2); \
    YOS(1) = YO(4); \
    CO_CHECK(); \
    g0a = CO_MUL(YO(10), RCT(1, 1)); \
    L0 = CO_MUL(YO(11), RCT(1, 0)); \
    g0b = CO_MUL(YO(13), RCT(1, 3)); \
    L1 = CO_MUL(YO(12), RCT(1, 2)); \
    g0a = CO_FMA(YO(11), RCT(1, 5), g0a); \
    L0 = CO_FMA(YO(28), RCT(1, 4), L0); \
    const double2 s13 = RCS2(12); \
    g0b = CO_FMA(YO(31), s13.y, g0b); \
    L1 = CO_FMA(YO(35), s13.x, L1); \
    const double2 s14 = RCS2(17); \
    g0a = CO_FMA(YO(31), s14.y, g0a); \
    L0 = CO_FMA(YO(32), s14.x, L0); \
    const double2 s15 = RCS2(28); \
    g0b = CO_FMA(YO(37), s15.x, g0b); \
    L1 = CO_FMA(YO(36), s15.y, L1); \
    const double2 s16 = RCS2(33); \
    g0a = CO_FMA(YO(36), s16.y, g0a); \
    L0 = CO_FMA(YO(38), s16.x, L0); \
    const double2 s17 = RCS2(52); \
    g0b = CO_FMA(YO(42), s17.y, g0b); \
    L1 = CO_FMA(YO(40), s17.x, L1); \
    const double2 s18 = RCS2(66); \
    g0a = CO_FMA(YO(39), s18.y, g0a); \
    L0 = CO_FMA(YO(42), s18.x, L0); \
    const double2 s19 = RCS2(78); \
    g0b = CO_FMA((YO(21) * YO(38)), s19.y, g0b); \
    L1 = CO_FMA(YO(45), s19.x, L1); \
    const double2 s20 = RCS2(79); \
    g0a = CO_FMA((YO(22) * YO(36)), s20.y, g0a); \
    L0 = CO_FMA(YO(45), s20.x, L0); \
    P0 = CO_MUL(YO(6), CO_ADD(g0a, g0b)); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 112, 120, 141); \
    TM_LD2(1, 2, 44, 130); \
    TM_LD2(1, 3, 60, 64); \
    g1a = CO_MUL(YO(9), RCT(0, 1)); \
    L1 = CO_FMA(YO(8), RCT(0, 0), L1); \
    g1a = CO_FMA(YO(17), RCT(0, 3), g1a); \
    L0 = CO_FMA(YO(13), RCT(0, 2), L0); \
    g1a = CO_FMA(YO(3), RCT(0, 4), g1a); \
    L1 = CO_ADD(L1, RCT(0, 5)); \
    g1a = CO_FMA(YO(26), RCT(0, 7), g1a); \
    L0 = CO_FMA(YO(27), RCT(0, 6), L0); \
    P1 = CO_MUL(YO(3), g1a); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 96, 58, 76); \
    TM_LD2(0, 2, 92, 37); \
    TM_LD2(0, 3, 156, 138); \
    g2a = CO_MUL((YO(4) * YO(2)), RCT(1, 7)); \
    L1 = CO_FMA(YO(14), RCT(1, 6), L1); \
    g2a = CO_FMA(YO(10), RCT(1, 1), g2a); \
    L0 = CO_FMA(YO(27), RCT(1, 0), L0); \
    g2a = CO_FMA((YO(11) * YO(4)), RCT(1, 3), g2a); \
    L1 = CO_FMA(YO(23), RCT(1, 2), L1); \
    const double2 s21 = RCS2(39); \
    g2a = CO_FMA((YO(13) * YO(10)), s21.y, g2a); \
    L0 = CO_FMA(YO(36), s21.x, L0); \
    P0 = CO_FMA(YO(8), g2a, P0); \
    v0 = CO_ADD(P0, P1); \
    v1 = CO_ADD(L0, L1); \
    CO_PUT(7, v0, v1); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(14), RCT(1, 6)); \
    e0a = CO_MUL(YO(28), RCT(1, 5)); \
    L0 = CO_MUL(YO(29), RCT(1, 4)); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 64, 107, 142); \
    TM_LD2(1, 2, 56, 61); \
    TM_LD2(1, 3, 144, 122); \
    e0b = CO_MUL(YO(13), RCT(0, 5)); \
    L1 = CO_MUL(YO(12), RCT(0, 4)); \
    e0a = CO_FMA(YO(20), RCT(0, 1), e0a); \
    L0 = CO_FMA(YO(14), RCT(0, 0), L0); \
    e0b = CO_FMA(YO(18), RCT(0, 3), e0b); \
    L1 = CO_FMA(YO(19), RCT(0, 2), L1); \
    e0a = CO_FMA(YO(25), RCT(0, 7), e0a); \
    L0 = CO_FMA(YO(23), RCT(0, 6), L0); \
    const double2 s22 = RCS2(32); \
    e0b = CO_FMA(YO(36), s22.y, e0b); \
    L1 = CO_FMA(YO(38), s22.x, L1); \
    const double2 s23 = RCS2(43); \
    e0a = CO_FMA(YO(38), s23.y, e0a); \
    L0 = CO_FMA(YO(39), s23.x, L0); \
    const double2 s24 = RCS2(53); \
    e0b = CO_FMA(YO(41), s24.y, e0b); \
    L1 = CO_FMA(YO(40), s24.x, L1); \
    const double2 s25 = RCS2(54); \
    e0a = CO_FMA(YO(42), s25.y, e0a); \
    L0 = CO_FMA(YO(40), s25.x, L0); \
    const double2 s26 = RCS2(71); \
    e0b = CO_FMA((YO(21) * YO(22)), s26.y, e0b); \
    L1 = CO_FMA(YO(43), s26.x, L1); \
    const double2 s27 = RCS2(86); \
    e0a = CO_FMA((YO(48) * YO(18)), s27.y, e0a); \
    L0 = CO_FMA(YO(46), s27.x, L0); \
    const double2 s28 = RCS2(94); \
    e0b = CO_FMA((YO(39) * YO(22)), s28.y, e0b); \
    L1 = CO_FMA(YO(48), s28.x, L1); \
    const double2 s29 = RCS2(97); \
    e0a = CO_FMA((YO(16) * YO(38)), s29.y, e0a); \
    L0 = CO_FMA(YO(48), s29.x, L0); \
    const double2 s30 = RCS2(98); \
    e0b = CO_FMA((YO(43) * YO(13)), s30.y, e0b); \
    L1 = CO_FMA(YO(48), s30.x, L1); \
    const double2 s31 = RCS2(102); \
    e0a = CO_FMA((YO(22) * YO(16)), s31.y, e0a); \
    L0 = CO_FMA(YO(47), s31.x, L0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 104, 102, 116); \
    TM_LD2(0, 2, 56, 61); \
    TM_LD2(0, 3, 152, 27); \
    g0a = CO_MUL(YO(8), RCT(1, 1)); \
    L1 = CO_FMA(YO(25), RCT(1, 0), L1); \
    g0b = CO_MUL(YO(23), RCT(1, 2)); \
    g0a = CO_FMA(YO(4), RCT(1, 7), g0a); \
    L0 = CO_FMA(YO(28), RCT(1, 6), L0); \
    const double2 s32 = RCS2(14); \
    g0b = CO_FMA(YO(28), s32.y, g0b); \
    L1 = CO_FMA(YO(35), s32.x, L1); \
    const double2 s33 = RCS2(20); \
    g0a = CO_FMA(YO(28), s33.y, g0a); \
    L0 = CO_FMA(YO(32), s33.x, L0); \
    const double2 s34 = RCS2(25); \
    g0b = CO_FMA(YO(21), s34.x, g0b); \
    L1 = CO_FMA(YO(36), s34.y, L1); \
    const double2 s35 = RCS2(48); \
    g0a = CO_FMA(YO(16), s35.y, g0a); \
    L0 = CO_FMA(YO(39), s35.x, L0); \
    const double2 s36 = RCS2(49); \
    g0b = CO_FMA(YO(22), s36.x, g0b); \
    L1 = CO_FMA(YO(38), s36.y, L1); \
    const double2 s37 = RCS2(95); \
    g0a = CO_FMA((YO(16) * YO(16)), s37.y, g0a); \
    L0 = CO_FMA(YO(48), s37.x, L0); \
    const double2 s38 = RCS2(101); \
    g0b = CO_FMA(YO(39), s38.y, g0b); \
    L1 = CO_FMA(YO(47), s38.x, L1); \
    P1 = CO_MUL(YO(13), CO_ADD(g0a, g0b)); \
    g1a = CO_MUL(YO(14), RCT(1, 4)); \
    g1a = CO_FMA(YO(14), RCT(1, 4), g1a); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 56, 61, 64); \
    TM_LD2(1, 2, 68, 142); \
    TM_LD2(1, 3, 104, 102); \
    g1a = CO_FMA(YO(21), RCT(0, 0), g1a); \
    L0 = CO_FMA(YO(26), RCT(0, 1), L0); \
    g1a = CO_FMA(YO(10), RCT(0, 6), g1a); \
    L1 = CO_FMA(YO(9), RCT(0, 7), L1); \
    const double2 s39 = RCS2(42); \
    g1a = CO_FMA(YO(39), s39.x, g1a); \
    L0 = CO_FMA((YO(25) * YO(13)), s39.y, L0); \
    P0 = CO_MUL(YO(3), g1a); \
    g2a = CO_MUL(YO(27), RCT(0, 2)); \
    L1 = CO_FMA(YO(26), RCT(0, 3), L1); \
    const double2 s40 = RCS2(72); \
    g2a = CO_FMA(YO(43), s40.x, g2a); \
    L0 = CO_FMA((YO(44) * YO(38)), s40.y, L0); \
    const double2 s41 = RCS2(103); \
    g2a = CO_FMA(YO(47), s41.x, g2a); \
    L1 = CO_FMA((YO(5) * YO(43)), s41.y, L1); \
    P1 = CO_FMA(YO(4), g2a, P1); \
    const double2 s42 = RCS2(15); \
    g0a = CO_MUL(YO(16), s42.y); \
    L0 = CO_FMA(YO(35), s42.x, L0); \
    const double2 s43 = RCS2(19); \
    g0a = CO_FMA(YO(16), s43.y, g0a); \
    L1 = CO_FMA(YO(32), s43.x, L1); \
    P0 = CO_FMA(YO(5), g0a, P0); \
    g1a = CO_MUL(YO(2), RCT(0, 5)); \
    g1a = CO_FMA(YO(2), RCT(0, 5), g1a); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 16, 23, 49); \
    TM_LD2(0, 2, 28, 118); \
    TM_LD2(0, 3, 152, 27); \
    g1a = CO_FMA(YO(4), RCT(1, 3), g1a); \
    g1a = CO_FMA(YO(18), RCT(1, 5), g1a); \
    L0 = CO_FMA(YO(8), g1a, L0); \
    const double2 s44 = RCS2(27); \
    P1 = CO_FMA(YO(36), s44.y, P1); \
    L1 = CO_FMA(YO(37), s44.x, L1); \
    const double2 s45 = RCS2(44); \
    P0 = CO_FMA(YO(39), s45.y, P0); \
    L0 = CO_FMA(YO(38), s45.x, L0); \
    const double2 s46 = RCS2(67); \
    P1 = CO_FMA(YO(43), s46.x, P1); \
    L1 = CO_FMA((YO(21) * YO(22)), s46.y, L1); \
    const double2 s47 = RCS2(96); \
    P0 = CO_FMA((YO(39) * YO(18)), s47.y, P0); \
    L0 = CO_FMA(YO(48), s47.x, L0); \
    const double2 s48 = RCS2(83); \
    L1 = CO_FMA(YO(46), s48.x, L1); \
    const double2 s49 = RCS2(85); \
    L0 = CO_FMA(YO(46), s49.x, L0); \
    CO_WAIT_Y(0); \
    CO_GET(0, 0, 1, 1); \
    P0 = CO_FMA(YO(0), CO_ADD(e0a, e0b), P0); \
    v0 = G0a; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    CO_PUT(0, v1, v0); \
    CO_PUT(1, v2, 0.0); \
    CO_ARRIVE_P(0); \
    G0a = CO_MUL((YO(8) * YOS(0)), RCT(1, 1)); \
    L0 = CO_MUL(YO(14), RCT(1, 0)); \
    G0a = CO_FMA(YO(26), RCT(1, 7), G0a); \
    L1 = CO_MUL(YO(21), RCT(1, 6)); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 80, 26, 109); \
    TM_LD2(1, 2, 140, 103); \
    TM_LD2(1, 3, 148, 150); \
    G0a = CO_FMA(YO(9), RCT(0, 7), G0a); \
    L0 = CO_FMA(YO(10), RCT(0, 6), L0); \
    const double2 s50 = RCS2(42); \
    G0a = CO_FMA((YO(25) * YO(13)), s50.y, G0a); \
    L1 = CO_FMA(YO(39), s50.x, L1); \
    e1a = CO_MUL(YO(8), RCT(0, 0)); \
    L0 = CO_FMA(YO(9), RCT(0, 1), L0); \
    e1a = CO_FMA(YO(13), RCT(0, 2), e1a); \
    L1 = CO_FMA(YO(17), RCT(0, 3), L1); \
    e1a = CO_FMA(YO(27), RCT(0, 4), e1a); \
    L0 = CO_FMA(YO(26), RCT(0, 5), L0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 80, 26, 109); \
    TM_LD2(0, 2, 24, 6); \
    TM_LD2(0, 3, 72, 8); \
    g0a = CO_MUL(YO(8), RCT(1, 1)); \
    L1 = CO_FMA(YO(10), RCT(1, 0), L1); \
    g0b = CO_MUL(YO(26), RCT(1, 3)); \
    L0 = CO_FMA(YO(25), RCT(1, 2), L0); \
    g0a = CO_FMA(YO(34), RCT(1, 7), g0a); \
    L1 = CO_FMA(YO(31), RCT(1, 6), L1); \
    const double2 s51 = RCS2(0); \
    g0b = CO_FMA(YO(32), s51.y, g0b); \
    L0 = CO_FMA(YO(30), s51.x, L0); \
    const double2 s52 = RCS2(1); \
    g0a = CO_FMA(YO(35), s52.y, g0a); \
    L1 = CO_FMA(YO(30), s52.x, L1); \
    const double2 s53 = RCS2(18); \
    g0b = CO_FMA(YO(31), s53.y, g0b); \
    L0 = CO_FMA(YO(32), s53.x, L0); \
    const double2 s54 = RCS2(56); \
    g0a = CO_FMA(YO(42), s54.y, g0a); \
    L1 = CO_FMA(YO(40), s54.x, L1); \
    P1 = CO_MUL(YO(4), CO_ADD(g0a, g0b)); \
    g1a = CO_MUL(YO(14), RCT(1, 5)); \
    L0 = CO_FMA(YO(21), RCT(1, 4), L0); \
    const double2 s55 = RCS2(24); \
    g1a = CO_FMA(YO(16), s55.y, g1a); \
    L1 = CO_FMA(YO(36), s55.x, L1); \
    P0 = CO_MUL(YO(8), g1a); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 144, 122, 150); \
    TM_LD2(1, 2, 0, 72); \
    TM_LD2(1, 3, 108, 116); \
    L0 = CO_FMA(YO(3), RCT(0, 4), L0); \
    L1 = CO_FMA(YO(3), RCT(0, 4), L1); \
    P1 = CO_FMA(YO(6), RCT(0, 7), P1); \
    L0 = CO_FMA(YO(4), RCT(0, 6), L0); \
    const double2 s56 = RCS2(26); \
    P0 = CO_FMA((YO(26) * YO(13)), s56.y, P0); \
    L1 = CO_FMA(YO(36), s56.x, L1); \
    CO_WAIT_Y(1); \
    CO_GET(3, 1, 0, 1); \
    P0 = CO_FMA(YO(1), e1a, P0); \
    P1 = CO_FMA(YO(1), RCT(0, 5), P1); \
    P0 = CO_FMA(YO(1), RCT(0, 5), P0); \
    v0 = G0a; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    CO_PUT(7, v1, v0); \
    CO_PUT(8, v2, 0.0); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(10), RCT(0, 0)); \
    L0 = CO_MUL(YO(8), RCT(0, 1)); \
    G0b = CO_MUL(YO(25), RCT(0, 2)); \
    L1 = CO_MUL(YO(26), RCT(0, 3)); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 8, 19, 106); \
    TM_LD2(0, 2, 4, 129); \
    TM_LD2(0, 3, 136, 60); \
    G0a = CO_FMA(YO(31), RCT(1, 2), G0a); \
    L0 = CO_FMA(YO(34), RCT(1, 3), L0); \
    const double2 s57 = RCS2(0); \
    G0b = CO_FMA(YO(30), s57.x, G0b); \
    L1 = CO_FMA(YO(32), s57.y, L1); \
    const double2 s58 = RCS2(1); \
    G0a = CO_FMA(YO(30), s58.x, G0a); \
    L0 = CO_FMA(YO(35), s58.y, L0); \
    const double2 s59 = RCS2(18); \
    G0b = CO_FMA(YO(32), s59.x, G0b); \
    L1 = CO_FMA(YO(31), s59.y, L1); \
    const double2 s60 = RCS2(55); \
    G0a = CO_FMA(YO(40), s60.x, G0a); \
    L0 = CO_FMA(YO(41), s60.y, L0); \
    e2a = CO_MUL(YO(26), RCT(1, 7)); \
    L1 = CO_FMA(YO(27), RCT(1, 6), L1); \
    e2a = CO_FMA(YO(28), RCT(1, 0), e2a); \
    L0 = CO_FMA(YO(13), RCT(1, 1), L0); \
    const double2 s61 = RCS2(72); \
    e2a = CO_FMA((YO(44) * YO(38)), s61.y, e2a); \
    L1 = CO_FMA(YO(43), s61.x, L1); \
    const double2 s62 = RCS2(103); \
    e2a = CO_FMA((YO(5) * YO(43)), s62.y, e2a); \
    L0 = CO_FMA(YO(47), s62.x, L0); \
    g0a = CO_MUL(YO(11), RCT(1, 5)); \
    L1 = CO_FMA(YO(17), RCT(1, 4), L1); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 72, 8, 143); \
    TM_LD2(1, 2, 60, 64); \
    TM_LD2(1, 3, 116, 141); \
    g0b = CO_MUL(YO(17), RCT(0, 5)); \
    L0 = CO_FMA(YO(29), RCT(0, 4), L0); \
    g0a = CO_FMA(YO(6), RCT(0, 1), g0a); \
    L1 = CO_FMA(YO(7), RCT(0, 0), L1); \
    g0b = CO_FMA(YO(27), RCT(0, 3), g0b); \
    L0 = CO_FMA(YO(21), RCT(0, 2), L0); \
    g0a = CO_FMA(YO(20), RCT(0, 7), g0a); \
    L1 = CO_FMA(YO(14), RCT(0, 6), L1); \
    const double2 s63 = RCS2(16); \
    g0b = CO_FMA(YO(31), s63.y, g0b); \
    L0 = CO_FMA(YO(35), s63.x, L0); \
    const double2 s64 = RCS2(22); \
    g0a = CO_FMA(YO(31), s64.y, g0a); \
    L1 = CO_FMA(YO(32), s64.x, L1); \
    const double2 s65 = RCS2(29); \
    g0b = CO_FMA(YO(37), s65.y, g0b); \
    L0 = CO_FMA(YO(36), s65.x, L0); \
    const double2 s66 = RCS2(36); \
    g0a = CO_FMA(YO(36), s66.y, g0a); \
    L1 = CO_FMA(YO(38), s66.x, L1); \
    const double2 s67 = RCS2(41); \
    g0b = CO_FMA(YO(38), s67.y, g0b); \
    L0 = CO_FMA(YO(39), s67.x, L0); \
    const double2 s68 = RCS2(57); \
    g0a = CO_FMA(YO(42), s68.y, g0a); \
    L1 = CO_FMA(YO(40), s68.x, L1); \
    const double2 s69 = RCS2(87); \
    g0b = CO_FMA((YO(48) * YO(18)), s69.y, g0b); \
    L0 = CO_FMA(YO(46), s69.x, L0); \
    const double2 s70 = RCS2(93); \
    g0a = CO_FMA((YO(39) * YO(22)), s70.y, g0a); \
    L1 = CO_FMA(YO(48), s70.x, L1); \
    P1 = CO_MUL(YO(5), CO_ADD(g0a, g0b)); \
    TM_WAIT(1, 4); \
    TM_LD8(0, 0, 0, 72, 129, 19, 106); \
    g1a = CO_MUL(YO(23), RCT(1, 2)); \
    const double2 s71 = RCS2(9); \
    g1b = CO_MUL(YO(18), s71.x); \
    L0 = CO_FMA(YO(35), s71.y, L0); \
    const double2 s72 = RCS2(21); \
    g1a = CO_FMA(YO(32), s72.x, g1a); \
    g1b = CO_FMA(YO(32), s72.x, g1b); \
    const double2 s73 = RCS2(38); \
    g1a = CO_FMA(YO(37), s73.x, g1a); \
    L1 = CO_FMA((YO(8) * YO(22)), s73.y, L1); \
    const double2 s74 = RCS2(46); \
    g1b = CO_FMA(YO(38), s74.x, g1b); \
    P0 = CO_MUL(YO(6), CO_ADD(g1a, g1b)); \
    g2a = CO_MUL(YO(14), RCT(1, 4)); \
    g2a = CO_FMA(YO(23), RCT(1, 6), g2a); \
    P1 = CO_FMA(YO(1), g2a, P1); \
    f2a = CO_MUL(YO(8), RCT(1, 5)); \
    g0a = CO_MUL(YO(10), RCT(1, 3)); \
    g0a = CO_FMA(YO(8), RCT(1, 7), g0a); \
    g0a = CO_FMA(YO(22), s74.y, g0a); \
    L1 = CO_FMA(YO(11), g0a, L1); \
    const double2 s75 = RCS2(21); \
    g1a = CO_MUL(YO(31), s75.y); \
    g1a = CO_FMA(YO(31), s75.y, g1a); \
    L0 = CO_FMA(YO(4), g1a, L0); \
    P0 = CO_FMA(YO(6), RCT(1, 1), P0); \
    H0 = RCT(1, 0); \
    const double2 s76 = RCS2(8); \
    P1 = CO_FMA(YO(33), s76.y, P1); \
    L1 = CO_FMA(YO(16), s76.x, L1); \
    const double2 s77 = RCS2(90); \
    L0 = CO_FMA(YO(46), s77.x, L0); \
    CO_WAIT_Y(0); \
    CO_GET(0, 2, 1, 1); \
    P0 = CO_FMA(YO(2), e2a, P0); \
    L0 = CO_FMA(YO(2), f2a, L0); \
    v0 = CO_ADD(G0a, G0b); \
    v1 = H0; \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    CO_PUT(0, v2, v0); \
    CO_PUT(1, v3, v1); \
    CO_ARRIVE_P(0); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 72, 8, 143); \
    TM_LD2(1, 2, 8, 19); \
    TM_LD2(1, 3, 136, 60); \
    G0a = CO_MUL(YO(17), RCT(0, 0)); \
    L0 = CO_MUL(YO(11), RCT(0, 1)); \
    G0b = CO_MUL(YO(29), RCT(0, 2)); \
    L1 = CO_MUL(YO(17), RCT(0, 3)); \
    G0a = CO_FMA(YO(7), RCT(0, 4), G0a); \
    L0 = CO_FMA(YO(6), RCT(0, 5), L0); \
    G0b = CO_FMA(YO(21), RCT(0, 6), G0b); \
    L1 = CO_FMA(YO(27), RCT(0, 7), L1); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 32, 35, 40); \
    TM_LD2(0, 2, 40, 124); \
    TM_LD2(0, 3, 124, 157); \
    G0a = CO_FMA(YO(14), RCT(1, 6), G0a); \
    L0 = CO_FMA(YO(20), RCT(1, 7), L0); \
    const double2 s78 = RCS2(16); \
    G0b = CO_FMA(YO(35), s78.x, G0b); \
    L1 = CO_FMA(YO(31), s78.y, L1); \
    const double2 s79 = RCS2(22); \
    G0a = CO_FMA(YO(32), s79.x, G0a); \
    L0 = CO_FMA(YO(31), s79.y, L0); \
    const double2 s80 = RCS2(29); \
    G0b = CO_FMA(YO(36), s80.x, G0b); \
    L1 = CO_FMA(YO(37), s80.y, L1); \
    const double2 s81 = RCS2(36); \
    G0a = CO_FMA(YO(38), s81.x, G0a); \
    L0 = CO_FMA(YO(36), s81.y, L0); \
    const double2 s82 = RCS2(41); \
    G0b = CO_FMA(YO(39), s82.x, G0b); \
    L1 = CO_FMA(YO(38), s82.y, L1); \
    const double2 s83 = RCS2(58); \
    G0a = CO_FMA(YO(40), s83.x, G0a); \
    L0 = CO_FMA(YO(41), s83.y, L0); \
    const double2 s84 = RCS2(87); \
    G0b = CO_FMA(YO(46), s84.x, G0b); \
    L1 = CO_FMA((YO(48) * YO(18)), s84.y, L1); \
    const double2 s85 = RCS2(90); \
    G0a = CO_FMA(YO(46), s85.x, G0a); \
    const double2 s86 = RCS2(93); \
    G0b = CO_FMA(YO(48), s86.x, G0b); \
    L0 = CO_FMA((YO(39) * YO(22)), s86.y, L0); \
    const double2 s87 = RCS2(103); \
    G0a = CO_FMA(YO(47), s87.x, G0a); \
    L1 = CO_FMA((YO(43) * YO(2)), s87.y, L1); \
    const double2 s88 = RCS2(15); \
    g0a = CO_MUL(YO(35), s88.x); \
    L0 = CO_FMA(YO(16), s88.y, L0); \
    const double2 s89 = RCS2(19); \
    g0a = CO_FMA(YO(32), s89.x, g0a); \
    L1 = CO_FMA(YO(16), s89.y, L1); \
    P0 = CO_MUL(YO(2), g0a); \
    CO_WAIT_Y(1); \
    CO_GET(3, 3, 0, 1); \
    v0 = CO_ADD(G0a, G0b); \
    v1 = P0; \
    v2 = CO_ADD(L0, L1); \
    CO_PUT(7, v1, v0); \
    CO_PUT(8, v2, 0.0); \
    CO_ARRIVE_P(1); \
    e4a = CO_MUL(YO(7), RCT(1, 4)); \
    H0 = RCT(1, 5); \
    e4b = CO_MUL(YO(3), RCT(1, 0)); \
    L0 = RCT(1, 1); \
    e4a = CO_FMA((YO(11) * YO(10)), RCT(1, 3), e4a); \
    L1 = CO_MUL(YO(23), RCT(1, 2)); \
    const double2 s90 = RCS2(38); \
    e4b = CO_FMA((YO(8) * YO(22)), s90.y, e4b); \
    L0 = CO_FMA(YO(37), s90.x, L0); \
    const double2 s91 = RCS2(46); \
    e4a = CO_FMA((YO(22) * YO(11)), s91.y, e4a); \
    L1 = CO_FMA(YO(38), s91.x, L1); \
    const double2 s92 = RCS2(21); \
    L0 = CO_FMA(YO(32), s92.x, L0); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 128, 41, 94); \
    TM_LD2(1, 2, 8, 19); \
    TM_LD2(1, 3, 124, 157); \
    g0a = CO_MUL(YO(11), RCT(0, 0)); \
    L1 = CO_FMA(YO(10), RCT(0, 1), L1); \
    g0b = CO_MUL(YO(12), RCT(0, 2)); \
    L0 = CO_FMA(YO(13), RCT(0, 3), L0); \
    g0a = CO_FMA(YO(28), RCT(0, 4), g0a); \
    L1 = CO_FMA(YO(11), RCT(0, 5), L1); \
    const double2 s93 = RCS2(12); \
    g0b = CO_FMA(YO(35), s93.x, g0b); \
    L0 = CO_FMA(YO(31), s93.y, L0); \
    const double2 s94 = RCS2(33); \
    g0a = CO_FMA(YO(38), s94.x, g0a); \
    L1 = CO_FMA(YO(36), s94.y, L1); \
    const double2 s95 = RCS2(51); \
    g0b = CO_FMA(YO(40), s95.x, g0b); \
    L0 = CO_FMA(YO(41), s95.y, L0); \
    const double2 s96 = RCS2(66); \
    g0a = CO_FMA(YO(42), s96.x, g0a); \
    L1 = CO_FMA(YO(39), s96.y, L1); \
    const double2 s97 = RCS2(78); \
    g0b = CO_FMA(YO(45), s97.x, g0b); \
    L0 = CO_FMA((YO(21) * YO(38)), s97.y, L0); \
    const double2 s98 = RCS2(79); \
    g0a = CO_FMA(YO(45), s98.x, g0a); \
    L1 = CO_FMA((YO(22) * YO(36)), s98.y, L1); \
    P1 = CO_MUL(YO(1), CO_ADD(g0a, g0b)); \
    g1a = CO_MUL(YO(23), RCT(0, 7)); \
    L0 = CO_FMA(YO(31), RCT(0, 6), L0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 48, 56, 69); \
    TM_LD2(0, 2, 16, 23); \
    TM_LD2(0, 3, 80, 26); \
    g1b = CO_MUL(YO(13), RCT(1, 1)); \
    L1 = CO_FMA(YO(12), RCT(1, 0), L1); \
    g1a = CO_FMA((YO(13) * YO(8)), RCT(1, 3), g1a); \
    L0 = CO_FMA(YO(24), RCT(1, 2), L0); \
    const double2 s99 = RCS2(7); \
    g1b = CO_FMA(YO(35), s99.y, g1b); \
    L1 = CO_FMA(YO(30), s99.x, L1); \
    const double2 s100 = RCS2(60); \
    g1a = CO_FMA(YO(42), s100.y, g1a); \
    L0 = CO_FMA(YO(40), s100.x, L0); \
    const double2 s101 = RCS2(80); \
    g1b = CO_FMA((YO(21) * YO(38)), s101.y, g1b); \
    L1 = CO_FMA(YO(45), s101.x, L1); \
    const double2 s102 = RCS2(81); \
    g1a = CO_FMA((YO(22) * YO(36)), s102.y, g1a); \
    L0 = CO_FMA(YO(45), s102.x, L0); \
    P0 = CO_MUL(YO(7), CO_ADD(g1a, g1b)); \
    CO_WAIT_Y(0); \
    CO_GET(0, 4, 1, 1); \
    const double2 s103 = RCS2(21); \
    e4b = CO_FMA((YO(31) * YOS(1)), s103.y, e4b); \
    P0 = CO_FMA(YO(4), CO_ADD(e4a, e4b), P0); \
    v0 = H0; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    CO_PUT(0, v1, v2); \
    CO_PUT(1, v0, 0.0); \
    CO_ARRIVE_P(0); \
    G0a = CO_MUL(YO(31), RCT(1, 6)); \
    L0 = CO_MUL(YO(23), RCT(1, 7)); \
    G0b = CO_MUL(YO(12), RCT(1, 0)); \
    L1 = CO_MUL(YO(13), RCT(1, 1)); \
    G0a = CO_FMA(YO(24), RCT(1, 2), G0a); \
    L0 = CO_FMA((YO(13) * YO(8)), RCT(1, 3), L0); \
    const double2 s104 = RCS2(6); \
    G0b = CO_FMA(YO(30), s104.x, G0b); \
    L1 = CO_FMA(YO(33), s104.y, L1); \
    const double2 s105 = RCS2(60); \
    G0a = CO_FMA(YO(40), s105.x, G0a); \
    L0 = CO_FMA(YO(42), s105.y, L0); \
    const double2 s106 = RCS2(80); \
    G0b = CO_FMA(YO(45), s106.x, G0b); \
    L1 = CO_FMA((YO(21) * YO(38)), s106.y, L1); \
    const double2 s107 = RCS2(81); \
    G0a = CO_FMA(YO(45), s107.x, G0a); \
    L0 = CO_FMA((YO(22) * YO(36)), s107.y, L0); \
    L1 = CO_FMA(YO(4), RCT(1, 4), L1); \
    CO_WAIT_Y(1); \
    CO_GET(3, 5, 0, 1); \
    G0b = CO_FMA(YO(5), RCT(1, 5), G0b); \
    v0 = CO_ADD(G0a, G0b); \
    v1 = CO_ADD(L0, L1); \
    CO_PUT(7, v0, v1); \
    CO_ARRIVE_P(1); \
    e6a = CO_MUL(YO(24), RCT(1, 2)); \
    H0 = CO_MUL(YO(13), RCT(1, 3)); \
    const double2 s108 = RCS2(38); \
    e6a = CO_FMA(YO(37), s108.x, e6a); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 112, 120, 141); \
    TM_LD2(1, 2, 60, 64); \
    TM_LD2(1, 3, 88, 30); \
    g0a = CO_MUL(YO(3), RCT(0, 5)); \
    L0 = CO_MUL(YO(1), RCT(0, 4)); \
    g0a = CO_FMA(YO(15), RCT(0, 0), g0a); \
    L1 = CO_MUL(YO(11), RCT(0, 1)); \
    g0a = CO_FMA(YO(20), RCT(0, 2), g0a); \
    L0 = CO_FMA(YO(10), RCT(0, 3), L0); \
    const double2 s109 = RCS2(13); \
    g0a = CO_FMA(YO(18), s109.y, g0a); \
    L1 = CO_FMA(YO(35), s109.x, L1); \
    P1 = CO_MUL(YO(9), g0a); \
    g1a = CO_MUL(YO(3), RCT(0, 6)); \
    L0 = CO_FMA(YO(4), RCT(0, 7), L0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 56, 61, 64); \
    TM_LD2(0, 2, 68, 142); \
    TM_LD2(0, 3, 140, 103); \
    g1a = CO_FMA(YO(13), RCT(1, 6), g1a); \
    L1 = CO_FMA(YO(12), RCT(1, 7), L1); \
    const double2 s110 = RCS2(37); \
    g1a = CO_FMA(YO(37), s110.x, g1a); \
    L0 = CO_FMA(YO(36), s110.y, L0); \
    P0 = CO_MUL(YO(10), g1a); \
    g2a = CO_MUL(YO(14), RCT(1, 4)); \
    g2a = CO_FMA(YO(27), RCT(1, 0), g2a); \
    L1 = CO_FMA(YO(10), RCT(1, 1), L1); \
    g2a = CO_FMA(YO(23), RCT(1, 2), g2a); \
    P1 = CO_FMA(YO(1), g2a, P1); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 64, 107, 142); \
    TM_LD2(1, 2, 16, 23); \
    TM_LD2(1, 3, 116, 141); \
    g0a = CO_MUL(YO(14), RCT(0, 0)); \
    g0a = CO_FMA(YO(21), RCT(0, 6), g0a); \
    L0 = CO_FMA(YO(14), RCT(0, 7), L0); \
    P0 = CO_FMA(YO(3), g0a, P0); \
    g1a = CO_MUL(YO(2), RCT(0, 1)); \
    g1a = CO_FMA(YO(4), RCT(0, 3), g1a); \
    g1a = CO_FMA(YO(18), RCT(0, 5), g1a); \
    L1 = CO_FMA(YO(2), g1a, L1); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 48, 56, 69); \
    TM_LD2(0, 2, 80, 26); \
    TM_LD2(0, 3, 152, 27); \
    g2a = CO_MUL(YO(11), RCT(1, 7)); \
    const double2 s111 = RCS2(38); \
    g2a = CO_FMA(YO(22), s111.y, g2a); \
    L0 = CO_FMA(YO(4), g2a, L0); \
    P1 = CO_FMA((YO(2) * YO(25)), RCT(1, 0), P1); \
    L1 = CO_FMA(YO(13), RCT(1, 1), L1); \
    P0 = CO_FMA((YO(23) * YO(13)), RCT(1, 2), P0); \
    CO_WAIT_Y(0); \
    CO_GET(0, 6, 1, 1); \
    P0 = CO_FMA(YO(6), e6a, P0); \
    v0 = H0; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    CO_PUT(0, v1, v2); \
    CO_PUT(1, v0, 0.0); \
    CO_ARRIVE_P(0); \
    G0a = CO_MUL(YO(1), RCT(1, 4)); \
    L0 = CO_MUL(YO(3), RCT(1, 5)); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 32, 35); \
    TM_LD2(1, 1, 76, 143); \
    TM_LD2(1, 2, 88, 30); \
    TM_LD2(1, 3, 112, 120); \
    G0a = CO_FMA(YO(11), RCT(0, 1), G0a); \
    L0 = CO_FMA(YO(15), RCT(0, 0), L0); \
    G0a = CO_FMA(YO(10), RCT(0, 3), G0a); \
    L0 = CO_FMA(YO(20), RCT(0, 2), L0); \
    P0 = CO_MUL((YO(3) * YO(10)), RCT(0, 6)); \
    L0 = CO_FMA(YO(2), RCT(0, 7), L0); \
    CO_WAIT_Y(1); \
    CO_GET(3, 7, 0, 1); \
    v0 = G0a; \
    v1 = P0; \
    v2 = L0; \
    CO_PUT(7, v1, v0); \
    CO_PUT(8, v2, 0.0); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(20), RCT(0, 2)); \
    G0a = CO_FMA(YO(2), RCT(0, 7), G0a); \
    L0 = CO_MUL(YO(3), RCT(0, 6)); \
    e8a = CO_MUL(YO(4), RCT(0, 5)); \
    L1 = CO_MUL(YO(3), RCT(0, 4)); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 48, 56, 69); \
    TM_LD2(0, 2, 32, 35); \
    TM_LD2(0, 3, 112, 120); \
    e8a = CO_FMA(YO(12), RCT(1, 5), e8a); \
    L0 = CO_FMA(YO(13), RCT(1, 4), L0); \
    const double2 s112 = RCS2(37); \
    e8a = CO_FMA(YO(36), s112.y, e8a); \
    L1 = CO_FMA(YO(37), s112.x, L1); \
    g0a = CO_MUL(YO(11), RCT(1, 0)); \
    L0 = CO_FMA(YO(6), RCT(1, 1), L0); \
    g0a = CO_FMA(YO(27), RCT(1, 6), g0a); \
    const double2 s113 = RCS2(30); \
    g0a = CO_FMA(YO(37), s113.x, g0a); \
    L1 = CO_FMA(YO(25), s113.y, L1); \
    const double2 s114 = RCS2(39); \
    g0a = CO_FMA(YO(36), s114.x, g0a); \
    P1 = CO_MUL(YO(1), g0a); \
    f8a = CO_MUL(YO(13), s114.y); \
    P0 = CO_MUL((YO(6) * YO(23)), RCT(1, 2)); \
    L1 = CO_FMA((YO(11) * YO(4)), RCT(1, 3), L1); \
    const double2 s115 = RCS2(40); \
    P1 = CO_FMA((YO(3) * YO(39)), s115.x, P1); \
    L0 = CO_FMA(YO(18), s115.y, L0); \
    CO_WAIT_Y(0); \
    CO_GET(0, 8, 1, 1); \
    P0 = CO_FMA(YO(8), e8a, P0); \
    L0 = CO_FMA(YO(8), f8a, L0); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 0, 72); \
    TM_LD2(1, 1, 40, 124); \
    TM_LD2(1, 2, 76, 143); \
    TM_LD2(1, 3, 116, 141); \
    L1 = CO_FMA(YO(8), RCT(0, 3), L1); \
    L0 = CO_FMA(YO(8), RCT(0, 7), L0); \
    v0 = G0a; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    CO_PUT(0, v1, v0); \
    CO_PUT(1, v2, 0.0); \
    CO_ARRIVE_P(0); \
    G0a = CO_MUL(YO(6), RCT(0, 5)); \
    L0 = CO_MUL(YO(1), RCT(0, 4)); \
    e9a = CO_MUL(YO(15), RCT(0, 0)); \
    L1 = CO_MUL(YO(8), RCT(0, 1)); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 88, 30, 37); \
    TM_LD2(0, 2, 36, 40); \
    TM_LD2(0, 3, 120, 155); \
    g0a = CO_MUL(YO(6), RCT(1, 4)); \
    H0 = CO_MUL(YO(4), RCT(1, 5)); \
    g0a = CO_FMA(YO(1), RCT(1, 6), g0a); \
    P1 = CO_MUL(YO(23), g0a); \
    g1a = CO_MUL(YO(8), RCT(1, 7)); \
    const double2 s116 = RCS2(46); \
    g1a = CO_FMA(YO(22), s116.y, g1a); \
    L0 = CO_FMA(YO(4), g1a, L0); \
    P0 = CO_MUL((YO(4) * YO(17)), RCT(1, 0)); \
    L1 = CO_FMA(YO(5), RCT(1, 1), L1); \
    P1 = CO_FMA((YO(1) * YO(28)), RCT(1, 2), P1); \
    L0 = CO_FMA(YO(6), RCT(1, 3), L0); \
    P0 = CO_FMA((YO(6) * YO(38)), s116.x, P0); \
    CO_WAIT_Y(1); \
    CO_GET(3, 9, 0, 1); \
    P0 = CO_FMA(YO(9), e9a, P0); \
    v0 = G0a; \
    v1 = H0; \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 88, 30, 37); \
    TM_LD2(1, 2, 36, 40); \
    TM_LD2(1, 3, 128, 41); \
    G0a = CO_MUL(YO(13), RCT(0, 0)); \
    L0 = CO_MUL(YO(8), RCT(0, 1)); \
    g0a = CO_MUL(YO(6), RCT(0, 5)); \
    L1 = CO_MUL(YO(1), RCT(0, 4)); \
    g0b = CO_MUL(YO(0), RCT(0, 3)); \
    L0 = CO_FMA(YO(2), RCT(0, 2), L0); \
    g0a = CO_FMA(YO(31), RCT(0, 6), g0a); \
    L1 = CO_FMA(YO(23), RCT(0, 7), L1); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 64, 107, 142); \
    TM_LD2(0, 2, 120, 155); \
    TM_LD2(0, 3, 128, 41); \
    g0b = CO_FMA(YO(7), RCT(1, 7), g0b); \
    L0 = CO_FMA(YO(6), RCT(1, 6), L0); \
    const double2 s117 = RCS2(2); \
    g0a = CO_FMA(YO(30), s117.x, g0a); \
    L1 = CO_FMA(YO(33), s117.y, L1); \
    const double2 s118 = RCS2(3); \
    g0b = CO_FMA(YO(30), s118.x, g0b); \
    L0 = CO_FMA(YO(32), s118.y, L0); \
    const double2 s119 = RCS2(4); \
    g0a = CO_FMA(YO(30), s119.x, g0a); \
    L1 = CO_FMA(YO(35), s119.y, L1); \
    const double2 s120 = RCS2(34); \
    g0b = CO_FMA(YO(38), s120.x, g0b); \
    L0 = CO_FMA(YO(36), s120.y, L0); \
    const double2 s121 = RCS2(73); \
    g0a = CO_FMA(YO(43), s121.x, g0a); \
    L1 = CO_FMA((YO(21) * YO(22)), s121.y, L1); \
    P0 = CO_MUL(YO(13), CO_ADD(g0a, g0b)); \
    v4 = G0a; \
    v5 = P0; \
    v6 = CO_ADD(L0, L1); \
    CO_PUT(7, v2, v0); \
    CO_PUT(8, v3, v1); \
    CO_PUT(9, v5, v4); \
    CO_PUT(10, v6, 0.0); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(1), RCT(1, 4)); \
    L0 = CO_MUL(YO(6), RCT(1, 5)); \
    G0b = CO_MUL(YO(8), RCT(1, 1)); \
    G0a = CO_FMA(YO(2), RCT(1, 2), G0a); \
    L1 = CO_MUL(YO(0), RCT(1, 3)); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 20, 49); \
    TM_LD2(1, 1, 88, 30); \
    TM_LD2(1, 2, 132, 94); \
    TM_LD2(1, 3, 144, 122); \
    G0b = CO_FMA(YO(23), RCT(0, 5), G0b); \
    L0 = CO_FMA(YO(31), RCT(0, 4), L0); \
    G0a = CO_FMA(YO(6), RCT(0, 6), G0a); \
    L1 = CO_FMA(YO(7), RCT(0, 7), L1); \
    const double2 s122 = RCS2(2); \
    G0b = CO_FMA(YO(33), s122.y, G0b); \
    L0 = CO_FMA(YO(30), s122.x, L0); \
    const double2 s123 = RCS2(4); \
    G0a = CO_FMA(YO(35), s123.y, G0a); \
    L1 = CO_FMA(YO(30), s123.x, L1); \
    const double2 s124 = RCS2(34); \
    G0b = CO_FMA(YO(36), s124.y, G0b); \
    L0 = CO_FMA(YO(38), s124.x, L0); \
    const double2 s125 = RCS2(73); \
    G0a = CO_FMA((YO(21) * YO(22)), s125.y, G0a); \
    L1 = CO_FMA(YO(43), s125.x, L1); \
    g0a = CO_MUL(YO(25), RCT(0, 0)); \
    L0 = CO_FMA(YO(8), RCT(0, 1), L0); \
    g0b = CO_MUL((YO(8) * YO(18)), RCT(0, 3)); \
    L1 = CO_FMA(YO(23), RCT(0, 2), L1); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 56, 61, 64); \
    TM_LD2(0, 2, 96, 58); \
    TM_LD2(0, 3, 136, 60); \
    g0a = CO_FMA(YO(28), RCT(1, 6), g0a); \
    L0 = CO_FMA(YO(4), RCT(1, 7), L0); \
    const double2 s126 = RCS2(20); \
    g0b = CO_FMA(YO(32), s126.x, g0b); \
    L1 = CO_FMA(YO(28), s126.y, L1); \
    const double2 s127 = RCS2(49); \
    g0a = CO_FMA(YO(38), s127.y, g0a); \
    L0 = CO_FMA(YO(22), s127.x, L0); \
    const double2 s128 = RCS2(85); \
    g0b = CO_FMA(YO(46), s128.x, g0b); \
    const double2 s129 = RCS2(95); \
    g0a = CO_FMA(YO(48), s129.x, g0a); \
    L1 = CO_FMA((YO(16) * YO(16)), s129.y, L1); \
    const double2 s130 = RCS2(98); \
    g0b = CO_FMA(YO(48), s130.x, g0b); \
    L0 = CO_FMA((YO(0) * YO(43)), s130.y, L0); \
    P0 = CO_MUL(YO(2), CO_ADD(g0a, g0b)); \
    g1a = CO_MUL(YO(17), RCT(1, 1)); \
    L1 = CO_FMA(YO(1), RCT(1, 0), L1); \
    const double2 s131 = RCS2(42); \
    g1a = CO_FMA(YO(39), s131.x, g1a); \
    L0 = CO_FMA((YO(25) * YO(2)), s131.y, L0); \
    P1 = CO_MUL(YO(3), g1a); \
    const double2 s132 = RCS2(39); \
    f10a = CO_MUL(YO(8), s132.y); \
    P0 = CO_FMA((YO(6) * YO(24)), RCT(1, 4), P0); \
    L0 = CO_FMA((YO(8) * YO(7)), RCT(1, 5), L0); \
    const double2 s133 = RCS2(35); \
    P1 = CO_FMA(YO(38), s133.y, P1); \
    L1 = CO_FMA(YO(21), s133.x, L1); \
    P0 = CO_FMA((YO(1) * YO(36)), s132.x, P0); \
    const double2 s134 = RCS2(50); \
    P1 = CO_FMA(YO(40), s134.x, P1); \
    L0 = CO_FMA(YO(18), s134.y, L0); \
    const double2 s135 = RCS2(82); \
    P0 = CO_FMA(YO(46), s135.x, P0); \
    const double2 s136 = RCS2(99); \
    P1 = CO_FMA(YO(47), s136.x, P1); \
    L1 = CO_FMA(YO(38), s136.y, L1); \
    CO_WAIT_Y(0); \
    CO_GET(0, 10, 1, 1); \
    L1 = CO_FMA(YO(10), f10a, L1); \
    L0 = CO_FMA(YO(10), RCT(1, 2), L0); \
    v0 = CO_ADD(G0a, G0b); \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    CO_PUT(0, v1, v0); \
    CO_PUT(1, v2, 0.0); \
    CO_ARRIVE_P(0); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 0, 72, 129); \
    TM_LD2(1, 2, 48, 56); \
    TM_LD2(1, 3, 140, 103); \
    g0a = CO_MUL(YO(0), RCT(0, 5)); \
    L0 = CO_MUL(YO(2), RCT(0, 4)); \
    g0a = CO_FMA(YO(5), RCT(0, 7), g0a); \
    L0 = CO_FMA(YO(4), RCT(0, 6), L0); \
    P0 = CO_MUL(YO(20), g0a); \
    g1a = CO_MUL((YO(8) * YO(2)), RCT(0, 1)); \
    L0 = CO_FMA(YO(3), RCT(0, 0), L0); \
    g1a = CO_FMA((YO(8) * YO(4)), RCT(0, 3), g1a); \
    L0 = CO_FMA(YO(1), RCT(0, 2), L0); \
    P0 = CO_FMA(YO(2), g1a, P0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 96, 58, 76); \
    TM_LD2(0, 2, 20, 49); \
    TM_LD2(0, 3, 68, 142); \
    P0 = CO_FMA((YO(3) * YO(21)), RCT(1, 6), P0); \
    L0 = CO_FMA(YO(8), RCT(1, 7), L0); \
    CO_WAIT_Y(1); \
    CO_GET(3, 11, 0, 1); \
    CO_GET(4, 12, 1, 1); \
    v0 = P0; \
    v1 = L0; \
    CO_PUT(7, v0, v1); \
    CO_ARRIVE_P(1); \
    P0 = CO_MUL((YO(11) * YO(8)), RCT(1, 5)); \
    L0 = CO_MUL(YO(9), RCT(1, 4)); \
    CO_WAIT_Y(0); \
    CO_GET(0, 13, 0, 1); \
    v0 = P0; \
    v1 = L0; \
    const double2 s137 = RCS2(15); \
    g0a = CO_MUL(YO(35), s137.x); \
    L0 = CO_MUL(YO(5), s137.y); \
    const double2 s138 = RCS2(19); \
    g0b = CO_MUL(YO(32), s138.x); \
    L1 = CO_MUL(YO(5), s138.y); \
    const double2 s139 = RCS2(48); \
    g0a = CO_FMA(YO(39), s139.x, g0a); \
    L0 = CO_FMA(YO(13), s139.y, L0); \
    const double2 s140 = RCS2(70); \
    g0b = CO_FMA(YO(43), s140.x, g0b); \
    L1 = CO_FMA(YO(22), s140.y, L1); \
    const double2 s141 = RCS2(84); \
    g0a = CO_FMA(YO(46), s141.x, g0a); \
    const double2 s142 = RCS2(85); \
    g0b = CO_FMA(YO(46), s142.x, g0b); \
    g0a = CO_FMA(YO(46), s142.x, g0a); \
    g0b = CO_FMA(YO(46), s142.x, g0b); \
    const double2 s143 = RCS2(95); \
    g0a = CO_FMA(YO(48), s143.x, g0a); \
    g0b = CO_FMA(YO(48), s143.x, g0b); \
    const double2 s144 = RCS2(97); \
    g0a = CO_FMA(YO(48), s144.x, g0a); \
    const double2 s145 = RCS2(100); \
    g0b = CO_FMA(YO(47), s145.x, g0b); \
    L0 = CO_FMA(YO(18), s145.y, L0); \
    const double2 s146 = RCS2(102); \
    g0a = CO_FMA(YO(47), s146.x, g0a); \
    P0 = CO_MUL(YO(2), CO_ADD(g0a, g0b)); \
    const double2 s147 = RCS2(89); \
    g1a = CO_MUL(YO(4), s147.x); \
    const double2 s148 = RCS2(90); \
    g1a = CO_FMA(YO(4), s148.x, g1a); \
    g1a = CO_FMA(YO(4), s148.x, g1a); \
    g1a = CO_FMA(YO(4), s148.x, g1a); \
    P1 = CO_MUL(YO(46), g1a); \
    const double2 s149 = RCS2(95); \
    g2a = CO_MUL(YO(13), s149.y); \
    g2a = CO_FMA(YO(13), s149.y, g2a); \
    L1 = CO_FMA(YO(16), g2a, L1); \
    const double2 s150 = RCS2(97); \
    g0a = CO_MUL(YO(38), s150.y); \
    const double2 s151 = RCS2(102); \
    g0a = CO_FMA(YO(22), s151.y, g0a); \
    L0 = CO_FMA(YO(0), g0a, L0); \
    const double2 s152 = RCS2(8); \
    P0 = CO_FMA(YO(33), s152.y, P0); \
    L1 = CO_FMA(YO(4), s152.x, L1); \
    const double2 s153 = RCS2(24); \
    P1 = CO_FMA((YO(3) * YO(36)), s153.x, P1); \
    L0 = CO_FMA(YO(8), s153.y, L0); \
    const double2 s154 = RCS2(64); \
    P0 = CO_FMA(YO(42), s154.x, P0); \
    L1 = CO_FMA(YO(13), s154.y, L1); \
    const double2 s155 = RCS2(82); \
    P1 = CO_FMA(YO(46), s155.x, P1); \
    P0 = CO_FMA(YO(46), s155.x, P0); \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    CO_PUT(0, v0, v1); \
    CO_PUT(1, v2, v3); \
    CO_ARRIVE_P(0); \
    P0 = CO_MUL((YO(11) * YO(5)), RCT(1, 1)); \
    L0 = CO_MUL(YO(4), RCT(1, 0)); \
    P0 = CO_FMA((YO(4) * YO(29)), RCT(1, 2), P0); \
    L0 = CO_FMA(YO(5), RCT(1, 3), L0); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 12, 106); \
    TM_LD2(1, 1, 52, 69); \
    TM_LD2(1, 2, 104, 102); \
    TM_LD2(1, 3, 136, 60); \
    P0 = CO_FMA((YO(13) * YO(1)), RCT(0, 4), P0); \
    L0 = CO_FMA(YO(3), RCT(0, 5), L0); \
    CO_WAIT_Y(1); \
    CO_GET(3, 14, 1, 1); \
    v0 = P0; \
    v1 = L0; \
    g0a = CO_MUL(YO(19), RCT(0, 2)); \
    L0 = CO_MUL(YO(0), RCT(0, 3)); \
    const double2 s156 = RCS2(86); \
    g0a = CO_FMA(YO(46), s156.x, g0a); \
    const double2 s157 = RCS2(96); \
    g0a = CO_FMA(YO(48), s157.x, g0a); \
    L1 = CO_MUL(YO(39), s157.y); \
    const double2 s158 = RCS2(100); \
    g0a = CO_FMA(YO(47), s158.x, g0a); \
    H0 = s158.y; \
    P0 = CO_MUL(YO(2), g0a); \
    const double2 s159 = RCS2(9); \
    g1a = CO_MUL(YO(35), s159.y); \
    L0 = CO_FMA(YO(6), s159.x, L0); \
    const double2 s160 = RCS2(87); \
    g1a = CO_FMA(YO(46), s160.x, g1a); \
    const double2 s161 = RCS2(89); \
    g1a = CO_FMA(YO(46), s161.x, g1a); \
    P1 = CO_MUL(YO(4), g1a); \
    const double2 s162 = RCS2(86); \
    g2a = CO_MUL(YO(0), s162.y); \
    g2a = CO_FMA(YO(5), s160.y, g2a); \
    L1 = CO_FMA(YO(48), g2a, L1); \
    P0 = CO_FMA((YO(13) * YO(23)), RCT(0, 6), P0); \
    L0 = CO_FMA((YO(8) * YO(2)), RCT(0, 7), L0); \
    const double2 s163 = RCS2(13); \
    P1 = CO_FMA((YO(8) * YO(35)), s163.x, P1); \
    L1 = CO_FMA(YO(9), s163.y, L1); \
    const double2 s164 = RCS2(40); \
    P0 = CO_FMA((YO(3) * YO(39)), s164.x, P0); \
    L0 = CO_FMA(YO(10), s164.y, L0); \
    const double2 s165 = RCS2(50); \
    P1 = CO_FMA(YO(40), s165.x, P1); \
    L1 = CO_FMA(YO(13), s165.y, L1); \
    const double2 s166 = RCS2(91); \
    P0 = CO_FMA(YO(48), s166.x, P0); \
    L0 = CO_FMA(YO(38), s166.y, L0); \
    v2 = H0; \
    v3 = CO_ADD(P0, P1); \
    v4 = CO_ADD(L0, L1); \
    CO_PUT(7, v0, v1); \
    CO_PUT(8, v3, v4); \
    CO_PUT(9, v2, 0.0); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(0), RCT(0, 3)); \
    L0 = CO_MUL(YO(2), RCT(0, 2)); \
    CO_WAIT_Y(0); \
    CO_GET(0, 15, 0, 1); \
    CO_GET(1, 16, 1, 1); \
    v0 = G0a; \
    v1 = L0; \
    g0a = CO_MUL(YO(2), RCT(0, 0)); \
    L0 = CO_MUL(YO(0), RCT(0, 1)); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 120, 155, 157); \
    TM_LD2(0, 2, 76, 143); \
    TM_LD2(0, 3, 140, 103); \
    g0a = CO_FMA(YO(4), RCT(1, 6), g0a); \
    L0 = CO_FMA(YO(5), RCT(1, 7), L0); \
    P0 = CO_MUL(YO(14), g0a); \
    P0 = CO_FMA((YO(10) * YO(8)), RCT(1, 3), P0); \
    L0 = CO_FMA(YO(9), RCT(1, 2), L0); \
    v2 = P0; \
    v3 = L0; \
    g0a = CO_MUL(YO(26), RCT(1, 5)); \
    L0 = CO_MUL(YO(3), RCT(1, 4)); \
    const double2 s167 = RCS2(25); \
    g0a = CO_FMA(YO(36), s167.y, g0a); \
    L1 = CO_MUL(YO(13), s167.x); \
    const double2 s168 = RCS2(71); \
    g0a = CO_FMA(YO(43), s168.x, g0a); \
    P0 = CO_MUL(YO(2), g0a); \
    const double2 s169 = RCS2(78); \
    g1a = CO_MUL(YO(1), s169.x); \
    const double2 s170 = RCS2(80); \
    g1a = CO_FMA(YO(6), s170.x, g1a); \
    P1 = CO_MUL(YO(45), g1a); \
    g2a = CO_MUL(YO(0), s168.y); \
    const double2 s171 = RCS2(73); \
    g2a = CO_FMA(YO(12), s171.y, g2a); \
    L0 = CO_FMA(YO(22), g2a, L0); \
    g0a = CO_MUL(YO(6), s169.y); \
    g0a = CO_FMA(YO(7), s170.y, g0a); \
    L1 = CO_FMA(YO(38), g0a, L1); \
    P0 = CO_FMA((YO(5) * YO(27)), RCT(1, 1), P0); \
    L0 = CO_FMA(YO(4), RCT(1, 0), L0); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 68, 142); \
    TM_LD2(1, 1, 116, 141); \
    TM_LD2(1, 2, 132, 94); \
    TM_LD2(1, 3, 156, 138); \
    P1 = CO_FMA((YO(14) * YO(8)), RCT(0, 7), P1); \
    L1 = CO_FMA(YO(3), RCT(0, 6), L1); \
    P0 = CO_FMA((YO(13) * YO(43)), s171.x, P0); \
    const double2 s172 = RCS2(75); \
    P1 = CO_FMA(YO(45), s172.x, P1); \
    L0 = CO_FMA(YO(39), s172.y, L0); \
    v4 = CO_ADD(P0, P1); \
    v5 = CO_ADD(L0, L1); \
    CO_PUT(0, v0, v1); \
    CO_PUT(1, v2, v3); \
    CO_PUT(2, v4, v5); \
    CO_ARRIVE_P(0); \
    const double2 s173 = RCS2(46); \
    g0a = CO_MUL(YO(6), s173.x); \
    const double2 s174 = RCS2(49); \
    g0a = CO_FMA(YO(2), s174.y, g0a); \
    L0 = CO_MUL(YO(13), s174.x); \
    P0 = CO_MUL(YO(38), g0a); \
    const double2 s175 = RCS2(71); \
    g1a = CO_MUL(YO(2), s175.x); \
    H0 = CO_MUL(YO(0), s175.y); \
    const double2 s176 = RCS2(73); \
    g1a = CO_FMA(YO(13), s176.x, g1a); \
    H0 = CO_FMA(YO(12), s176.y, H0); \
    P1 = CO_MUL(YO(43), g1a); \
    const double2 s177 = RCS2(38); \
    g2a = CO_MUL(YO(8), s177.y); \
    g2a = CO_FMA(YO(11), s173.y, g2a); \
    L1 = CO_MUL(YO(4), g2a); \
    P0 = CO_FMA((YO(6) * YO(37)), s177.x, P0); \
    const double2 s178 = RCS2(67); \
    P1 = CO_FMA(YO(43), s178.x, P1); \
    H0 = CO_FMA(YO(2), s178.y, H0); \
    const double2 s179 = RCS2(68); \
    P0 = CO_FMA(YO(43), s179.x, P0); \
    L0 = CO_FMA(YO(22), s179.y, L0); \
    L1 = CO_FMA(YO(22), s179.y, L1); \
    P1 = CO_FMA(YO(43), s179.x, P1); \
    const double2 s180 = RCS2(69); \
    P0 = CO_FMA(YO(43), s180.y, P0); \
    L0 = CO_FMA(YO(22), s180.x, L0); \
    L1 = CO_FMA(YO(22), s180.x, L1); \
    P1 = CO_FMA(YO(43), s180.y, P1); \
    const double2 s181 = RCS2(77); \
    P0 = CO_FMA(YO(45), s181.x, P0); \
    L0 = CO_FMA(YO(38), s181.y, L0); \
    const double2 s182 = RCS2(93); \
    P1 = CO_FMA((YO(4) * YO(48)), s182.x, P1); \
    L1 = CO_FMA((YO(5) * YO(39)), s182.y, L1); \
    CO_WAIT_Y(1); \
    CO_GET(3, 17, 0, 1); \
    CO_GET(4, 18, 1, 1); \
    v0 = H0; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    CO_PUT(7, v1, v2); \
    CO_PUT(8, v0, 0.0); \
    CO_ARRIVE_P(1); \
    g0a = CO_MUL(YO(13), RCT(0, 0)); \
    L0 = CO_MUL(YO(12), RCT(0, 1)); \
    g0a = CO_FMA(YO(6), RCT(0, 2), g0a); \
    L1 = CO_MUL(YO(7), RCT(0, 3)); \
    P0 = CO_MUL(YO(31), g0a); \
    g1a = CO_MUL((YO(11) * YO(10)), RCT(0, 5)); \
    L0 = CO_FMA(YO(6), RCT(0, 4), L0); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 28, 118); \
    TM_LD2(0, 1, 64, 107); \
    TM_LD2(0, 2, 84, 109); \
    TM_LD2(0, 3, 108, 116); \
    g1a = CO_FMA((YO(11) * YO(8)), RCT(1, 3), g1a); \
    L1 = CO_FMA(YO(1), RCT(1, 2), L1); \
    P1 = CO_MUL(YO(4), g1a); \
    P0 = CO_FMA(((YO(18) * YO(8)) * YO(2)), RCT(1, 1), P0); \
    L0 = CO_FMA(YO(13), RCT(1, 0), L0); \
    P1 = CO_FMA((YO(0) * YO(25)), RCT(1, 7), P1); \
    L1 = CO_FMA(YO(2), RCT(1, 6), L1); \
    CO_WAIT_Y(0); \
    CO_GET(0, 19, 0, 1); \
    CO_GET(1, 20, 1, 1); \
    CO_GET(2, 21, 0, 1); \
    v0 = CO_ADD(P0, P1); \
    v1 = CO_ADD(L0, L1); \
    P0 = CO_MUL(((YO(13) * YO(8)) * YO(7)), RCT(1, 5)); \
    L0 = CO_MUL(YO(6), RCT(1, 4)); \
    v2 = P0; \
    v3 = L0; \
    CO_PUT(0, v0, v1); \
    CO_PUT(1, v2, v3); \
    CO_ARRIVE_P(0); \
    G0a = CO_MUL(YO(2), RCT(1, 6)); \
    L0 = CO_MUL(YO(0), RCT(1, 7)); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 104, 102, 116); \
    TM_LD2(1, 2, 12, 106); \
    TM_LD2(1, 3, 28, 118); \
    P0 = CO_MUL((YO(13) * YO(8)), RCT(0, 3)); \
    L0 = CO_FMA(YO(2), RCT(0, 2), L0); \
    P0 = CO_FMA((YO(4) * YO(26)), RCT(0, 5), P0); \
    L0 = CO_FMA(YO(3), RCT(0, 4), L0); \
    const double2 s183 = RCS2(42); \
    P0 = CO_FMA((YO(3) * YO(39)), s183.x, P0); \
    L0 = CO_FMA((YO(13) * YO(2)), s183.y, L0); \
    CO_WAIT_Y(1); \
    CO_GET(3, 22, 1, 1); \
    v0 = G0a; \
    v1 = P0; \
    v2 = L0; \
    CO_PUT(7, v1, v0); \
    CO_PUT(8, v2, 0.0); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(3), RCT(0, 4)); \
    L0 = CO_MUL(YO(4), RCT(0, 5)); \
    g0a = CO_MUL(YO(1), RCT(0, 0)); \
    L0 = CO_FMA(YO(3), RCT(0, 1), L0); \
    g0a = CO_FMA(YO(4), RCT(0, 6), g0a); \
    L0 = CO_FMA(YO(2), RCT(0, 7), L0); \
    P0 = CO_MUL(YO(27), g0a); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 40, 124, 130); \
    TM_LD2(0, 2, 112, 120); \
    TM_LD2(0, 3, 144, 122); \
    P0 = CO_FMA((YO(21) * YO(3)), RCT(1, 0), P0); \
    L0 = CO_FMA(YO(2), RCT(1, 1), L0); \
    CO_WAIT_Y(0); \
    CO_GET(0, 23, 0, 1); \
    CO_GET(1, 24, 1, 1); \
    v0 = G0a; \
    v1 = P0; \
    v2 = L0; \
    CO_PUT(0, v1, v0); \
    CO_PUT(1, v2, 0.0); \
    CO_ARRIVE_P(0); \
    G0a = CO_MUL(YO(3), RCT(1, 7)); \
    L0 = CO_MUL(YO(1), RCT(1, 6)); \
    G0a = CO_FMA(YO(2), RCT(1, 3), G0a); \
    L0 = CO_FMA(YO(4), RCT(1, 2), L0); \
    P0 = CO_MUL((YO(21) * YO(4)), RCT(1, 4)); \
    L0 = CO_FMA(YO(5), RCT(1, 5), L0); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 120, 155, 157); \
    TM_LD2(1, 2, 4, 129); \
    TM_LD2(1, 3, 148, 150); \
    P0 = CO_FMA((YO(10) * YO(8)), RCT(0, 5), P0); \
    L0 = CO_FMA(YO(1), RCT(0, 4), L0); \
    CO_WAIT_Y(1); \
    CO_GET(3, 25, 0, 1); \
    v0 = G0a; \
    v1 = P0; \
    v2 = L0; \
    g0a = CO_MUL(YO(29), RCT(0, 2)); \
    L0 = CO_MUL(YO(0), RCT(0, 3)); \
    const double2 s184 = RCS2(14); \
    g0a = CO_FMA(YO(35), s184.x, g0a); \
    L0 = CO_FMA(YO(13), s184.y, L0); \
    P0 = CO_MUL(YO(2), g0a); \
    P0 = CO_FMA((YO(11) * YO(6)), RCT(0, 1), P0); \
    L0 = CO_FMA(YO(1), RCT(0, 0), L0); \
    P0 = CO_FMA((YO(13) * YO(4)), RCT(0, 7), P0); \
    L0 = CO_FMA(YO(2), RCT(0, 6), L0); \
    v3 = P0; \
    v4 = L0; \
    CO_PUT(7, v1, v0); \
    CO_PUT(8, v2, v3); \
    CO_PUT(9, v4, 0.0); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(0), RCT(0, 3)); \
    L0 = CO_MUL(YO(2), RCT(0, 2)); \
    TM_WAIT(1, 4); \
    P0 = CO_MUL((YO(17) * YO(5)), RCT(1, 5)); \
    L0 = CO_FMA(YO(4), RCT(1, 4), L0); \
    CO_WAIT_Y(0); \
    CO_GET(0, 26, 1, 1); \
    v0 = G0a; \
    v1 = P0; \
    v2 = L0; \
    const double2 s185 = RCS2(0); \
    g0a = CO_MUL(YO(4), s185.y); \
    L0 = CO_MUL(YO(3), s185.x); \
    const double2 s186 = RCS2(3); \
    g0a = CO_FMA(YO(12), s186.y, g0a); \
    L1 = CO_MUL(YO(13), s186.x); \
    const double2 s187 = RCS2(5); \
    g0a = CO_FMA(YO(7), s187.y, g0a); \
    L0 = CO_FMA(YO(6), s187.x, L0); \
    P0 = CO_MUL(YO(32), g0a); \
    const double2 s188 = RCS2(1); \
    g1a = CO_MUL(YO(4), s188.y); \
    L1 = CO_FMA(YO(3), s188.x, L1); \
    const double2 s189 = RCS2(4); \
    g1a = CO_FMA(YO(12), s189.y, g1a); \
    L0 = CO_FMA(YO(13), s189.x, L0); \
    const double2 s190 = RCS2(7); \
    g1a = CO_FMA(YO(7), s190.y, g1a); \
    L1 = CO_FMA(YO(6), s190.x, L1); \
    P1 = CO_MUL(YO(35), g1a); \
    const double2 s191 = RCS2(2); \
    g2a = CO_MUL(YO(12), s191.y); \
    L0 = CO_FMA(YO(13), s191.x, L0); \
    const double2 s192 = RCS2(6); \
    g2a = CO_FMA(YO(7), s192.y, g2a); \
    L1 = CO_FMA(YO(6), s192.x, L1); \
    P0 = CO_FMA(YO(33), g2a, P0); \
    v3 = CO_ADD(P0, P1); \
    v4 = CO_ADD(L0, L1); \
    CO_PUT(0, v1, v0); \
    CO_PUT(1, v2, v3); \
    CO_PUT(2, v4, 0.0); \
    CO_ARRIVE_P(0); \
    const double2 s193 = RCS2(17); \
    g0a = CO_MUL(YO(1), s193.x); \
    L0 = CO_MUL(YO(6), s193.y); \
    const double2 s194 = RCS2(21); \
    g0a = CO_FMA(YO(6), s194.x, g0a); \
    L1 = CO_MUL((YO(4) * YO(4)), s194.y); \
    P0 = CO_MUL(YO(32), g0a); \
    const double2 s195 = RCS2(12); \
    g1a = CO_MUL(YO(1), s195.x); \
    L0 = CO_FMA(YO(6), s195.y, L0); \
    const double2 s196 = RCS2(16); \
    g1a = CO_FMA(YO(4), s196.x, g1a); \
    L1 = CO_FMA(YO(5), s196.y, L1); \
    P1 = CO_MUL(YO(35), g1a); \
    g2a = CO_MUL(YO(12), RCT(1, 1)); \
    L0 = CO_FMA(YO(13), RCT(1, 0), L0); \
    g2a = CO_FMA(YO(7), RCT(1, 3), g2a); \
    L1 = CO_FMA(YO(6), RCT(1, 2), L1); \
    P0 = CO_FMA(YO(23), g2a, P0); \
    P1 = CO_FMA((YO(4) * YO(34)), RCT(1, 7), P1); \
    L0 = CO_FMA(YO(3), RCT(1, 6), L0); \
    const double2 s197 = RCS2(10); \
    P0 = CO_FMA(YO(35), s197.x, P0); \
    L1 = CO_FMA(YO(2), s197.y, L1); \
    CO_WAIT_Y(1); \
    CO_GET(3, 27, 0, 1); \
    CO_GET(4, 28, 1, 1); \
    v0 = CO_ADD(P0, P1); \
    v1 = CO_ADD(L0, L1); \
    CO_PUT(7, v0, v1); \
    CO_ARRIVE_P(1); \
    const double2 s198 = RCS2(17); \
    G0a = CO_MUL(YO(6), s198.y); \
    L0 = CO_MUL(YO(1), s198.x); \
    const double2 s199 = RCS2(18); \
    G0a = CO_FMA(YO(4), s199.y, G0a); \
    L1 = CO_MUL(YO(3), s199.x); \
    const double2 s200 = RCS2(21); \
    G0a = CO_FMA((YO(4) * YO(4)), s200.y, G0a); \
    L0 = CO_FMA(YO(6), s200.x, L0); \
    const double2 s201 = RCS2(22); \
    G0a = CO_FMA(YO(5), s201.y, G0a); \
    L1 = CO_FMA(YO(4), s201.x, L1); \
    const double2 s202 = RCS2(23); \
    G0a = CO_FMA(YO(2), s202.y, G0a); \
    L0 = CO_ADD(L0, s202.x); \
    const double2 s203 = RCS2(0); \
    e30a = CO_MUL(YO(3), s203.x); \
    L1 = CO_FMA(YO(4), s203.y, L1); \
    const double2 s204 = RCS2(3); \
    e30a = CO_FMA(YO(13), s204.x, e30a); \
    L0 = CO_FMA(YO(12), s204.y, L0); \
    const double2 s205 = RCS2(5); \
    e30a = CO_FMA(YO(6), s205.x, e30a); \
    L1 = CO_FMA(YO(7), s205.y, L1); \
    CO_WAIT_Y(0); \
    CO_GET(0, 29, 0, 1); \
    CO_GET(1, 30, 1, 1); \
    P0 = CO_MUL(YO(30), e30a); \
    v0 = G0a; \
    v1 = P0; \
    v2 = CO_ADD(L0, L1); \
    CO_PUT(0, v1, v0); \
    CO_PUT(1, v2, 0.0); \
    CO_ARRIVE_P(0); \
    e31a = CO_MUL(YO(3), RCT(1, 6)); \
    L0 = CO_MUL(YO(4), RCT(1, 7)); \
    CO_WAIT_Y(1); \
    CO_GET(3, 31, 0, 1); \
    P0 = CO_MUL(YO(31), e31a); \
    v0 = P0; \
    v1 = L0; \
    const double2 s206 = RCS2(9); \
    g0a = CO_MUL(YO(6), s206.x); \
    L0 = CO_MUL(YO(4), s206.y); \
    const double2 s207 = RCS2(13); \
    g0a = CO_FMA(YO(9), s207.y, g0a); \
    L0 = CO_FMA(YO(8), s207.x, L0); \
    P0 = CO_MUL(YO(18), g0a); \
    const double2 s208 = RCS2(10); \
    P0 = CO_FMA((YO(31) * YO(2)), s208.y, P0); \
    L0 = CO_ADD(L0, s208.x); \
    const double2 s209 = RCS2(11); \
    P0 = CO_FMA((YO(13) * YO(11)), s209.y, P0); \
    L0 = CO_ADD(L0, s209.x); \
    const double2 s210 = RCS2(15); \
    P0 = CO_FMA((YO(16) * YO(5)), s210.y, P0); \
    L0 = CO_FMA(YO(2), s210.x, L0); \
    v2 = P0; \
    v3 = L0; \
    const double2 s211 = RCS2(25); \
    g0a = CO_MUL(YO(21), s211.x); \
    L0 = CO_MUL(YO(2), s211.y); \
    const double2 s212 = RCS2(34); \
    g0a = CO_FMA(YO(38), s212.x, g0a); \
    L1 = CO_MUL(YO(12), s212.y); \
    const double2 s213 = RCS2(39); \
    g0a = CO_FMA((YO(10) * YO(8)), s213.y, g0a); \
    L0 = CO_FMA(YO(1), s213.x, L0); \
    P0 = CO_MUL(YO(13), g0a); \
    const double2 s214 = RCS2(79); \
    g1a = CO_MUL(YO(1), s214.x); \
    const double2 s215 = RCS2(81); \
    g1a = CO_FMA(YO(6), s215.x, g1a); \
    P1 = CO_MUL(YO(45), g1a); \
    g2a = CO_MUL(YO(6), s214.y); \
    g2a = CO_FMA(YO(7), s215.y, g2a); \
    L1 = CO_FMA(YO(22), g2a, L1); \
    const double2 s216 = RCS2(24); \
    P0 = CO_FMA((YO(16) * YO(8)), s216.y, P0); \
    L0 = CO_FMA(YO(3), s216.x, L0); \
    const double2 s217 = RCS2(31); \
    P1 = CO_FMA(YO(38), s217.y, P1); \
    L1 = CO_FMA(YO(2), s217.x, L1); \
    const double2 s218 = RCS2(32); \
    P0 = CO_FMA((YO(2) * YO(38)), s218.x, P0); \
    L0 = CO_FMA(YO(0), s218.y, L0); \
    v4 = CO_ADD(P0, P1); \
    v5 = CO_ADD(L0, L1); \
    CO_PUT(7, v0, v1); \
    CO_PUT(8, v2, v3); \
    CO_PUT(9, v4, v5); \
    CO_ARRIVE_P(1); \
    CO_WAIT_Y(0); \
    CO_GET(0, 32, 1, 1); \
    CO_GET(1, 33, 0, 1); \
    const double2 s219 = RCS2(31); \
    G0a = CO_MUL(YO(2), s219.x); \
    L0 = s219.y; \
    const double2 s220 = RCS2(32); \
    G0a = CO_FMA(YO(0), s220.y, G0a); \
    L1 = CO_MUL(YO(2), s220.x); \
    const double2 s221 = RCS2(33); \
    G0a = CO_FMA(YO(6), s221.y, G0a); \
    L0 = CO_FMA(YO(1), s221.x, L0); \
    const double2 s222 = RCS2(34); \
    G0a = CO_FMA(YO(12), s222.y, G0a); \
    L1 = CO_FMA(YO(13), s222.x, L1); \
    const double2 s223 = RCS2(41); \
    g0a = CO_MUL(YO(4), s223.x); \
    L0 = CO_FMA(YO(5), s223.y, L0); \
    const double2 s224 = RCS2(45); \
    g0a = CO_FMA(YO(1), s224.y, g0a); \
    L1 = CO_FMA(YO(6), s224.x, L1); \
    P0 = CO_MUL(YO(39), g0a); \
    const double2 s225 = RCS2(44); \
    P1 = CO_MUL(YO(39), s225.y); \
    L0 = CO_FMA(YO(2), s225.x, L0); \
    const double2 s226 = RCS2(77); \
    P0 = CO_FMA(YO(45), s226.x, P0); \
    L1 = CO_FMA(YO(22), s226.y, L1); \
    const double2 s227 = RCS2(80); \
    P1 = CO_FMA((YO(6) * YO(45)), s227.x, P1); \
    L0 = CO_FMA((YO(21) * YO(7)), s227.y, L0); \
    const double2 s228 = RCS2(97); \
    P0 = CO_FMA((YO(2) * YO(48)), s228.x, P0); \
    L1 = CO_FMA((YO(0) * YO(16)), s228.y, L1); \
    v0 = G0a; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    CO_PUT(0, v1, v0); \
    CO_PUT(1, v2, 0.0); \
    CO_ARRIVE_P(0); \
    const double2 s229 = RCS2(41); \
    G0a = CO_MUL(YO(5), s229.y); \
    L0 = CO_MUL(YO(4), s229.x); \
    const double2 s230 = RCS2(43); \
    G0a = CO_FMA(YO(0), s230.y, G0a); \
    L1 = CO_MUL(YO(2), s230.x); \
    const double2 s231 = RCS2(44); \
    G0a = CO_FMA(YO(2), s231.x, G0a); \
    L0 = CO_ADD(L0, s231.y); \
    const double2 s232 = RCS2(45); \
    G0a = CO_FMA(YO(6), s232.x, G0a); \
    L1 = CO_FMA(YO(1), s232.y, L1); \
    const double2 s233 = RCS2(96); \
    g0a = CO_MUL(YO(48), s233.x); \
    L0 = CO_FMA(YO(18), s233.y, L0); \
    const double2 s234 = RCS2(101); \
    g0a = CO_FMA(YO(47), s234.x, g0a); \
    L1 = CO_FMA(YO(13), s234.y, L1); \
    P0 = CO_MUL(YO(2), g0a); \
    const double2 s235 = RCS2(65); \
    P1 = CO_MUL(YO(42), s235.y); \
    L0 = CO_FMA(YO(2), s235.x, L0); \
    const double2 s236 = RCS2(92); \
    P0 = CO_FMA(YO(48), s236.x, P0); \
    L1 = CO_FMA(YO(16), s236.y, L1); \
    CO_WAIT_Y(1); \
    CO_GET(3, 34, 1, 1); \
    CO_GET(4, 35, 0, 1); \
    CO_GET(5, 36, 1, 1); \
    v0 = G0a; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    const double2 s237 = RCS2(55); \
    g0a = CO_MUL(YO(4), s237.y); \
    L0 = CO_MUL(YO(3), s237.x); \
    const double2 s238 = RCS2(58); \
    g0a = CO_FMA(YO(5), s238.y, g0a); \
    L0 = CO_FMA(YO(4), s238.x, L0); \
    P0 = CO_MUL(YO(41), g0a); \
    const double2 s239 = RCS2(54); \
    g1a = CO_MUL(YO(0), s239.y); \
    L0 = CO_FMA(YO(2), s239.x, L0); \
    const double2 s240 = RCS2(56); \
    g1a = CO_FMA(YO(4), s240.y, g1a); \
    L0 = CO_FMA(YO(3), s240.x, L0); \
    P0 = CO_FMA(YO(42), g1a, P0); \
    v3 = P0; \
    v4 = L0; \
    CO_PUT(7, v1, v0); \
    CO_PUT(8, v2, v3); \
    CO_PUT(9, v4, 0.0); \
    CO_ARRIVE_P(1); \
    const double2 s241 = RCS2(62); \
    G0a = CO_MUL(YO(2), s241.x); \
    L0 = s241.y; \
    const double2 s242 = RCS2(63); \
    G0a = CO_FMA(YO(6), s242.y, G0a); \
    L0 = CO_FMA(YO(1), s242.x, L0); \
    const double2 s243 = RCS2(61); \
    P0 = CO_MUL(YO(42), s243.y); \
    L0 = CO_ADD(L0, s243.x); \
    CO_WAIT_Y(0); \
    CO_GET(0, 37, 0, 1); \
    CO_GET(1, 38, 1, 1); \
    v0 = G0a; \
    v1 = P0; \
    v2 = L0; \
    CO_PUT(0, v1, v0); \
    CO_PUT(1, v2, 0.0); \
    CO_ARRIVE_P(0); \
    const double2 s244 = RCS2(65); \
    e39a = CO_MUL(YO(2), s244.x); \
    L0 = s244.y; \
    const double2 s245 = RCS2(66); \
    e39a = CO_FMA(YO(6), s245.y, e39a); \
    L0 = CO_FMA(YO(1), s245.x, L0); \
    const double2 s246 = RCS2(60); \
    e40a = CO_MUL(YO(6), s246.x); \
    L0 = CO_FMA(YO(7), s246.y, L0); \
    const double2 s247 = RCS2(64); \
    P0 = CO_MUL((YO(16) * YO(13)), s247.y); \
    L0 = CO_ADD(L0, s247.x); \
    CO_WAIT_Y(1); \
    CO_GET(3, 39, 0, 1); \
    CO_GET(4, 40, 1, 1); \
    P0 = CO_FMA(YO(39), e39a, P0); \
    P0 = CO_FMA(YO(40), e40a, P0); \
    v0 = P0; \
    v1 = L0; \
    const double2 s248 = RCS2(70); \
    P0 = CO_MUL((YO(22) * YO(16)), s248.y); \
    L0 = CO_MUL(YO(2), s248.x); \
    const double2 s249 = RCS2(98); \
    P0 = CO_FMA((YO(2) * YO(48)), s249.x, P0); \
    L0 = CO_FMA((YO(0) * YO(13)), s249.y, L0); \
    const double2 s250 = RCS2(103); \
    P0 = CO_FMA((YO(4) * YO(47)), s250.x, P0); \
    L0 = CO_FMA((YO(5) * YO(2)), s250.y, L0); \
    v2 = P0; \
    v3 = L0; \
    CO_PUT(7, v0, v1); \
    CO_PUT(8, v2, v3); \
    CO_ARRIVE_P(1); \
    CO_WAIT_Y(0); \
    CO_GET(0, 41, 0, 1); \
    const double2 s251 = RCS2(77); \
    P0 = CO_MUL((YO(38) * YO(22)), s251.y); \
    L0 = s251.x; \
    v0 = P0; \
    v1 = L0; \
    const double2 s252 = RCS2(86); \
    g0a = CO_MUL((YO(18) * YO(0)), s252.y); \
    L0 = CO_MUL(YO(2), s252.x); \
    const double2 s253 = RCS2(87); \
    g0a = CO_FMA((YO(18) * YO(5)), s253.y, g0a); \
    L1 = CO_MUL(YO(4), s253.x); \
    P0 = CO_MUL(YO(48), g0a); \
    const double2 s254 = RCS2(82); \
    L0 = CO_ADD(L0, s254.x); \
    const double2 s255 = RCS2(83); \
    L1 = CO_FMA(YO(2), s255.x, L1); \
    const double2 s256 = RCS2(84); \
    L0 = CO_FMA(YO(2), s256.x, L0); \
    const double2 s257 = RCS2(85); \
    L1 = CO_FMA(YO(2), s257.x, L1); \
    v2 = P0; \
    v3 = CO_ADD(L0, L1); \
    CO_PUT(0, v0, v1); \
    CO_PUT(1, v2, v3); \
    CO_ARRIVE_P(0); \
    const double2 s258 = RCS2(103); \
    e43a = CO_MUL((YO(5) * YO(2)), s258.y); \
    L0 = CO_MUL(YO(4), s258.x); \
    const double2 s259 = RCS2(100); \
    g0a = CO_MUL(YO(18), s259.y); \
    L0 = CO_FMA(YO(2), s259.x, L0); \
    const double2 s260 = RCS2(102); \
    g0a = CO_FMA((YO(22) * YO(0)), s260.y, g0a); \
    L0 = CO_FMA(YO(2), s260.x, L0); \
    P0 = CO_MUL(YO(16), g0a); \
    const double2 s261 = RCS2(99); \
    P0 = CO_FMA((YO(38) * YO(13)), s261.y, P0); \
    L0 = CO_ADD(L0, s261.x); \
    CO_WAIT_Y(1); \
    CO_GET(3, 42, 1, 1); \
    CO_GET(4, 43, 0, 1); \
    P0 = CO_FMA(YO(43), e43a, P0); \
    v0 = P0; \
    v1 = L0; \
    const double2 s262 = RCS2(91); \
    g0a = CO_MUL(YO(38), s262.y); \
    L0 = s262.x; \
    const double2 s263 = RCS2(96); \
    g0a = CO_FMA(YO(39), s263.y, g0a); \
    L0 = CO_FMA(YO(2), s263.x, L0); \
    P0 = CO_MUL(YO(18), g0a); \
    const double2 s264 = RCS2(98); \
    P0 = CO_FMA(((YO(43) * YO(0)) * YO(13)), s264.y, P0); \
    L0 = CO_FMA(YO(2), s264.x, L0); \
    v2 = P0; \
    v3 = L0; \
    CO_PUT(7, v0, v1); \
    CO_PUT(8, v2, v3); \
    CO_ARRIVE_P(1); \
    CO_WAIT_Y(0); \
    CO_GET(0, 44, 1, 1); \
    CO_GET(1, 45, 0, 1); \
    CO_GET(2, 46, 1, 1); \
} while (0)
#define UC_CO_SUMS_1() do { \
    double G0a, G0b, G1a, G1b, H0, L0, L1, P0, P1, e0a, e0b, e11a, e13a, e1a, e2a, e2b, e30a, e31a, e40a, e4a, e4b, e5a, e8a, f2a, f8a, g0a, g0b, g1a, g1b, g2a, v0, v1, v2, v3, v4, v5, v6; \
    TM_LD8(0, 0, 0, 1, 2, 164, 165); \
    TM_WAIT(0, 4); \
    TM_LD8(1, 0, 112, 43, 70, 82, 87); \
    g0a = CO_MUL(YO(4), RCT(0, 1)); \
    L0 = CO_MUL(YO(3), RCT(0, 0)); \
    g0b = CO_MUL(YO(5), RCT(0, 3)); \
    L1 = CO_MUL(YO(4), RCT(0, 2)); \
    g0a = CO_FMA(YO(30), RCT(0, 4), g0a); \
    L0 = CO_FMA(YO(33), RCT(0, 5), L0); \
    g0b = CO_FMA(YO(30), RCT(0, 6), g0b); \
    L1 = CO_FMA(YO(32), RCT(0, 7), L1); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 144, 97); \
    TM_LD2(0, 1, 188, 153); \
    TM_LD2(0, 2, 196, 166); \
    TM_LD2(0, 3, 208, 4); \
    g0a = CO_FMA(YO(13), RCT(1, 0), g0a); \
    L0 = CO_FMA(YO(15), RCT(1, 1), L0); \
    g0b = CO_FMA(YO(17), RCT(1, 2), g0b); \
    L1 = CO_FMA(YO(11), RCT(1, 3), L1); \
    g0a = CO_FMA(YO(18), RCT(1, 4), g0a); \
    L0 = CO_FMA(YO(16), RCT(1, 5), L0); \
    g0b = CO_FMA(YO(16), RCT(1, 6), g0b); \
    L1 = CO_FMA(YO(22), RCT(1, 7), L1); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 264, 25, 32); \
    TM_LD2(1, 2, 240, 11); \
    TM_LD2(1, 3, 256, 17); \
    g0a = CO_FMA(YO(22), RCT(0, 0), g0a); \
    L0 = CO_FMA(YO(21), RCT(0, 1), L0); \
    g0b = CO_FMA(YO(31), RCT(0, 2), g0b); \
    L1 = CO_FMA(YO(23), RCT(0, 3), L1); \
    g0a = CO_FMA(YO(30), RCT(0, 4), g0a); \
    L0 = CO_FMA(YO(35), RCT(0, 5), L0); \
    g0b = CO_FMA(YO(2), RCT(0, 6), g0b); \
    L1 = CO_ADD(L1, RCT(0, 7)); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 288, 42); \
    TM_LD2(0, 1, 384, 121); \
    TM_LD2(0, 2, 392, 152); \
    TM_LD2(0, 3, 456, 131); \
    g0a = CO_FMA(YO(6), RCT(1, 4), g0a); \
    L0 = CO_FMA(YO(1), RCT(1, 5), L0); \
    g0b = CO_FMA(YO(7), RCT(1, 6), g0b); \
    L1 = CO_FMA(YO(6), RCT(1, 7), L1); \
    g0a = CO_FMA(YO(10), RCT(1, 0), g0a); \
    L0 = CO_FMA(YO(8), RCT(1, 1), L0); \
    g0b = CO_FMA(YO(11), RCT(1, 2), g0b); \
    L1 = CO_FMA(YO(10), RCT(1, 3), L1); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 408, 50, 63); \
    TM_LD2(1, 2, 328, 62); \
    TM_LD2(1, 3, 420, 96); \
    g0a = CO_FMA(YO(13), RCT(0, 0), g0a); \
    L0 = CO_FMA(YO(14), RCT(0, 1), L0); \
    g0b = CO_FMA(YO(28), RCT(0, 2), g0b); \
    L1 = CO_FMA(YO(11), RCT(0, 3), L1); \
    g0a = CO_FMA(YO(31), RCT(0, 4), g0a); \
    L0 = CO_FMA(YO(34), RCT(0, 5), L0); \
    g0b = CO_FMA(YO(29), RCT(0, 6), g0b); \
    L1 = CO_FMA(YO(17), RCT(0, 7), L1); \
    const double2 s0 = RCS2(84); \
    g0a = CO_FMA(YO(46), s0.x, g0a); \
    const double2 s1 = RCS2(85); \
    g0b = CO_FMA(YO(46), s1.x, g0b); \
    P0 = CO_MUL(YO(2), CO_ADD(g0a, g0b)); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 88, 13); \
    TM_LD2(0, 1, 148, 101); \
    TM_LD2(0, 2, 172, 134); \
    TM_LD2(0, 3, 176, 144); \
    g1a = CO_MUL(YO(3), RCT(1, 4)); \
    L0 = CO_FMA(YO(8), RCT(1, 5), L0); \
    g1a = CO_FMA(YO(1), RCT(1, 2), g1a); \
    L1 = CO_FMA(YO(9), RCT(1, 3), L1); \
    P1 = CO_MUL(YO(14), g1a); \
    P0 = CO_FMA((YO(13) * YO(13)), RCT(1, 0), P0); \
    L0 = CO_FMA(YO(16), RCT(1, 1), L0); \
    P1 = CO_FMA(YO(16), RCT(1, 6), P1); \
    L1 = CO_FMA(YO(21), RCT(1, 7), L1); \
    CO_WAIT_Y(1); \
    CO_GET(3, 47, 1, 0); \
    CO_GET(4, 48, 0, 0); \
    v0 = CO_ADD(P0, P1); \
    v1 = CO_ADD(L0, L1); \
    CO_PUT(1, v0, v1); \
    CO_ARRIVE_P(0); \
    YOS(0) = YO(4); \
    YOS(1) = YO(6); \
    YOS(2) = YO(2); \
    YOS(3) = YO(13); \
    YOS(4) = YO(16); \
    YOS(5) = YO(14); \
    YOS(6) = YO(8); \
    YOS(7) = YO(22); \
    CO_CHECK(); \
    G0a = CO_MUL(YO(9), RCT(1, 3)); \
    L0 = CO_MUL(YO(14), RCT(1, 2)); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 240, 11, 92); \
    TM_LD2(1, 2, 204, 158); \
    TM_LD2(1, 3, 236, 14); \
    g0a = CO_MUL(YO(3), RCT(0, 0)); \
    L1 = CO_MUL(YO(4), RCT(0, 1)); \
    g0b = CO_MUL(YO(21), RCT(0, 3)); \
    L0 = CO_FMA(YO(22), RCT(0, 2), L0); \
    g0a = CO_FMA(YO(28), RCT(0, 5), g0a); \
    L1 = CO_FMA(YO(29), RCT(0, 4), L1); \
    g0b = CO_FMA(YO(23), RCT(0, 6), g0b); \
    L0 = CO_FMA(YO(31), RCT(0, 7), L0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 248, 16, 29); \
    TM_LD2(0, 2, 356, 85); \
    TM_LD2(0, 3, 484, 74); \
    g0a = CO_FMA(YO(34), RCT(1, 5), g0a); \
    L1 = CO_FMA(YO(31), RCT(1, 4), L1); \
    g0b = CO_FMA(YO(4), RCT(1, 6), g0b); \
    L0 = CO_FMA(YO(5), RCT(1, 7), L0); \
    g0a = CO_FMA(YO(2), RCT(1, 0), g0a); \
    H0 = RCT(1, 1); \
    g0b = CO_FMA(YO(22), RCT(1, 3), g0b); \
    L1 = CO_FMA(YO(16), RCT(1, 2), L1); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 312, 48, 55); \
    TM_LD2(1, 2, 32, 0); \
    TM_LD2(1, 3, 372, 114); \
    g0a = CO_FMA(YO(6), RCT(0, 0), g0a); \
    L0 = CO_FMA(YO(7), RCT(0, 1), L0); \
    g0b = CO_FMA(YO(8), RCT(0, 3), g0b); \
    L1 = CO_FMA(YO(10), RCT(0, 2), L1); \
    g0a = CO_FMA(YO(16), RCT(0, 5), g0a); \
    L0 = CO_FMA(YO(18), RCT(0, 4), L0); \
    g0b = CO_FMA(YO(11), RCT(0, 7), g0b); \
    L1 = CO_FMA(YO(17), RCT(0, 6), L1); \
    const double2 s2 = RCS2(45); \
    g0a = CO_FMA(YO(38), s2.x, g0a); \
    L0 = CO_FMA(YO(39), s2.y, L0); \
    const double2 s3 = RCS2(51); \
    g0b = CO_FMA(YO(41), s3.y, g0b); \
    L1 = CO_FMA(YO(40), s3.x, L1); \
    const double2 s4 = RCS2(63); \
    g0a = CO_FMA(YO(39), s4.y, g0a); \
    L0 = CO_FMA(YO(41), s4.x, L0); \
    P0 = CO_MUL(YO(6), CO_ADD(g0a, g0b)); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 336, 67, 99); \
    TM_LD2(0, 2, 156, 104); \
    TM_LD2(0, 3, 228, 115); \
    g1a = CO_MUL(YO(3), RCT(1, 5)); \
    L1 = CO_FMA(YO(2), RCT(1, 4), L1); \
    g1a = CO_FMA(YO(11), RCT(1, 1), g1a); \
    L0 = CO_FMA(YO(13), RCT(1, 0), L0); \
    g1a = CO_FMA((YO(8) * YO(2)), RCT(1, 3), g1a); \
    L1 = CO_FMA(YO(15), RCT(1, 2), L1); \
    g1a = CO_FMA((YO(8) * YO(8)), RCT(1, 7), g1a); \
    L0 = CO_FMA(YO(26), RCT(1, 6), L0); \
    P1 = CO_MUL(YO(4), g1a); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 212, 9); \
    TM_LD2(1, 1, 228, 115); \
    TM_LD2(1, 2, 380, 119); \
    TM_LD2(1, 3, 492, 100); \
    g2a = CO_MUL(YO(3), RCT(0, 1)); \
    L1 = CO_FMA(YO(20), RCT(0, 0), L1); \
    g2a = CO_FMA(YO(11), RCT(0, 3), g2a); \
    L0 = CO_FMA(YO(22), RCT(0, 2), L0); \
    const double2 s5 = RCS2(30); \
    g2a = CO_FMA(YO(25), s5.y, g2a); \
    L1 = CO_FMA(YO(37), s5.x, L1); \
    P0 = CO_FMA(YO(10), g2a, P0); \
    g0a = CO_MUL(YO(11), RCT(0, 5)); \
    L0 = CO_FMA(YO(21), RCT(0, 4), L0); \
    g0a = CO_FMA((YO(9) * YO(2)), RCT(0, 7), g0a); \
    L1 = CO_FMA(YO(26), RCT(0, 6), L1); \
    P1 = CO_FMA(YO(8), g0a, P1); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 0, 1, 2); \
    TM_LD2(0, 2, 240, 11); \
    TM_LD2(0, 3, 316, 55); \
    P0 = CO_FMA(YO(6), RCT(1, 1), P0); \
    L0 = CO_FMA(YO(2), RCT(1, 0), L0); \
    P1 = CO_FMA((YO(20) * YO(9)), RCT(1, 5), P1); \
    L1 = CO_FMA(YO(27), RCT(1, 4), L1); \
    P0 = CO_FMA((YO(23) * YO(3)), RCT(1, 7), P0); \
    L0 = CO_FMA(YO(22), RCT(1, 6), L0); \
    v0 = G0a; \
    v1 = H0; \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    CO_PUT(8, v2, v0); \
    CO_PUT(9, v3, v1); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(26), RCT(1, 2)); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 8, 164, 165); \
    TM_LD4(1, 2, 112, 43, 70); \
    G0a = CO_FMA(YO(15), RCT(0, 6), G0a); \
    L0 = CO_MUL(YO(6), RCT(0, 4)); \
    e0a = CO_MUL(YO(3), RCT(0, 0)); \
    L1 = CO_MUL(YO(4), RCT(0, 1)); \
    e0b = CO_MUL(YO(4), RCT(0, 2)); \
    L0 = CO_FMA(YO(5), RCT(0, 3), L0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 120, 82, 87); \
    TM_LD2(0, 2, 144, 97); \
    TM_LD2(0, 3, 188, 153); \
    e0a = CO_FMA(YO(33), RCT(1, 1), e0a); \
    L1 = CO_FMA(YO(30), RCT(1, 0), L1); \
    e0b = CO_FMA(YO(32), RCT(1, 3), e0b); \
    L0 = CO_FMA(YO(30), RCT(1, 2), L0); \
    e0a = CO_FMA(YO(15), RCT(1, 5), e0a); \
    L1 = CO_FMA(YO(13), RCT(1, 4), L1); \
    e0b = CO_FMA(YO(11), RCT(1, 7), e0b); \
    L0 = CO_FMA(YO(17), RCT(1, 6), L0); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 264, 25, 32); \
    TM_LD2(1, 2, 196, 166); \
    TM_LD2(1, 3, 256, 17); \
    e0a = CO_FMA(YO(16), RCT(0, 1), e0a); \
    L1 = CO_FMA(YO(18), RCT(0, 0), L1); \
    e0b = CO_FMA(YO(22), RCT(0, 3), e0b); \
    L0 = CO_FMA(YO(16), RCT(0, 2), L0); \
    e0a = CO_FMA(YO(21), RCT(0, 5), e0a); \
    L1 = CO_FMA(YO(22), RCT(0, 4), L1); \
    e0b = CO_FMA(YO(23), RCT(0, 7), e0b); \
    L0 = CO_FMA(YO(31), RCT(0, 6), L0); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 288, 42); \
    TM_LD2(0, 1, 384, 121); \
    TM_LD2(0, 2, 392, 152); \
    TM_LD2(0, 3, 456, 131); \
    e0a = CO_FMA(YO(35), RCT(1, 5), e0a); \
    L1 = CO_FMA(YO(30), RCT(1, 4), L1); \
    e0b = CO_FMA(YO(6), RCT(1, 7), e0b); \
    L0 = CO_FMA(YO(7), RCT(1, 6), L0); \
    e0a = CO_FMA(YO(8), RCT(1, 1), e0a); \
    L1 = CO_FMA(YO(10), RCT(1, 0), L1); \
    e0b = CO_FMA(YO(10), RCT(1, 3), e0b); \
    L0 = CO_FMA(YO(11), RCT(1, 2), L0); \
    TM_WAIT(0, 4); \
    TM_LD8(1, 0, 32, 0, 18, 10, 21); \
    e0a = CO_FMA(YO(14), RCT(0, 1), e0a); \
    L1 = CO_FMA(YO(13), RCT(0, 0), L1); \
    e0b = CO_FMA(YO(11), RCT(0, 3), e0b); \
    L0 = CO_FMA(YO(28), RCT(0, 2), L0); \
    e0a = CO_FMA(YO(34), RCT(0, 5), e0a); \
    L1 = CO_FMA(YO(31), RCT(0, 4), L1); \
    e0b = CO_FMA(YO(17), RCT(0, 7), e0b); \
    L0 = CO_FMA(YO(29), RCT(0, 6), L0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 320, 54, 59); \
    TM_LD2(0, 2, 368, 112); \
    TM_LD2(0, 3, 440, 105); \
    g0a = CO_MUL(YO(3), RCT(1, 1)); \
    H0 = RCT(1, 0); \
    g0b = CO_MUL(YO(5), RCT(1, 3)); \
    L1 = CO_FMA(YO(7), RCT(1, 2), L1); \
    g0a = CO_FMA(YO(4), RCT(1, 5), g0a); \
    L0 = CO_FMA(YO(6), RCT(1, 4), L0); \
    g0b = CO_FMA(YO(8), RCT(1, 6), g0b); \
    L1 = CO_FMA(YO(9), RCT(1, 7), L1); \
    TM_WAIT(0, 4); \
    TM_LD8(1, 0, 64, 12, 45, 66, 90); \
    g0a = CO_FMA(YO(15), RCT(0, 0), g0a); \
    L0 = CO_FMA(YO(11), RCT(0, 1), L0); \
    g0b = CO_FMA(YO(14), RCT(0, 2), g0b); \
    L1 = CO_FMA(YO(11), RCT(0, 3), L1); \
    g0a = CO_FMA(YO(26), RCT(0, 4), g0a); \
    g0b = CO_FMA(YO(21), RCT(0, 6), g0b); \
    L0 = CO_FMA(YO(25), RCT(0, 7), L0); \
    P1 = CO_MUL(YO(4), CO_ADD(g0a, g0b)); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 304, 46, 51); \
    TM_LD2(0, 2, 104, 137); \
    TM_LD2(0, 3, 224, 113); \
    g1a = CO_MUL(YO(5), RCT(1, 1)); \
    L1 = CO_FMA(YO(6), RCT(1, 0), L1); \
    g1a = CO_FMA(YO(13), RCT(1, 2), g1a); \
    L0 = CO_FMA(YO(11), RCT(1, 3), L0); \
    g1a = CO_FMA(YO(20), RCT(1, 4), g1a); \
    L1 = CO_FMA(YO(8), RCT(1, 5), L1); \
    g1a = CO_FMA(YO(16), RCT(1, 6), g1a); \
    L0 = CO_FMA(YO(23), RCT(1, 7), L0); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 344, 68, 71); \
    TM_LD2(1, 2, 224, 113); \
    TM_LD2(1, 3, 416, 65); \
    g1a = CO_FMA(YO(26), RCT(0, 6), g1a); \
    P0 = CO_MUL(YO(3), g1a); \
    g2a = CO_MUL(YO(10), RCT(0, 5)); \
    L1 = CO_FMA(YO(23), RCT(0, 4), L1); \
    g2a = CO_FMA(YO(14), RCT(0, 0), g2a); \
    L0 = CO_FMA(YO(16), RCT(0, 1), L0); \
    g2a = CO_FMA(YO(13), RCT(0, 2), g2a); \
    L1 = CO_FMA(YO(18), RCT(0, 3), L1); \
    P1 = CO_FMA(YO(13), g2a, P1); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 228, 115); \
    TM_LD2(0, 1, 316, 55); \
    TM_LD2(0, 2, 368, 112); \
    TM_LD2(0, 3, 416, 65); \
    g0a = CO_MUL(YO(20), RCT(1, 0)); \
    L0 = CO_FMA(YO(11), RCT(1, 1), L0); \
    g0a = CO_FMA(YO(15), RCT(1, 3), g0a); \
    L1 = CO_FMA(YO(17), RCT(1, 2), L1); \
    P0 = CO_FMA(YO(5), g0a, P0); \
    g1a = CO_MUL(YO(14), RCT(1, 6)); \
    g1a = CO_FMA(YO(14), RCT(1, 6), g1a); \
    P1 = CO_FMA(YO(14), g1a, P1); \
    const double2 s6 = RCS2(70); \
    g2a = CO_MUL(YO(22), s6.y); \
    L0 = CO_FMA(YO(43), s6.x, L0); \
    const double2 s7 = RCS2(100); \
    g2a = CO_FMA(YO(18), s7.y, g2a); \
    L1 = CO_FMA(YO(47), s7.x, L1); \
    P0 = CO_FMA(YO(16), g2a, P0); \
    g0a = CO_MUL(YO(8), RCT(1, 5)); \
    TM_WAIT(0, 4); \
    TM_LD8(1, 0, 48, 5, 7, 52, 136); \
    g0a = CO_FMA(YO(9), RCT(0, 1), g0a); \
    g0a = CO_FMA(YO(4), RCT(0, 3), g0a); \
    g0a = CO_FMA(YO(10), RCT(0, 5), g0a); \
    L0 = CO_FMA(YO(8), g0a, L0); \
    g1a = CO_MUL(YO(21), RCT(0, 7)); \
    g1a = CO_FMA(YO(21), RCT(0, 7), g1a); \
    L1 = CO_FMA(YO(2), g1a, L1); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 208, 4, 9); \
    TM_LD2(0, 2, 140, 80); \
    TM_LD2(0, 3, 152, 98); \
    P1 = CO_FMA(YO(5), RCT(1, 1), P1); \
    L0 = CO_FMA(YO(4), RCT(1, 0), L0); \
    P0 = CO_FMA(YO(4), RCT(1, 3), P0); \
    L1 = CO_FMA(YO(3), RCT(1, 2), L1); \
    P1 = CO_FMA(YO(12), RCT(1, 5), P1); \
    L0 = CO_FMA(YO(13), RCT(1, 4), L0); \
    P0 = CO_FMA(YO(23), RCT(1, 6), P0); \
    L1 = CO_FMA(YO(25), RCT(1, 7), L1); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 216, 24, 31); \
    TM_LD2(1, 2, 428, 75); \
    TM_LD2(1, 3, 432, 86); \
    P1 = CO_FMA(YO(19), RCT(0, 4), P1); \
    L0 = CO_FMA(YO(18), RCT(0, 5), L0); \
    P0 = CO_FMA(YO(22), RCT(0, 6), P0); \
    L1 = CO_FMA(YO(21), RCT(0, 7), L1); \
    L0 = CO_FMA(YO(2), RCT(0, 0), L0); \
    L1 = CO_FMA(YO(2), RCT(0, 0), L1); \
    P1 = CO_FMA(YO(6), RCT(0, 3), P1); \
    H0 = CO_ADD(H0, RCT(0, 2)); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 448, 111, 125); \
    TM_LD2(0, 2, 240, 11); \
    TM_LD2(0, 3, 436, 95); \
    P0 = CO_FMA(YO(10), RCT(1, 0), P0); \
    L0 = CO_FMA(YO(8), RCT(1, 1), L0); \
    P1 = CO_FMA(YO(11), RCT(1, 3), P1); \
    L1 = CO_FMA(YO(10), RCT(1, 2), L1); \
    P0 = CO_FMA(YO(17), RCT(1, 4), P0); \
    L0 = CO_FMA(YO(11), RCT(1, 5), L0); \
    P1 = CO_FMA(YO(18), RCT(1, 6), P1); \
    L1 = CO_FMA(YO(16), RCT(1, 7), L1); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 64, 12, 45); \
    TM_LD2(1, 2, 0, 1); \
    TM_LD2(1, 3, 208, 4); \
    P0 = CO_FMA(YO(16), RCT(0, 6), P0); \
    L0 = CO_FMA(YO(22), RCT(0, 7), L0); \
    P1 = CO_FMA((YO(15) * YO(8)), RCT(0, 1), P1); \
    L1 = CO_FMA(YO(26), RCT(0, 0), L1); \
    P0 = CO_FMA(YO(28), RCT(0, 2), P0); \
    L0 = CO_FMA(YO(11), RCT(0, 3), L0); \
    const double2 s8 = RCS2(10); \
    P1 = CO_FMA(YO(35), s8.x, P1); \
    L1 = CO_FMA(YO(31), s8.y, L1); \
    const double2 s9 = RCS2(23); \
    P0 = CO_FMA(YO(32), s9.x, P0); \
    L0 = CO_FMA(YO(31), s9.y, L0); \
    const double2 s10 = RCS2(31); \
    P1 = CO_FMA(YO(38), s10.y, P1); \
    L1 = CO_FMA(YO(36), s10.x, L1); \
    const double2 s11 = RCS2(62); \
    P0 = CO_FMA(YO(41), s11.y, P0); \
    L0 = CO_FMA(YO(39), s11.x, L0); \
    const double2 s12 = RCS2(65); \
    P1 = CO_FMA(YO(42), s12.y, P1); \
    L1 = CO_FMA(YO(39), s12.x, L1); \
    const double2 s13 = RCS2(84); \
    L0 = CO_FMA(YO(46), s13.x, L0); \
    CO_WAIT_Y(0); \
    CO_GET(0, 0, 0, 1); \
    G0a = CO_FMA(YO(0), RCT(0, 5), G0a); \
    P0 = CO_FMA(YO(0), CO_ADD(e0a, e0b), P0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 72, 66, 90); \
    TM_LD2(0, 2, 32, 0); \
    TM_LD2(0, 3, 224, 113); \
    P1 = CO_FMA(YO(0), RCT(1, 7), P1); \
    P0 = CO_FMA(YO(0), RCT(1, 7), P0); \
    v0 = G0a; \
    v1 = H0; \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    CO_PUT(2, v2, v0); \
    CO_PUT(3, v3, v1); \
    CO_ARRIVE_P(0); \
    G0a = CO_MUL(YO(4), RCT(1, 5)); \
    L0 = CO_MUL(YO(0), RCT(1, 4)); \
    G0b = CO_MUL(YO(6), RCT(1, 0)); \
    L1 = CO_MUL(YO(5), RCT(1, 1)); \
    G0a = CO_FMA(YO(11), RCT(1, 3), G0a); \
    L0 = CO_FMA(YO(13), RCT(1, 2), L0); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 88, 13); \
    TM_LD2(1, 1, 128, 77); \
    TM_LD2(1, 2, 336, 67); \
    TM_LD2(1, 3, 492, 100); \
    G0b = CO_FMA(YO(8), RCT(0, 1), G0b); \
    L1 = CO_FMA(YO(20), RCT(0, 0), L1); \
    G0a = CO_FMA(YO(23), RCT(0, 3), G0a); \
    L0 = CO_FMA(YO(16), RCT(0, 2), L0); \
    G0b = CO_FMA((YO(8) * YO(8)), RCT(0, 7), G0b); \
    L1 = CO_FMA(YO(26), RCT(0, 6), L1); \
    L0 = CO_FMA(YO(4), RCT(0, 5), L0); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 164, 132); \
    TM_LD2(0, 1, 180, 151); \
    TM_LD2(0, 2, 232, 3); \
    TM_LD2(0, 3, 260, 20); \
    e1a = CO_MUL(YO(4), RCT(1, 1)); \
    L1 = CO_FMA(YO(6), RCT(1, 0), L1); \
    e1a = CO_FMA(YO(20), RCT(1, 4), e1a); \
    L0 = CO_FMA(YO(10), RCT(1, 5), L0); \
    e1a = CO_FMA(YO(22), RCT(1, 6), e1a); \
    L1 = CO_FMA(YO(23), RCT(1, 7), L1); \
    g0a = CO_MUL(YO(18), RCT(1, 3)); \
    L0 = CO_FMA(YO(19), RCT(1, 2), L0); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 272, 33, 39); \
    TM_LD2(1, 2, 352, 83); \
    TM_LD2(1, 3, 424, 73); \
    g0b = CO_MUL(YO(28), RCT(0, 1)); \
    L1 = CO_FMA(YO(29), RCT(0, 0), L1); \
    g0a = CO_FMA(YO(23), RCT(0, 3), g0a); \
    L0 = CO_FMA(YO(31), RCT(0, 2), L0); \
    g0b = CO_FMA(YO(4), RCT(0, 5), g0b); \
    L1 = CO_FMA(YO(5), RCT(0, 4), L1); \
    g0a = CO_FMA(YO(6), RCT(0, 7), g0a); \
    L0 = CO_FMA(YO(7), RCT(0, 6), L0); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 108, 139); \
    TM_LD2(0, 1, 292, 89); \
    TM_LD2(0, 2, 328, 62); \
    TM_LD2(0, 3, 508, 167); \
    g0b = CO_FMA(YO(10), RCT(1, 1), g0b); \
    L1 = CO_FMA(YO(11), RCT(1, 0), L1); \
    g0a = CO_FMA(YO(13), RCT(1, 3), g0a); \
    L0 = CO_FMA(YO(12), RCT(1, 2), L0); \
    g0b = CO_FMA(YO(16), RCT(1, 5), g0b); \
    L1 = CO_FMA(YO(18), RCT(1, 4), L1); \
    g0a = CO_FMA(YO(11), RCT(1, 7), g0a); \
    L0 = CO_FMA(YO(17), RCT(1, 6), L0); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 52, 7); \
    TM_LD2(1, 1, 332, 108); \
    TM_LD2(1, 2, 376, 117); \
    TM_LD2(1, 3, 488, 84); \
    g0b = CO_FMA(YO(33), RCT(0, 7), g0b); \
    L1 = CO_FMA(YO(30), RCT(0, 6), L1); \
    const double2 s14 = RCS2(55); \
    g0a = CO_FMA(YO(41), s14.y, g0a); \
    L0 = CO_FMA(YO(40), s14.x, L0); \
    P1 = CO_MUL(YO(4), CO_ADD(g0a, g0b)); \
    g1a = CO_MUL(YO(11), RCT(0, 1)); \
    L1 = CO_FMA(YO(23), RCT(0, 0), L1); \
    g1a = CO_FMA(YO(13), RCT(0, 3), g1a); \
    L0 = CO_FMA(YO(16), RCT(0, 2), L0); \
    const double2 s15 = RCS2(40); \
    g1a = CO_FMA(YO(18), s15.y, g1a); \
    L1 = CO_FMA(YO(39), s15.x, L1); \
    P0 = CO_MUL(YO(10), g1a); \
    g2a = CO_MUL(YO(0), RCT(0, 5)); \
    L0 = CO_FMA(YO(14), RCT(0, 4), L0); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 0, 1); \
    TM_LD2(0, 1, 32, 0); \
    TM_LD2(0, 2, 88, 13); \
    TM_LD2(0, 3, 128, 77); \
    g2a = CO_FMA(YO(20), RCT(1, 5), g2a); \
    L1 = CO_FMA(YO(27), RCT(1, 4), L1); \
    P1 = CO_FMA(YO(8), g2a, P1); \
    P0 = CO_FMA(YO(4), RCT(1, 1), P0); \
    H0 = RCT(1, 0); \
    P1 = CO_FMA((YO(14) * YO(9)), RCT(1, 3), P1); \
    L0 = CO_FMA(YO(25), RCT(1, 2), L0); \
    P0 = CO_FMA((YO(13) * YO(11)), RCT(1, 7), P0); \
    L1 = CO_FMA(YO(18), RCT(1, 6), L1); \
    CO_WAIT_Y(1); \
    CO_GET(3, 1, 1, 1); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 164, 132); \
    TM_LD2(1, 1, 180, 151); \
    TM_LD2(1, 2, 232, 3); \
    TM_LD2(1, 3, 260, 20); \
    G0a = CO_FMA(YO(1), RCT(0, 2), G0a); \
    P0 = CO_FMA(YO(1), e1a, P0); \
    v0 = CO_ADD(G0a, G0b); \
    v1 = H0; \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    CO_PUT(9, v2, v0); \
    CO_PUT(10, v3, v1); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(0), RCT(0, 0)); \
    G0b = CO_MUL(YO(6), RCT(0, 4)); \
    L0 = CO_MUL(YO(1), RCT(0, 5)); \
    G0a = CO_FMA(YO(19), RCT(0, 6), G0a); \
    L1 = CO_MUL(YO(18), RCT(0, 7)); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 272, 33, 39); \
    TM_LD2(0, 2, 352, 83); \
    TM_LD2(0, 3, 424, 73); \
    G0b = CO_FMA(YO(29), RCT(1, 0), G0b); \
    L0 = CO_FMA(YO(28), RCT(1, 1), L0); \
    G0a = CO_FMA(YO(31), RCT(1, 2), G0a); \
    L1 = CO_FMA(YO(23), RCT(1, 3), L1); \
    G0b = CO_FMA(YO(5), RCT(1, 4), G0b); \
    L0 = CO_FMA(YO(4), RCT(1, 5), L0); \
    L1 = CO_FMA(YO(4), RCT(1, 5), L1); \
    G0a = CO_FMA(YO(5), RCT(1, 4), G0a); \
    G0b = CO_FMA(YO(7), RCT(1, 6), G0b); \
    L0 = CO_FMA(YO(6), RCT(1, 7), L0); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 4, 2); \
    TM_LD2(1, 1, 32, 0); \
    TM_LD2(1, 2, 52, 7); \
    TM_LD2(1, 3, 508, 167); \
    G0a = CO_FMA(YO(11), RCT(0, 0), G0a); \
    L1 = CO_FMA(YO(10), RCT(0, 1), L1); \
    G0b = CO_FMA(YO(12), RCT(0, 2), G0b); \
    L0 = CO_FMA(YO(13), RCT(0, 3), L0); \
    G0a = CO_FMA(YO(18), RCT(0, 4), G0a); \
    L1 = CO_FMA(YO(16), RCT(0, 5), L1); \
    G0b = CO_FMA(YO(17), RCT(0, 6), G0b); \
    L0 = CO_FMA(YO(11), RCT(0, 7), L0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 40, 10, 21); \
    TM_LD2(0, 2, 36, 18); \
    TM_LD2(0, 3, 320, 54); \
    G0a = CO_FMA(YO(30), RCT(1, 6), G0a); \
    L1 = CO_FMA(YO(33), RCT(1, 7), L1); \
    const double2 s16 = RCS2(56); \
    G0b = CO_FMA(YO(40), s16.x, G0b); \
    L0 = CO_FMA(YO(42), s16.y, L0); \
    L1 = CO_ADD(L1, RCT(1, 5)); \
    e2a = CO_MUL(YO(5), RCT(1, 1)); \
    L0 = CO_FMA(YO(0), RCT(1, 0), L0); \
    e2b = CO_MUL(YO(1), RCT(1, 2)); \
    H0 = RCT(1, 3); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 16, 161); \
    TM_LD2(1, 1, 324, 59); \
    TM_LD2(1, 2, 368, 112); \
    TM_LD2(1, 3, 440, 105); \
    e2a = CO_FMA(YO(7), RCT(0, 4), e2a); \
    L1 = CO_FMA(YO(5), RCT(0, 5), L1); \
    e2b = CO_FMA(YO(6), RCT(0, 0), e2b); \
    L0 = CO_FMA(YO(4), RCT(0, 1), L0); \
    L1 = CO_FMA(YO(4), RCT(0, 1), L1); \
    e2a = CO_FMA(YO(6), RCT(0, 0), e2a); \
    e2b = CO_FMA(YO(9), RCT(0, 3), e2b); \
    L0 = CO_FMA(YO(8), RCT(0, 2), L0); \
    e2a = CO_FMA(YO(11), RCT(0, 7), e2a); \
    L1 = CO_FMA(YO(15), RCT(0, 6), L1); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 24, 28, 148); \
    TM_LD2(0, 2, 20, 162); \
    TM_LD2(0, 3, 96, 34); \
    e2b = CO_FMA(YO(11), RCT(1, 3), e2b); \
    L0 = CO_FMA(YO(14), RCT(1, 2), L0); \
    e2a = CO_FMA((YO(10) * YO(8)), RCT(1, 5), e2a); \
    L1 = CO_FMA(YO(26), RCT(1, 4), L1); \
    e2b = CO_FMA(YO(25), RCT(1, 7), e2b); \
    L0 = CO_FMA(YO(21), RCT(1, 6), L0); \
    g0a = CO_MUL(YO(33), RCT(1, 1)); \
    L1 = CO_FMA(YO(30), RCT(1, 0), L1); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 160, 128); \
    TM_LD2(1, 1, 184, 149); \
    TM_LD2(1, 2, 192, 163); \
    TM_LD2(1, 3, 236, 14); \
    g0b = CO_MUL(YO(32), RCT(0, 5)); \
    L0 = CO_FMA(YO(30), RCT(0, 4), L0); \
    g0a = CO_FMA(YO(8), RCT(0, 1), g0a); \
    L1 = CO_FMA(YO(10), RCT(0, 0), L1); \
    g0b = CO_FMA(YO(34), RCT(0, 3), g0b); \
    L0 = CO_FMA(YO(31), RCT(0, 2), L0); \
    g0a = CO_FMA(YO(10), RCT(0, 7), g0a); \
    L1 = CO_FMA(YO(11), RCT(0, 6), L1); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 296, 44, 78); \
    TM_LD2(0, 2, 280, 38); \
    TM_LD2(0, 3, 360, 88); \
    g0b = CO_FMA(YO(28), RCT(1, 1), g0b); \
    L0 = CO_FMA(YO(29), RCT(1, 0), L0); \
    g0a = CO_FMA(YO(23), RCT(1, 3), g0a); \
    L1 = CO_FMA(YO(31), RCT(1, 2), L1); \
    g0b = CO_FMA(YO(35), RCT(1, 5), g0b); \
    L0 = CO_FMA(YO(30), RCT(1, 4), L0); \
    g0a = CO_FMA(YO(1), RCT(1, 7), g0a); \
    L1 = CO_FMA(YO(6), RCT(1, 6), L1); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 80, 22, 47); \
    TM_LD2(1, 2, 388, 123); \
    TM_LD2(1, 3, 500, 140); \
    g0b = CO_FMA(YO(13), RCT(0, 5), g0b); \
    L0 = CO_FMA(YO(12), RCT(0, 4), L0); \
    g0a = CO_FMA(YO(15), RCT(0, 1), g0a); \
    L1 = CO_FMA(YO(13), RCT(0, 0), L1); \
    g0b = CO_FMA(YO(18), RCT(0, 3), g0b); \
    L0 = CO_FMA(YO(19), RCT(0, 2), L0); \
    g0a = CO_FMA(YO(22), RCT(0, 7), g0a); \
    L1 = CO_FMA(YO(16), RCT(0, 6), L1); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 312, 48, 55); \
    TM_LD2(0, 2, 92, 93); \
    TM_LD2(0, 3, 372, 114); \
    g0b = CO_FMA(YO(11), RCT(1, 5), g0b); \
    L0 = CO_FMA(YO(28), RCT(1, 4), L0); \
    g0a = CO_FMA(YO(25), RCT(1, 7), g0a); \
    L1 = CO_FMA(YO(23), RCT(1, 6), L1); \
    const double2 s17 = RCS2(58); \
    g0b = CO_FMA(YO(41), s17.y, g0b); \
    L0 = CO_FMA(YO(40), s17.x, L0); \
    P1 = CO_MUL(YO(5), CO_ADD(g0a, g0b)); \
    g1a = CO_MUL(YO(8), RCT(1, 0)); \
    L1 = CO_FMA(YO(9), RCT(1, 1), L1); \
    g1a = CO_FMA(YO(13), RCT(1, 2), g1a); \
    L0 = CO_FMA(YO(17), RCT(1, 3), L0); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 400, 15, 127); \
    TM_LD2(1, 2, 48, 5); \
    TM_LD2(1, 3, 460, 135); \
    g1a = CO_FMA(YO(16), RCT(0, 4), g1a); \
    L1 = CO_FMA(YO(24), RCT(0, 5), L1); \
    P0 = CO_MUL(YO(6), g1a); \
    g2a = CO_MUL(YO(13), RCT(0, 0)); \
    L0 = CO_FMA(YO(11), RCT(0, 1), L0); \
    g2a = CO_FMA(YO(15), RCT(0, 2), g2a); \
    g2a = CO_FMA(YO(26), RCT(0, 6), g2a); \
    L1 = CO_FMA((YO(8) * YO(8)), RCT(0, 7), L1); \
    P1 = CO_FMA(YO(1), g2a, P1); \
    f2a = CO_MUL(YO(8), RCT(0, 3)); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 0, 1, 2); \
    TM_LD4(0, 2, 48, 5, 7); \
    P0 = CO_FMA(YO(5), RCT(1, 5), P0); \
    P1 = CO_FMA(YO(7), RCT(1, 1), P1); \
    L1 = CO_FMA(YO(4), RCT(1, 0), L1); \
    L0 = CO_FMA(YO(4), RCT(1, 0), L0); \
    P0 = CO_FMA(YO(7), RCT(1, 1), P0); \
    P1 = CO_FMA((YO(28) * YO(8)), RCT(1, 3), P1); \
    L1 = CO_FMA(YO(25), RCT(1, 2), L1); \
    P0 = CO_FMA(YO(29), RCT(1, 6), P0); \
    L0 = CO_FMA(YO(13), RCT(1, 7), L0); \
    const double2 s18 = RCS2(88); \
    L1 = CO_FMA(YO(46), s18.x, L1); \
    const double2 s19 = RCS2(89); \
    L0 = CO_FMA(YO(46), s19.x, L0); \
    CO_WAIT_Y(0); \
    CO_GET(0, 2, 0, 1); \
    TM_WAIT(0, 4); \
    TM_LD8(1, 0, 16, 161, 162, 28, 148); \
    G0a = CO_FMA(YO(2), RCT(0, 6), G0a); \
    P0 = CO_FMA(YO(2), CO_ADD(e2a, e2b), P0); \
    L0 = CO_FMA(YO(2), f2a, L0); \
    L1 = CO_FMA(YO(2), RCT(0, 1), L1); \
    L0 = CO_FMA(YO(2), RCT(0, 4), L0); \
    v0 = CO_ADD(G0a, G0b); \
    v1 = H0; \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    CO_PUT(2, v2, v0); \
    CO_PUT(3, v3, v1); \
    CO_ARRIVE_P(0); \
    G0a = CO_MUL(YO(0), RCT(0, 2)); \
    L0 = CO_MUL(YO(2), RCT(0, 3)); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 48, 5); \
    TM_LD2(0, 1, 96, 34); \
    TM_LD2(0, 2, 160, 128); \
    TM_LD2(0, 3, 184, 149); \
    G0b = CO_MUL(YO(30), RCT(1, 0)); \
    L1 = CO_MUL(YO(33), RCT(1, 1)); \
    G0a = CO_FMA(YO(30), RCT(1, 2), G0a); \
    L0 = CO_FMA(YO(32), RCT(1, 3), L0); \
    G0b = CO_FMA(YO(10), RCT(1, 4), G0b); \
    L1 = CO_FMA(YO(8), RCT(1, 5), L1); \
    G0a = CO_FMA(YO(31), RCT(1, 6), G0a); \
    L0 = CO_FMA(YO(34), RCT(1, 7), L0); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 232, 3, 14); \
    TM_LD2(1, 2, 192, 163); \
    TM_LD2(1, 3, 280, 38); \
    G0b = CO_FMA(YO(2), RCT(0, 0), G0b); \
    L1 = CO_ADD(L1, RCT(0, 1)); \
    G0a = CO_FMA(YO(11), RCT(0, 2), G0a); \
    L0 = CO_FMA(YO(10), RCT(0, 3), L0); \
    G0b = CO_FMA(YO(29), RCT(0, 4), G0b); \
    L1 = CO_FMA(YO(28), RCT(0, 5), L1); \
    G0a = CO_FMA(YO(31), RCT(0, 6), G0a); \
    L0 = CO_FMA(YO(23), RCT(0, 7), L0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 296, 44, 78); \
    TM_LD2(0, 2, 360, 88); \
    TM_LD2(0, 3, 388, 123); \
    G0b = CO_FMA(YO(30), RCT(1, 4), G0b); \
    L1 = CO_FMA(YO(35), RCT(1, 5), L1); \
    G0a = CO_FMA(YOS(0), RCT(1, 1), G0a); \
    G0b = CO_FMA(YO(6), RCT(1, 2), G0b); \
    L0 = CO_FMA(YO(1), RCT(1, 3), L0); \
    G0a = CO_FMA(YO(12), RCT(1, 6), G0a); \
    L1 = CO_FMA(YO(13), RCT(1, 7), L1); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 36, 18); \
    TM_LD2(1, 1, 64, 12); \
    TM_LD2(1, 2, 344, 68); \
    TM_LD2(1, 3, 500, 140); \
    G0b = CO_FMA(YO(13), RCT(0, 0), G0b); \
    L0 = CO_FMA(YO(15), RCT(0, 1), L0); \
    G0a = CO_FMA(YO(19), RCT(0, 2), G0a); \
    L1 = CO_FMA(YO(18), RCT(0, 3), L1); \
    G0b = CO_FMA(YO(16), RCT(0, 4), G0b); \
    L0 = CO_FMA(YO(22), RCT(0, 5), L0); \
    G0a = CO_FMA(YO(28), RCT(0, 6), G0a); \
    L1 = CO_FMA(YO(11), RCT(0, 7), L1); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 64, 12); \
    TM_LD2(0, 1, 232, 3); \
    TM_LD2(0, 2, 348, 71); \
    TM_LD2(0, 3, 476, 160); \
    G0b = CO_FMA(YO(23), RCT(1, 6), G0b); \
    L0 = CO_FMA(YO(25), RCT(1, 7), L0); \
    const double2 s20 = RCS2(57); \
    G0a = CO_FMA(YO(40), s20.x, G0a); \
    L1 = CO_FMA(YO(42), s20.y, L1); \
    const double2 s21 = RCS2(88); \
    G0b = CO_FMA(YO(46), s21.x, G0b); \
    const double2 s22 = RCS2(89); \
    G0a = CO_FMA(YO(46), s22.x, G0a); \
    g0a = CO_MUL(YO(7), RCT(1, 0)); \
    H0 = RCT(1, 1); \
    g0a = CO_FMA(YO(6), RCT(1, 2), g0a); \
    g0a = CO_FMA(YO(11), RCT(1, 5), g0a); \
    L0 = CO_FMA(YO(20), RCT(1, 4), L0); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 80, 22, 47); \
    TM_LD2(1, 2, 88, 13); \
    TM_LD2(1, 3, 236, 14); \
    g0a = CO_FMA(YO(17), RCT(0, 4), g0a); \
    L1 = CO_FMA(YO(15), RCT(0, 5), L1); \
    P0 = CO_MUL(YO(2), g0a); \
    P1 = CO_MUL(YO(30), RCT(0, 6)); \
    L0 = CO_FMA(YO(16), RCT(0, 7), L0); \
    CO_WAIT_Y(1); \
    CO_GET(3, 3, 1, 1); \
    L1 = CO_FMA(YO(3), RCT(0, 1), L1); \
    L0 = CO_FMA(YO(3), RCT(0, 2), L0); \
    v0 = CO_ADD(G0a, G0b); \
    v1 = H0; \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    CO_PUT(9, v2, v0); \
    CO_PUT(10, v3, v1); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(3), RCT(0, 1)); \
    L0 = CO_MUL(YO(2), RCT(0, 0)); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 40, 10); \
    TM_LD2(0, 1, 92, 93); \
    TM_LD2(0, 2, 148, 101); \
    TM_LD2(0, 3, 172, 134); \
    G0a = CO_FMA(YO(1), RCT(1, 7), G0a); \
    e4a = CO_MUL(YO(9), RCT(1, 1)); \
    L1 = CO_MUL(YO(8), RCT(1, 0)); \
    e4b = CO_MUL(YO(17), RCT(1, 3)); \
    L0 = CO_FMA(YO(13), RCT(1, 2), L0); \
    e4a = CO_FMA(YO(1), RCT(1, 5), e4a); \
    L1 = CO_FMA(YO(3), RCT(1, 4), L1); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 176, 144); \
    TM_LD2(1, 1, 204, 158); \
    TM_LD2(1, 2, 212, 9); \
    TM_LD2(1, 3, 240, 11); \
    e4b = CO_FMA(YO(24), RCT(0, 3), e4b); \
    L0 = CO_FMA(YO(16), RCT(0, 2), L0); \
    const double2 s23 = RCS2(9); \
    e4a = CO_FMA(YO(35), s23.y, e4a); \
    L1 = CO_FMA(YO(18), s23.x, L1); \
    L0 = CO_FMA(YO(2), RCT(0, 0), L0); \
    g0a = CO_MUL(YO(22), RCT(0, 4)); \
    L1 = CO_FMA(YO(21), RCT(0, 5), L1); \
    g0b = CO_MUL(YO(29), RCT(0, 6)); \
    L0 = CO_FMA(YO(28), RCT(0, 7), L0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 248, 16, 29); \
    TM_LD2(0, 2, 244, 92); \
    TM_LD2(0, 3, 356, 85); \
    g0a = CO_FMA(YO(31), RCT(1, 1), g0a); \
    L1 = CO_FMA(YO(23), RCT(1, 0), L1); \
    g0b = CO_FMA(YO(31), RCT(1, 2), g0b); \
    L0 = CO_FMA(YO(34), RCT(1, 3), L0); \
    g0a = CO_FMA(YO(2), RCT(1, 4), g0a); \
    L1 = CO_ADD(L1, RCT(1, 5)); \
    g0b = CO_FMA(YO(0), RCT(1, 7), g0b); \
    L0 = CO_FMA(YO(2), RCT(1, 6), L0); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 100, 36); \
    TM_LD2(1, 1, 132, 81); \
    TM_LD2(1, 2, 168, 133); \
    TM_LD2(1, 3, 484, 74); \
    g0a = CO_FMA(YO(16), RCT(0, 4), g0a); \
    L1 = CO_FMA(YO(22), RCT(0, 5), L1); \
    g0b = CO_FMA(YO(7), RCT(0, 1), g0b); \
    L0 = CO_FMA(YO(6), RCT(0, 0), L0); \
    L1 = CO_FMA(YO(6), RCT(0, 0), L1); \
    g0a = CO_FMA(YO(7), RCT(0, 1), g0a); \
    g0b = CO_FMA(YO(10), RCT(0, 2), g0b); \
    L0 = CO_FMA(YO(8), RCT(0, 3), L0); \
    g0a = CO_FMA(YO(18), RCT(0, 6), g0a); \
    L1 = CO_FMA(YO(16), RCT(0, 7), L1); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 256, 17, 20); \
    TM_LD2(0, 2, 40, 10); \
    TM_LD2(0, 3, 396, 156); \
    g0b = CO_FMA(YO(17), RCT(1, 6), g0b); \
    L0 = CO_FMA(YO(11), RCT(1, 7), L0); \
    const double2 s24 = RCS2(17); \
    g0a = CO_FMA(YO(32), s24.x, g0a); \
    L1 = CO_FMA(YO(31), s24.y, L1); \
    const double2 s25 = RCS2(28); \
    g0b = CO_FMA(YO(36), s25.y, g0b); \
    L0 = CO_FMA(YO(37), s25.x, L0); \
    const double2 s26 = RCS2(45); \
    g0a = CO_FMA(YO(39), s26.y, g0a); \
    L1 = CO_FMA(YO(38), s26.x, L1); \
    const double2 s27 = RCS2(52); \
    g0b = CO_FMA(YO(40), s27.x, g0b); \
    L0 = CO_FMA(YO(42), s27.y, L0); \
    const double2 s28 = RCS2(63); \
    g0a = CO_FMA(YO(41), s28.x, g0a); \
    L1 = CO_FMA(YO(39), s28.y, L1); \
    P1 = CO_MUL(YO(1), CO_ADD(g0a, g0b)); \
    g1a = CO_MUL(YO(10), RCT(1, 1)); \
    L0 = CO_FMA(YO(11), RCT(1, 0), L0); \
    g1b = CO_MUL(YO(18), RCT(1, 3)); \
    L1 = CO_FMA(YO(19), RCT(1, 2), L1); \
    g1a = CO_FMA(YO(28), RCT(1, 5), g1a); \
    L0 = CO_FMA(YO(29), RCT(1, 4), L0); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 100, 36); \
    TM_LD2(1, 1, 132, 81); \
    TM_LD2(1, 2, 236, 14); \
    TM_LD2(1, 3, 260, 20); \
    g1b = CO_FMA(YO(2), RCT(0, 0), g1b); \
    L1 = CO_FMA(YO(0), RCT(0, 1), L1); \
    g1a = CO_FMA(YO(3), RCT(0, 2), g1a); \
    g1b = CO_FMA(YO(34), RCT(0, 7), g1b); \
    L0 = CO_FMA(YO(31), RCT(0, 6), L0); \
    const double2 s29 = RCS2(5); \
    g1a = CO_FMA(YO(32), s29.y, g1a); \
    L1 = CO_FMA(YO(30), s29.x, L1); \
    const double2 s30 = RCS2(6); \
    g1b = CO_FMA(YO(33), s30.y, g1b); \
    L0 = CO_FMA(YO(30), s30.x, L0); \
    const double2 s31 = RCS2(59); \
    g1a = CO_FMA(YO(41), s31.y, g1a); \
    L1 = CO_FMA(YO(40), s31.x, L1); \
    P0 = CO_MUL(YO(7), CO_ADD(g1a, g1b)); \
    CO_WAIT_Y(0); \
    CO_GET(0, 4, 0, 1); \
    e4b = CO_FMA(YOS(0), RCT(0, 5), e4b); \
    P0 = CO_FMA(YO(4), CO_ADD(e4a, e4b), P0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 256, 17, 20); \
    TM_LD2(0, 2, 168, 133); \
    TM_LD2(0, 3, 248, 16); \
    L0 = CO_FMA(YO(4), RCT(1, 4), L0); \
    L1 = CO_FMA(YO(4), RCT(1, 7), L1); \
    v0 = G0a; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    CO_PUT(2, v1, v0); \
    CO_PUT(3, v2, 0.0); \
    CO_ARRIVE_P(0); \
    G0a = CO_MUL(YO(11), RCT(1, 0)); \
    L0 = CO_MUL(YO(10), RCT(1, 1)); \
    G0b = CO_MUL(YO(19), RCT(1, 2)); \
    L1 = CO_MUL(YO(18), RCT(1, 3)); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 36, 18); \
    TM_LD2(1, 1, 224, 113); \
    TM_LD2(1, 2, 396, 156); \
    TM_LD2(1, 3, 400, 15); \
    G0a = CO_FMA(YO(29), RCT(0, 4), G0a); \
    L0 = CO_FMA(YO(28), RCT(0, 5), L0); \
    G0b = CO_FMA(YOS(1), RCT(0, 6), G0b); \
    L1 = CO_FMA(YO(1), RCT(0, 7), L1); \
    G0a = CO_FMA(YO(0), RCT(0, 1), G0a); \
    L0 = CO_FMA(YO(2), RCT(0, 0), L0); \
    G0b = CO_FMA(YO(4), RCT(0, 3), G0b); \
    L1 = CO_FMA(YO(3), RCT(0, 2), L1); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 368, 112, 114); \
    TM_LD2(0, 2, 228, 115); \
    TM_LD2(0, 3, 448, 111); \
    G0a = CO_FMA(YO(31), RCT(1, 4), G0a); \
    L0 = CO_FMA(YO(34), RCT(1, 5), L0); \
    const double2 s32 = RCS2(5); \
    G0b = CO_FMA(YO(30), s32.x, G0b); \
    L1 = CO_FMA(YO(32), s32.y, L1); \
    const double2 s33 = RCS2(7); \
    G0a = CO_FMA(YO(30), s33.x, G0a); \
    L0 = CO_FMA(YO(35), s33.y, L0); \
    const double2 s34 = RCS2(59); \
    G0b = CO_FMA(YO(40), s34.x, G0b); \
    L1 = CO_FMA(YO(41), s34.y, L1); \
    e5a = CO_MUL(YO(4), RCT(1, 1)); \
    L0 = CO_FMA(YO(2), RCT(1, 0), L0); \
    P1 = CO_MUL((YO(4) * YOS(0)), RCT(1, 6)); \
    L1 = CO_ADD(L1, RCT(1, 7)); \
    CO_WAIT_Y(1); \
    CO_GET(3, 5, 1, 1); \
    P0 = CO_MUL(YO(5), e5a); \
    v0 = CO_ADD(G0a, G0b); \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    CO_PUT(8, v1, v0); \
    CO_PUT(9, v2, 0.0); \
    CO_ARRIVE_P(1); \
    g0a = CO_MUL(YO(3), RCT(1, 2)); \
    g0b = CO_MUL(YO(3), RCT(1, 2)); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 72, 66); \
    TM_LD2(1, 1, 156, 104); \
    TM_LD2(1, 2, 252, 29); \
    TM_LD2(1, 3, 316, 55); \
    g0a = CO_FMA(YO(1), RCT(0, 4), g0a); \
    g0b = CO_FMA(YO(4), RCT(0, 0), g0b); \
    g0a = CO_FMA(YO(1), RCT(0, 2), g0a); \
    g0b = CO_FMA(YO(1), RCT(0, 2), g0b); \
    g0a = CO_FMA(YO(2), RCT(0, 6), g0a); \
    L0 = CO_MUL(YO(15), RCT(0, 7)); \
    P0 = CO_MUL(YO(26), CO_ADD(g0a, g0b)); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 24, 28); \
    TM_LD2(0, 1, 80, 22); \
    TM_LD2(0, 2, 328, 62); \
    TM_LD2(0, 3, 376, 117); \
    g1a = CO_MUL(YO(21), RCT(1, 2)); \
    L1 = CO_MUL(YO(11), RCT(1, 3)); \
    g1a = CO_FMA(YO(10), RCT(1, 4), g1a); \
    g1a = CO_FMA(YO(15), RCT(1, 6), g1a); \
    const double2 s35 = RCS2(39); \
    g1a = CO_FMA(YO(36), s35.x, g1a); \
    L0 = CO_FMA((YO(13) * YO(10)), s35.y, L0); \
    P1 = CO_MUL(YO(1), g1a); \
    g2a = CO_MUL(YO(20), RCT(1, 0)); \
    L1 = CO_FMA(YO(2), RCT(1, 1), L1); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 44, 21); \
    TM_LD2(1, 1, 224, 113); \
    TM_LD2(1, 2, 264, 25); \
    TM_LD2(1, 3, 404, 127); \
    g2a = CO_FMA(YO(14), RCT(0, 4), g2a); \
    L0 = CO_FMA(YO(0), RCT(0, 5), L0); \
    g2a = CO_FMA(YO(27), RCT(0, 6), g2a); \
    L1 = CO_FMA(YO(20), RCT(0, 7), L1); \
    const double2 s36 = RCS2(24); \
    g2a = CO_FMA(YO(36), s36.x, g2a); \
    L0 = CO_FMA(YO(16), s36.y, L0); \
    P0 = CO_FMA(YO(3), g2a, P0); \
    g0a = CO_MUL(YO(10), RCT(0, 0)); \
    L1 = CO_FMA(YO(5), RCT(0, 1), L1); \
    g0a = CO_FMA(YO(9), RCT(0, 3), g0a); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 368, 112, 114); \
    TM_LD2(0, 2, 228, 115); \
    TM_LD2(0, 3, 316, 55); \
    g0a = CO_FMA(YO(25), RCT(1, 6), g0a); \
    L0 = CO_FMA(YO(28), RCT(1, 7), L0); \
    P1 = CO_FMA(YO(4), g0a, P1); \
    g1a = CO_MUL(YO(9), RCT(1, 1)); \
    L1 = CO_FMA(YO(4), RCT(1, 0), L1); \
    g1a = CO_FMA(YO(10), RCT(1, 4), g1a); \
    L0 = CO_FMA(YO(0), RCT(1, 5), L0); \
    P0 = CO_FMA(YO(2), g1a, P0); \
    g2a = CO_MUL(YO(8), RCT(1, 3)); \
    g2a = CO_FMA(YO(8), RCT(1, 3), g2a); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 200, 147); \
    TM_LD2(1, 1, 216, 24); \
    TM_LD2(1, 2, 444, 110); \
    TM_LD2(1, 3, 464, 145); \
    g2a = CO_FMA(YO(9), RCT(0, 5), g2a); \
    g2a = CO_FMA(YO(4), RCT(0, 7), g2a); \
    g2a = CO_FMA(YO(10), RCT(0, 1), g2a); \
    L1 = CO_FMA(YO(2), g2a, L1); \
    g0a = CO_MUL(YO(4), RCT(0, 3)); \
    g0a = CO_FMA(YO(4), RCT(0, 3), g0a); \
    L0 = CO_FMA(YO(8), g0a, L0); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 44, 21); \
    TM_LD2(0, 1, 80, 22); \
    TM_LD2(0, 2, 228, 115); \
    TM_LD2(0, 3, 252, 29); \
    P1 = CO_FMA(YO(34), RCT(1, 0), P1); \
    L1 = CO_FMA(YO(13), RCT(1, 1), L1); \
    P0 = CO_FMA(YO(10), RCT(1, 2), P0); \
    L0 = CO_FMA(YO(2), RCT(1, 3), L0); \
    P1 = CO_FMA((YO(25) * YO(13)), RCT(1, 4), P1); \
    L1 = CO_FMA(YO(18), RCT(1, 5), L1); \
    P0 = CO_FMA(YO(23), RCT(1, 6), P0); \
    L0 = CO_FMA(YO(13), RCT(1, 7), L0); \
    CO_WAIT_Y(0); \
    CO_GET(0, 6, 0, 1); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 24, 28); \
    TM_LD2(1, 1, 332, 108); \
    TM_LD2(1, 2, 380, 119); \
    TM_LD2(1, 3, 412, 63); \
    L1 = CO_FMA(YO(6), RCT(0, 2), L1); \
    L0 = CO_FMA(YO(6), RCT(0, 7), L0); \
    v0 = CO_ADD(P0, P1); \
    v1 = CO_ADD(L0, L1); \
    CO_PUT(2, v0, v1); \
    CO_ARRIVE_P(0); \
    G0a = CO_MUL(YO(4), RCT(0, 0)); \
    L0 = CO_MUL(YO(2), RCT(0, 1)); \
    G0a = CO_FMA(YO(6), RCT(0, 2), G0a); \
    L1 = CO_MUL(YO(4), RCT(0, 3)); \
    const double2 s37 = RCS2(13); \
    G0a = CO_FMA(YO(35), s37.x, G0a); \
    L0 = CO_FMA(YO(18), s37.y, L0); \
    g0a = CO_MUL(YO(26), RCT(0, 4)); \
    H0 = CO_MUL(YO(2), RCT(0, 5)); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 96, 34); \
    TM_LD2(0, 1, 216, 24); \
    TM_LD2(0, 2, 252, 29); \
    TM_LD2(0, 3, 264, 25); \
    g0a = CO_FMA(YO(27), RCT(1, 4), g0a); \
    L1 = CO_FMA(YO(20), RCT(1, 5), L1); \
    g0a = CO_FMA(YO(14), RCT(1, 6), g0a); \
    L0 = CO_FMA(YO(0), RCT(1, 7), L0); \
    P0 = CO_MUL(YO(1), g0a); \
    P1 = CO_MUL((YO(3) * YO(25)), RCT(1, 2)); \
    L1 = CO_FMA(YO(14), RCT(1, 3), L1); \
    CO_WAIT_Y(1); \
    CO_GET(3, 7, 1, 1); \
    v0 = G0a; \
    v1 = H0; \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    CO_PUT(9, v2, v0); \
    CO_PUT(10, v3, v1); \
    CO_ARRIVE_P(1); \
    e8a = CO_MUL(YO(5), RCT(1, 1)); \
    L0 = CO_MUL(YO(4), RCT(1, 0)); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 100, 36); \
    TM_LD2(1, 1, 104, 137); \
    TM_LD2(1, 2, 268, 32); \
    TM_LD2(1, 3, 272, 33); \
    e8a = CO_FMA(YO(2), RCT(0, 3), e8a); \
    L1 = RCT(0, 2); \
    e8a = CO_FMA(YO(6), RCT(0, 5), e8a); \
    L0 = CO_FMA(YO(1), RCT(0, 4), L0); \
    e8a = CO_FMA(YO(0), RCT(0, 7), e8a); \
    L1 = CO_FMA(YO(2), RCT(0, 6), L1); \
    g0a = CO_MUL(YO(4), RCT(0, 0)); \
    L0 = CO_FMA(YO(5), RCT(0, 1), L0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 336, 67, 99); \
    TM_LD2(0, 2, 108, 139); \
    TM_LD2(0, 3, 368, 112); \
    g0a = CO_FMA(YO(6), RCT(1, 0), g0a); \
    L1 = CO_FMA(YO(7), RCT(1, 1), L1); \
    g0a = CO_FMA(YO(2), RCT(1, 4), g0a); \
    L0 = CO_FMA(YO(0), RCT(1, 5), L0); \
    g0a = CO_FMA(YO(3), RCT(1, 6), g0a); \
    L1 = CO_FMA(YO(4), RCT(1, 7), L1); \
    P1 = CO_MUL(YO(11), g0a); \
    g1a = CO_MUL(YO(2), RCT(1, 2)); \
    L0 = CO_FMA(YO(13), RCT(1, 3), L0); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 220, 31); \
    TM_LD2(1, 1, 292, 89); \
    TM_LD2(1, 2, 368, 112); \
    TM_LD2(1, 3, 468, 146); \
    g1a = CO_FMA(YO(3), RCT(0, 4), g1a); \
    L1 = CO_FMA(YO(11), RCT(0, 5), L1); \
    P0 = CO_MUL(YO(23), g1a); \
    g2a = CO_MUL(YO(20), RCT(0, 0)); \
    L0 = CO_FMA(YO(3), RCT(0, 1), L0); \
    g2a = CO_FMA(YO(22), RCT(0, 2), g2a); \
    L1 = CO_FMA(YO(11), RCT(0, 3), L1); \
    P1 = CO_FMA(YO(1), g2a, P1); \
    f8a = CO_MUL(YO(2), RCT(0, 7)); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 96, 34, 36); \
    TM_LD2(0, 2, 220, 31); \
    TM_LD2(0, 3, 268, 32); \
    P0 = CO_FMA(YO(11), RCT(1, 1), P0); \
    L1 = CO_FMA(YO(2), RCT(1, 0), L1); \
    P1 = CO_FMA((YO(3) * YO(16)), RCT(1, 2), P1); \
    L0 = CO_FMA(YO(13), RCT(1, 3), L0); \
    P0 = CO_FMA((YO(4) * YO(26)), RCT(1, 4), P0); \
    P1 = CO_FMA(YO(31), RCT(1, 6), P1); \
    L1 = CO_FMA(YO(13), RCT(1, 7), L1); \
    CO_WAIT_Y(0); \
    CO_GET(0, 8, 0, 1); \
    P0 = CO_FMA(YO(8), e8a, P0); \
    L0 = CO_FMA(YO(8), f8a, L0); \
    v0 = CO_ADD(P0, P1); \
    v1 = CO_ADD(L0, L1); \
    CO_PUT(2, v0, v1); \
    CO_ARRIVE_P(0); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 156, 104); \
    TM_LD2(1, 1, 272, 33); \
    TM_LD2(1, 2, 312, 48); \
    TM_LD2(1, 3, 340, 99); \
    G0a = CO_MUL(YO(5), RCT(0, 1)); \
    L0 = CO_MUL(YO(4), RCT(0, 0)); \
    G0a = CO_FMA(YO(7), RCT(0, 3), G0a); \
    L1 = CO_MUL(YO(6), RCT(0, 2)); \
    G0a = CO_FMA(YO(2), RCT(0, 4), G0a); \
    L0 = CO_ADD(L0, RCT(0, 5)); \
    G0a = CO_FMA(YO(0), RCT(0, 7), G0a); \
    L1 = CO_FMA(YO(2), RCT(0, 6), L1); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 68, 45); \
    TM_LD2(0, 1, 108, 139); \
    TM_LD2(0, 2, 424, 73); \
    TM_LD2(0, 3, 484, 74); \
    G0a = CO_FMA(YO(4), RCT(1, 3), G0a); \
    L0 = CO_FMA(YO(3), RCT(1, 2), L0); \
    g0a = CO_MUL(YO(21), RCT(1, 0)); \
    L1 = CO_FMA(YO(8), RCT(1, 1), L1); \
    g0a = CO_FMA(YO(13), RCT(1, 4), g0a); \
    L0 = CO_FMA(YO(4), RCT(1, 5), L0); \
    g0a = CO_FMA(YO(22), RCT(1, 6), g0a); \
    H0 = RCT(1, 7); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 320, 54, 59); \
    TM_LD2(1, 2, 388, 123); \
    TM_LD2(1, 3, 488, 84); \
    g0a = CO_FMA(YO(17), RCT(0, 6), g0a); \
    L1 = CO_FMA(YO(6), RCT(0, 7), L1); \
    P0 = CO_MUL(YO(1), g0a); \
    g1a = CO_MUL(YO(13), RCT(0, 0)); \
    L0 = CO_FMA(YO(2), RCT(0, 1), L0); \
    g1a = CO_FMA(YO(23), RCT(0, 2), g1a); \
    H0 = CO_ADD(H0, RCT(0, 3)); \
    g1a = CO_FMA(YO(17), RCT(0, 4), g1a); \
    L1 = CO_FMA(YO(4), RCT(0, 5), L1); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 116, 70); \
    TM_LD2(0, 1, 344, 68); \
    TM_LD2(0, 2, 384, 121); \
    TM_LD2(0, 3, 428, 75); \
    g1a = CO_FMA(YO(18), RCT(1, 6), g1a); \
    L0 = CO_FMA(YO(13), RCT(1, 7), L0); \
    P1 = CO_MUL(YO(3), g1a); \
    g2a = CO_MUL(YO(15), RCT(1, 0)); \
    L1 = CO_FMA(YO(2), RCT(1, 1), L1); \
    g2a = CO_FMA(YO(14), RCT(1, 2), g2a); \
    L0 = CO_FMA(YO(2), RCT(1, 3), L0); \
    g2a = CO_FMA(YO(28), RCT(1, 4), g2a); \
    L1 = CO_FMA(YO(5), RCT(1, 5), L1); \
    P0 = CO_FMA(YO(4), g2a, P0); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 56, 52); \
    TM_LD2(1, 1, 276, 39); \
    TM_LD2(1, 2, 280, 38); \
    TM_LD2(1, 3, 452, 125); \
    g0a = CO_MUL(YO(17), RCT(0, 0)); \
    L0 = CO_FMA(YO(0), RCT(0, 1), L0); \
    g0a = CO_FMA(YO(28), RCT(0, 4), g0a); \
    L1 = CO_FMA(YO(0), RCT(0, 5), L1); \
    P1 = CO_FMA(YO(2), g0a, P1); \
    P0 = CO_FMA((YO(5) * YO(20)), RCT(0, 2), P0); \
    L0 = CO_FMA(YO(2), RCT(0, 3), L0); \
    P1 = CO_FMA(YO(17), RCT(0, 6), P1); \
    L1 = CO_FMA(YO(2), RCT(0, 7), L1); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 68, 45); \
    TM_LD2(0, 1, 284, 79); \
    TM_LD2(0, 2, 312, 48); \
    TM_LD2(0, 3, 504, 154); \
    P0 = CO_FMA(YO(28), RCT(1, 6), P0); \
    L0 = CO_FMA(YO(2), RCT(1, 7), L0); \
    const double2 s38 = RCS2(11); \
    P1 = CO_FMA(YO(35), s38.x, P1); \
    L1 = CO_FMA(YO(13), s38.y, L1); \
    CO_WAIT_Y(1); \
    CO_GET(3, 9, 1, 1); \
    v0 = G0a; \
    v1 = H0; \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    g0a = CO_MUL(YO(2), RCT(1, 0)); \
    L0 = RCT(1, 1); \
    g0a = CO_FMA(YO(4), RCT(1, 3), g0a); \
    L0 = CO_FMA(YO(3), RCT(1, 2), L0); \
    g0a = CO_FMA(YO(5), RCT(1, 5), g0a); \
    L0 = CO_FMA(YO(4), RCT(1, 4), L0); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 280, 38, 79); \
    TM_LD2(1, 2, 56, 52); \
    TM_LD2(1, 3, 276, 39); \
    g0a = CO_FMA(YO(19), RCT(0, 2), g0a); \
    L0 = CO_FMA(YO(18), RCT(0, 3), L0); \
    g0a = CO_FMA(YO(31), RCT(0, 6), g0a); \
    L0 = CO_FMA(YO(34), RCT(0, 7), L0); \
    P0 = CO_MUL(YO(13), g0a); \
    v4 = P0; \
    v5 = L0; \
    CO_PUT(11, v2, v0); \
    CO_PUT(12, v3, v1); \
    CO_PUT(13, v4, v5); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(2), RCT(0, 1)); \
    L0 = CO_MUL(YO(3), RCT(0, 0)); \
    G0a = CO_FMA(YO(4), RCT(0, 5), G0a); \
    L1 = CO_MUL(YO(1), RCT(0, 4)); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 304, 46, 51); \
    TM_LD2(0, 2, 104, 137); \
    TM_LD2(0, 3, 504, 154); \
    G1a = RCT(1, 5); \
    L0 = CO_FMA(YO(2), RCT(1, 4), L0); \
    G1b = CO_MUL(YO(3), RCT(1, 6)); \
    L1 = CO_FMA(YO(4), RCT(1, 7), L1); \
    G1a = CO_FMA(YO(4), RCT(1, 0), G1a); \
    L0 = CO_FMA(YO(5), RCT(1, 1), L0); \
    G1b = CO_FMA(YO(18), RCT(1, 3), G1b); \
    L1 = CO_FMA(YO(19), RCT(1, 2), L1); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 288, 42, 89); \
    TM_LD2(1, 2, 112, 43); \
    TM_LD2(1, 3, 408, 50); \
    G1a = CO_FMA(YO(34), RCT(0, 7), G1a); \
    L0 = CO_FMA(YO(31), RCT(0, 6), L0); \
    const double2 s39 = RCS2(3); \
    G1b = CO_FMA(YO(32), s39.y, G1b); \
    L1 = CO_FMA(YO(30), s39.x, L1); \
    g0a = CO_MUL(YO(23), RCT(0, 4)); \
    g0b = CO_MUL(YO(16), RCT(0, 1)); \
    L0 = CO_FMA(YO(14), RCT(0, 0), L0); \
    g0a = CO_FMA(YO(18), RCT(0, 3), g0a); \
    L1 = CO_FMA(YO(13), RCT(0, 2), L1); \
    L0 = CO_FMA(YO(13), RCT(0, 2), L0); \
    g0b = CO_FMA(YO(18), RCT(0, 3), g0b); \
    const double2 s40 = RCS2(14); \
    g0a = CO_FMA(YO(35), s40.x, g0a); \
    L1 = CO_FMA(YO(28), s40.y, L1); \
    const double2 s41 = RCS2(25); \
    g0b = CO_FMA(YO(36), s41.y, g0b); \
    L0 = CO_FMA(YO(21), s41.x, L0); \
    const double2 s42 = RCS2(48); \
    g0a = CO_FMA(YO(39), s42.x, g0a); \
    L1 = CO_FMA(YO(16), s42.y, L1); \
    const double2 s43 = RCS2(84); \
    g0b = CO_FMA(YO(46), s43.x, g0b); \
    const double2 s44 = RCS2(101); \
    g0a = CO_FMA(YO(47), s44.x, g0a); \
    L0 = CO_FMA(YO(39), s44.y, L0); \
    P0 = CO_MUL(YO(2), CO_ADD(g0a, g0b)); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 84, 47); \
    TM_LD2(0, 1, 136, 53); \
    TM_LD2(0, 2, 200, 147); \
    TM_LD2(0, 3, 488, 84); \
    g1a = CO_MUL(YO(15), RCT(1, 5)); \
    L1 = CO_FMA(YO(2), RCT(1, 4), L1); \
    g1a = CO_FMA(YO(14), RCT(1, 1), g1a); \
    L0 = CO_FMA(YO(2), RCT(1, 0), L0); \
    g1a = CO_FMA(YO(16), RCT(1, 7), g1a); \
    L1 = CO_FMA(YO(13), RCT(1, 6), L1); \
    L0 = CO_FMA(YO(13), RCT(1, 6), L0); \
    g1a = CO_FMA(YO(16), RCT(1, 7), g1a); \
    P1 = CO_MUL(YO(0), g1a); \
    g2a = CO_MUL(YO(16), RCT(1, 2)); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 296, 44); \
    TM_LD2(1, 1, 444, 110); \
    TM_LD2(1, 2, 460, 135); \
    TM_LD2(1, 3, 464, 145); \
    g2a = CO_FMA(YO(18), RCT(0, 6), g2a); \
    H0 = RCT(0, 7); \
    const double2 s45 = RCS2(26); \
    g2a = CO_FMA(YO(36), s45.x, g2a); \
    L1 = CO_FMA(YO(26), s45.y, L1); \
    P0 = CO_FMA(YO(3), g2a, P0); \
    g0a = CO_MUL(YO(17), RCT(0, 1)); \
    L0 = CO_FMA(YO(6), RCT(0, 0), L0); \
    const double2 s46 = RCS2(88); \
    g0a = CO_FMA(YO(46), s46.x, g0a); \
    const double2 s47 = RCS2(90); \
    g0a = CO_FMA(YO(46), s47.x, g0a); \
    P1 = CO_FMA(YO(4), g0a, P1); \
    P0 = CO_FMA(YO(19), RCT(0, 3), P0); \
    L1 = CO_FMA(YO(13), RCT(0, 2), L1); \
    L0 = CO_FMA(YO(13), RCT(0, 2), L0); \
    P1 = CO_FMA(YO(19), RCT(0, 3), P1); \
    P0 = CO_FMA(YO(34), RCT(0, 4), P0); \
    L1 = CO_FMA(YO(8), RCT(0, 5), L1); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 104, 137); \
    TM_LD2(0, 1, 292, 89); \
    TM_LD2(0, 2, 468, 146); \
    TM_LD2(0, 3, 472, 159); \
    P1 = CO_FMA((YO(5) * YO(15)), RCT(1, 1), P1); \
    L0 = CO_FMA(YO(4), RCT(1, 0), L0); \
    P0 = CO_FMA((YO(8) * YO(18)), RCT(1, 3), P0); \
    L1 = CO_FMA(YO(25), RCT(1, 2), L1); \
    P1 = CO_FMA(YO(29), RCT(1, 4), P1); \
    L0 = CO_FMA(YO(4), RCT(1, 5), L0); \
    P0 = CO_FMA(YO(23), RCT(1, 6), P0); \
    L1 = CO_FMA(YO(8), RCT(1, 7), L1); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 288, 42); \
    TM_LD2(1, 1, 304, 46); \
    TM_LD2(1, 2, 324, 59); \
    TM_LD2(1, 3, 416, 65); \
    P1 = CO_FMA(YO(31), RCT(0, 4), P1); \
    P0 = CO_FMA(YO(30), RCT(0, 6), P0); \
    L0 = CO_FMA(YO(28), RCT(0, 7), L0); \
    const double2 s48 = RCS2(11); \
    P1 = CO_FMA(YO(35), s48.x, P1); \
    H0 = CO_ADD(H0, s48.y); \
    const double2 s49 = RCS2(47); \
    P0 = CO_FMA(YO(39), s49.y, P0); \
    L1 = CO_FMA(YO(22), s49.x, L1); \
    const double2 s50 = RCS2(64); \
    P1 = CO_FMA(YO(42), s50.x, P1); \
    L0 = CO_FMA(YO(16), s50.y, L0); \
    const double2 s51 = RCS2(74); \
    P0 = CO_FMA(YO(43), s51.y, P0); \
    L1 = CO_FMA(YO(37), s51.x, L1); \
    CO_WAIT_Y(0); \
    CO_GET(0, 10, 0, 1); \
    L0 = CO_FMA(YO(10), RCT(0, 1), L0); \
    L1 = CO_FMA(YO(10), RCT(0, 3), L1); \
    L0 = CO_FMA(YO(10), RCT(0, 5), L0); \
    v0 = G0a; \
    v1 = CO_ADD(G1a, G1b); \
    v2 = H0; \
    v3 = CO_ADD(P0, P1); \
    v4 = CO_ADD(L0, L1); \
    CO_PUT(2, v3, v0); \
    CO_PUT(3, v1, v4); \
    CO_PUT(4, v2, 0.0); \
    CO_ARRIVE_P(0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 328, 62, 108); \
    TM_LD2(0, 2, 412, 63); \
    TM_LD2(0, 3, 480, 57); \
    G0a = CO_MUL(YO(2), RCT(1, 0)); \
    L0 = CO_MUL(YO(0), RCT(1, 1)); \
    e11a = CO_MUL(YO(2), RCT(1, 5)); \
    L1 = CO_MUL(YO(4), RCT(1, 4)); \
    g0a = CO_MUL(YO(16), RCT(1, 3)); \
    H0 = RCT(1, 2); \
    g0a = CO_FMA((YO(21) * YOS(2)), RCT(1, 7), g0a); \
    L0 = CO_FMA(YO(14), RCT(1, 6), L0); \
    L1 = CO_FMA(YO(14), RCT(1, 6), L1); \
    g0a = CO_FMA((YO(21) * YOS(2)), RCT(1, 7), g0a); \
    P1 = CO_MUL(YO(2), g0a); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 112, 43); \
    TM_LD2(1, 1, 296, 44); \
    TM_LD2(1, 2, 316, 55); \
    TM_LD2(1, 3, 320, 54); \
    g1a = CO_MUL(YO(8), RCT(0, 1)); \
    L0 = CO_FMA(YO(3), RCT(0, 0), L0); \
    g1a = CO_FMA(YO(9), RCT(0, 5), g1a); \
    L1 = CO_FMA(YO(1), RCT(0, 4), L1); \
    P0 = CO_MUL(YO(0), g1a); \
    P1 = CO_FMA((YO(3) * YO(25)), RCT(0, 2), P1); \
    L0 = CO_FMA(YO(9), RCT(0, 3), L0); \
    P0 = CO_FMA(YO(15), RCT(0, 6), P0); \
    L1 = CO_ADD(L1, RCT(0, 7)); \
    CO_WAIT_Y(1); \
    CO_GET(3, 11, 1, 1); \
    CO_GET(4, 12, 0, 1); \
    P0 = CO_FMA(YO(11), e11a, P0); \
    v0 = G0a; \
    v1 = H0; \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    CO_PUT(8, v2, v0); \
    CO_PUT(9, v3, v1); \
    CO_ARRIVE_P(1); \
    G0a = RCT(0, 7); \
    L0 = RCT(0, 6); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 124, 87); \
    TM_LD2(0, 1, 304, 46); \
    TM_LD2(0, 2, 348, 71); \
    TM_LD2(0, 3, 448, 111); \
    e13a = CO_MUL(YO(2), RCT(1, 0)); \
    L1 = CO_MUL(YO(0), RCT(1, 1)); \
    e13a = CO_FMA(YO(4), RCT(1, 2), e13a); \
    L0 = CO_FMA(YO(5), RCT(1, 3), L0); \
    g0a = CO_MUL((YO(8) * YO(4)), RCT(1, 5)); \
    L1 = CO_FMA(YO(1), RCT(1, 4), L1); \
    g0a = CO_FMA(YO(11), RCT(1, 7), g0a); \
    L0 = CO_FMA(YO(4), RCT(1, 6), L0); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 360, 88, 91); \
    TM_LD2(1, 2, 244, 92); \
    TM_LD2(1, 3, 436, 95); \
    g0a = CO_FMA(YO(17), RCT(0, 4), g0a); \
    L1 = CO_FMA(YO(5), RCT(0, 5), L1); \
    g0a = CO_FMA(YO(26), RCT(0, 6), g0a); \
    L0 = CO_FMA(YO(8), RCT(0, 7), L0); \
    P1 = CO_MUL(YO(2), g0a); \
    CO_WAIT_Y(0); \
    CO_GET(0, 13, 1, 1); \
    P0 = CO_MUL(YO(13), e13a); \
    v0 = G0a; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    G0a = CO_MUL(YO(13), RCT(0, 2)); \
    L0 = CO_MUL(YO(2), RCT(0, 3)); \
    g0a = CO_MUL(YO(0), RCT(0, 1)); \
    L1 = CO_MUL(YO(2), RCT(0, 0)); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 352, 83, 85); \
    TM_LD2(0, 2, 120, 82); \
    TM_LD2(0, 3, 292, 89); \
    g0b = CO_MUL(YO(6), RCT(1, 5)); \
    L0 = CO_FMA(YO(1), RCT(1, 4), L0); \
    g0a = CO_FMA(YO(5), RCT(1, 1), g0a); \
    L1 = CO_FMA(YO(4), RCT(1, 0), L1); \
    g0b = CO_FMA(YO(18), RCT(1, 3), g0b); \
    L0 = CO_FMA(YO(16), RCT(1, 2), L0); \
    L1 = CO_FMA(YO(16), RCT(1, 2), L1); \
    g0a = CO_FMA(YO(18), RCT(1, 3), g0a); \
    g0b = CO_FMA(YO(2), RCT(1, 7), g0b); \
    L0 = CO_ADD(L0, RCT(1, 6)); \
    P0 = CO_MUL(YO(22), CO_ADD(g0a, g0b)); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 76, 90); \
    TM_LD2(1, 1, 92, 93); \
    TM_LD2(1, 2, 408, 50); \
    TM_LD2(1, 3, 420, 96); \
    g1a = CO_MUL(YO(2), RCT(0, 4)); \
    L1 = CO_FMA(YO(0), RCT(0, 5), L1); \
    g1a = CO_FMA(YO(3), RCT(0, 0), g1a); \
    L0 = CO_FMA(YO(4), RCT(0, 1), L0); \
    g1a = CO_FMA(YO(1), RCT(0, 2), g1a); \
    L1 = CO_FMA(YO(6), RCT(0, 3), L1); \
    P1 = CO_MUL(YO(18), g1a); \
    const double2 s52 = RCS2(83); \
    g2a = CO_MUL(YO(2), s52.x); \
    const double2 s53 = RCS2(88); \
    g2a = CO_FMA(YO(4), s53.x, g2a); \
    P0 = CO_FMA(YO(46), g2a, P0); \
    g0a = CO_MUL(YO(10), RCT(0, 7)); \
    L0 = CO_FMA(YO(3), RCT(0, 6), L0); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 116, 70); \
    TM_LD2(0, 1, 348, 71); \
    TM_LD2(0, 2, 432, 86); \
    TM_LD2(0, 3, 476, 160); \
    g0a = CO_FMA(YOS(3), RCT(1, 4), g0a); \
    L1 = CO_FMA(YO(0), RCT(1, 5), L1); \
    P1 = CO_FMA(YO(13), g0a, P1); \
    P0 = CO_FMA((YO(2) * YO(23)), RCT(1, 1), P0); \
    L0 = CO_FMA(YO(3), RCT(1, 0), L0); \
    P1 = CO_FMA((YO(4) * YO(24)), RCT(1, 3), P1); \
    L1 = CO_FMA(YO(6), RCT(1, 2), L1); \
    P0 = CO_FMA((YO(0) * YO(21)), RCT(1, 7), P0); \
    L0 = CO_ADD(L0, RCT(1, 6)); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 424, 73, 75); \
    TM_LD2(1, 2, 84, 47); \
    TM_LD2(1, 3, 484, 74); \
    P1 = CO_FMA(YO(18), RCT(0, 4), P1); \
    L1 = CO_FMA(YO(2), RCT(0, 5), L1); \
    P0 = CO_FMA(YO(30), RCT(0, 6), P0); \
    L0 = CO_FMA(YO(5), RCT(0, 7), L0); \
    const double2 s54 = RCS2(76); \
    P1 = CO_FMA(YO(45), s54.x, P1); \
    L1 = CO_FMA(YO(36), s54.y, L1); \
    const double2 s55 = RCS2(92); \
    P0 = CO_FMA(YO(48), s55.x, P0); \
    L0 = CO_FMA(YO(39), s55.y, L0); \
    v3 = G0a; \
    v4 = CO_ADD(P0, P1); \
    v5 = CO_ADD(L0, L1); \
    CO_PUT(2, v1, v0); \
    CO_PUT(3, v2, v4); \
    CO_PUT(4, v3, v5); \
    CO_ARRIVE_P(0); \
    G0a = CO_MUL(YO(5), RCT(0, 3)); \
    L0 = CO_MUL(YO(2), RCT(0, 2)); \
    g0a = CO_MUL(YO(0), RCT(0, 1)); \
    L1 = CO_MUL(YO(2), RCT(0, 0)); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 120, 82); \
    TM_LD2(0, 1, 352, 83); \
    TM_LD2(0, 2, 456, 131); \
    TM_LD2(0, 3, 496, 126); \
    g0a = CO_FMA(YO(4), RCT(1, 1), g0a); \
    L0 = CO_FMA(YO(3), RCT(1, 0), L0); \
    g0a = CO_FMA(YO(2), RCT(1, 3), g0a); \
    L1 = CO_ADD(L1, RCT(1, 2)); \
    g0a = CO_FMA(YO(6), RCT(1, 7), g0a); \
    L0 = CO_FMA(YO(1), RCT(1, 6), L0); \
    P0 = CO_MUL(YO(11), g0a); \
    P1 = CO_MUL((YO(13) * YO(6)), RCT(1, 4)); \
    L1 = CO_FMA(YO(4), RCT(1, 5), L1); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 128, 77); \
    TM_LD2(1, 1, 356, 85); \
    TM_LD2(1, 2, 364, 91); \
    TM_LD2(1, 3, 432, 86); \
    P0 = CO_FMA((YO(2) * YO(29)), RCT(0, 4), P0); \
    L0 = CO_FMA(YO(0), RCT(0, 5), L0); \
    P1 = CO_FMA(YO(28), RCT(0, 7), P1); \
    L1 = CO_ADD(L1, RCT(0, 6)); \
    CO_WAIT_Y(1); \
    CO_GET(3, 14, 0, 1); \
    v0 = G0a; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    G0a = CO_MUL(YO(0), RCT(0, 1)); \
    L0 = CO_MUL(YO(2), RCT(0, 0)); \
    G0a = CO_FMA(YO(4), RCT(0, 3), G0a); \
    L1 = CO_MUL(YO(3), RCT(0, 2)); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 132, 81); \
    TM_LD2(0, 1, 284, 79); \
    TM_LD2(0, 2, 300, 78); \
    TM_LD2(0, 3, 308, 51); \
    G0a = CO_FMA(YO(6), RCT(1, 3), G0a); \
    L0 = CO_FMA(YO(1), RCT(1, 2), L0); \
    G0a = CO_FMA(YOS(4), RCT(1, 4), G0a); \
    L1 = CO_FMA(YO(22), RCT(1, 5), L1); \
    G0a = CO_FMA(YO(2), RCT(1, 7), G0a); \
    L0 = CO_ADD(L0, RCT(1, 6)); \
    g0a = CO_MUL(YO(3), RCT(1, 0)); \
    L1 = CO_FMA(YO(4), RCT(1, 1), L1); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 128, 77); \
    TM_LD2(1, 1, 140, 80); \
    TM_LD2(1, 2, 444, 110); \
    TM_LD2(1, 3, 488, 84); \
    g0a = CO_FMA(YO(6), RCT(0, 0), g0a); \
    L0 = CO_FMA(YO(7), RCT(0, 1), L0); \
    g0a = CO_FMA(YO(13), RCT(0, 2), g0a); \
    L1 = CO_FMA(YO(12), RCT(0, 3), L1); \
    g0a = CO_FMA(YO(4), RCT(0, 4), g0a); \
    L0 = CO_FMA(YO(5), RCT(0, 5), L0); \
    P0 = CO_MUL(YO(19), g0a); \
    g1a = CO_MUL(YOS(3), RCT(0, 6)); \
    L1 = CO_FMA(YO(2), RCT(0, 7), L1); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 132, 81); \
    TM_LD2(0, 1, 140, 80); \
    TM_LD2(0, 2, 284, 79); \
    TM_LD2(0, 3, 300, 78); \
    g1a = CO_FMA(YO(25), RCT(1, 4), g1a); \
    L0 = CO_FMA(YO(8), RCT(1, 5), L0); \
    g1a = CO_FMA(YO(11), RCT(1, 7), g1a); \
    L1 = CO_FMA(YO(3), RCT(1, 6), L1); \
    P1 = CO_MUL(YO(13), g1a); \
    P0 = CO_FMA(YO(19), RCT(1, 2), P0); \
    L0 = CO_FMA(YO(2), RCT(1, 3), L0); \
    const double2 s56 = RCS2(82); \
    P1 = CO_FMA(YO(46), s56.x, P1); \
    const double2 s57 = RCS2(83); \
    P0 = CO_FMA((YO(2) * YO(46)), s57.x, P0); \
    v3 = G0a; \
    v4 = CO_ADD(P0, P1); \
    v5 = CO_ADD(L0, L1); \
    CO_PUT(10, v1, v0); \
    CO_PUT(11, v2, v4); \
    CO_PUT(12, v3, v5); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(4), RCT(1, 1)); \
    L0 = CO_MUL(YO(3), RCT(1, 0)); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 376, 117, 119); \
    TM_LD2(1, 2, 72, 66); \
    TM_LD2(1, 3, 136, 53); \
    G0a = CO_FMA(YO(7), RCT(0, 1), G0a); \
    L1 = CO_MUL(YO(6), RCT(0, 0)); \
    G0a = CO_FMA(YO(2), RCT(0, 3), G0a); \
    L0 = CO_ADD(L0, RCT(0, 2)); \
    G0a = CO_FMA(YO(12), RCT(0, 5), G0a); \
    L1 = CO_FMA(YO(13), RCT(0, 4), L1); \
    G0a = CO_FMA(YO(5), RCT(0, 7), G0a); \
    L0 = CO_FMA(YO(4), RCT(0, 6), L0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 144, 97, 101); \
    TM_LD2(0, 2, 336, 67); \
    TM_LD2(0, 3, 344, 68); \
    P0 = CO_MUL((YO(13) * YOS(3)), RCT(1, 6)); \
    L1 = CO_ADD(L1, RCT(1, 7)); \
    CO_WAIT_Y(0); \
    CO_GET(0, 15, 1, 1); \
    CO_GET(1, 16, 0, 1); \
    v0 = G0a; \
    v1 = P0; \
    v2 = CO_ADD(L0, L1); \
    g0a = CO_MUL(YO(3), RCT(1, 0)); \
    L0 = CO_MUL(YO(8), RCT(1, 1)); \
    g0a = CO_FMA(YO(1), RCT(1, 2), g0a); \
    L0 = CO_FMA(YO(9), RCT(1, 3), L0); \
    P0 = CO_MUL(YO(27), g0a); \
    g1a = CO_MUL(YO(8), RCT(1, 5)); \
    L0 = CO_FMA(YO(3), RCT(1, 4), L0); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 152, 98, 104); \
    TM_LD4(1, 2, 416, 65, 96); \
    g1a = CO_FMA(YO(11), RCT(0, 7), g1a); \
    L0 = CO_FMA(YO(5), RCT(0, 6), L0); \
    P0 = CO_FMA(YO(2), g1a, P0); \
    P0 = CO_FMA((YO(10) * YO(3)), RCT(0, 5), P0); \
    L0 = CO_FMA(YO(1), RCT(0, 4), L0); \
    v3 = P0; \
    v4 = L0; \
    g0a = CO_MUL(YO(2), RCT(0, 0)); \
    L0 = CO_MUL(YO(0), RCT(0, 1)); \
    g0a = CO_FMA(YO(1), RCT(0, 2), g0a); \
    L1 = CO_MUL(YO(6), RCT(0, 3)); \
    P0 = CO_MUL(YO(22), g0a); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 144, 97, 101); \
    TM_LD2(0, 2, 152, 98); \
    TM_LD2(0, 3, 440, 105); \
    g1a = CO_MUL(YO(2), RCT(1, 5)); \
    const double2 s58 = RCS2(67); \
    g1a = CO_FMA(YO(22), s58.y, g1a); \
    L0 = CO_FMA(YO(2), g1a, L0); \
    P1 = CO_MUL(YO(22), RCT(1, 0)); \
    L1 = CO_FMA(YO(2), RCT(1, 1), L1); \
    P0 = CO_FMA((YO(11) * YO(8)), RCT(1, 3), P0); \
    L0 = CO_FMA(YO(1), RCT(1, 2), L0); \
    P1 = CO_FMA((YO(14) * YOS(5)), RCT(1, 4), P1); \
    P0 = CO_FMA(YO(16), RCT(1, 6), P0); \
    L1 = CO_FMA(YO(0), RCT(1, 7), L1); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 360, 88, 91); \
    TM_LD2(1, 2, 124, 87); \
    TM_LD2(1, 3, 244, 92); \
    P1 = CO_FMA((YO(2) * YO(25)), RCT(0, 7), P1); \
    L0 = CO_FMA(YO(4), RCT(0, 6), L0); \
    const double2 s59 = RCS2(35); \
    P0 = CO_FMA(YO(38), s59.y, P0); \
    L1 = CO_FMA(YO(13), s59.x, L1); \
    const double2 s60 = RCS2(67); \
    P1 = CO_FMA(YO(43), s60.x, P1); \
    v5 = CO_ADD(P0, P1); \
    v6 = CO_ADD(L0, L1); \
    CO_PUT(3, v1, v0); \
    CO_PUT(4, v2, v3); \
    CO_PUT(5, v4, v5); \
    CO_PUT(6, v6, 0.0); \
    CO_ARRIVE_P(0); \
    G0a = CO_MUL(YO(0), RCT(0, 1)); \
    L0 = CO_MUL(YO(2), RCT(0, 0)); \
    G0a = CO_FMA(YO(6), RCT(0, 3), G0a); \
    L1 = CO_MUL(YO(1), RCT(0, 2)); \
    G0a = CO_FMA(YO(2), RCT(0, 5), G0a); \
    L0 = CO_ADD(L0, RCT(0, 4)); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 340, 99); \
    TM_LD2(0, 1, 364, 91); \
    TM_LD2(0, 2, 436, 95); \
    TM_LD2(0, 3, 492, 100); \
    g0a = CO_MUL(YO(16), RCT(1, 4)); \
    L1 = CO_FMA(YO(0), RCT(1, 5), L1); \
    const double2 s61 = RCS2(70); \
    g0a = CO_FMA(YO(43), s61.x, g0a); \
    L0 = CO_FMA(YO(16), s61.y, L0); \
    const double2 s62 = RCS2(94); \
    g0a = CO_FMA(YO(48), s62.x, g0a); \
    const double2 s63 = RCS2(102); \
    g0a = CO_FMA(YO(47), s63.x, g0a); \
    P0 = CO_MUL(YO(2), g0a); \
    g1a = CO_MUL(YO(1), RCT(1, 6)); \
    L1 = CO_FMA(YO(6), RCT(1, 7), L1); \
    g1a = CO_FMA(YO(4), RCT(1, 0), g1a); \
    L0 = CO_FMA(YO(5), RCT(1, 1), L0); \
    g1a = CO_FMA(YOS(4), RCT(1, 2), g1a); \
    P1 = CO_MUL(YO(16), g1a); \
    const double2 s64 = RCS2(79); \
    g2a = CO_MUL(YO(1), s64.x); \
    const double2 s65 = RCS2(81); \
    g2a = CO_FMA(YO(6), s65.x, g2a); \
    P0 = CO_FMA(YO(45), g2a, P0); \
    g0a = CO_MUL(YO(6), s64.y); \
    g0a = CO_FMA(YO(7), s65.y, g0a); \
    L1 = CO_FMA(YO(36), g0a, L1); \
    const double2 s66 = RCS2(94); \
    g1a = CO_MUL(YO(39), s66.y); \
    const double2 s67 = RCS2(102); \
    g1a = CO_FMA(YO(16), s67.y, g1a); \
    L0 = CO_FMA(YO(0), g1a, L0); \
    TM_WAIT(0, 4); \
    TM_LD8(1, 0, 176, 144, 151, 149, 153); \
    P1 = CO_FMA((YO(11) * YO(10)), RCT(0, 1), P1); \
    L1 = CO_FMA(YO(1), RCT(0, 0), L1); \
    P0 = CO_FMA(YO(16), RCT(0, 4), P0); \
    L0 = CO_FMA(YO(2), RCT(0, 5), L0); \
    P1 = CO_FMA((YO(3) * YO(23)), RCT(0, 7), P1); \
    L1 = CO_FMA(YO(1), RCT(0, 6), L1); \
    const double2 s68 = RCS2(47); \
    P0 = CO_FMA(YO(39), s68.y, P0); \
    L0 = CO_FMA(YO(13), s68.x, L0); \
    CO_WAIT_Y(1); \
    CO_GET(3, 17, 1, 1); \
    CO_GET(4, 18, 0, 1); \
    L1 = CO_FMA(YO(18), RCT(0, 3), L1); \
    v0 = G0a; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    CO_PUT(9, v1, v0); \
    CO_PUT(10, v2, 0.0); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(1), RCT(0, 6)); \
    L0 = CO_MUL(YO(3), RCT(0, 7)); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 104, 137, 139); \
    TM_LD2(0, 2, 60, 136); \
    TM_LD2(0, 3, 500, 140); \
    g0a = CO_MUL(YO(1), RCT(1, 1)); \
    L1 = CO_MUL(YO(6), RCT(1, 0)); \
    g0a = CO_FMA(YO(3), RCT(1, 2), g0a); \
    L0 = CO_FMA(YO(4), RCT(1, 3), L0); \
    g0a = CO_FMA(YO(4), RCT(1, 4), g0a); \
    L1 = CO_FMA(YO(5), RCT(1, 5), L1); \
    g0a = CO_FMA(YO(2), RCT(1, 6), g0a); \
    L0 = CO_FMA(YO(0), RCT(1, 7), L0); \
    P0 = CO_MUL(YO(31), g0a); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 60, 136); \
    TM_LD2(1, 1, 76, 90); \
    TM_LD2(1, 2, 92, 93); \
    TM_LD2(1, 3, 464, 145); \
    g1a = CO_MUL(YO(2), RCT(0, 5)); \
    L1 = CO_ADD(L1, RCT(0, 4)); \
    g1a = CO_FMA(YO(5), RCT(0, 7), g1a); \
    L0 = CO_FMA(YO(4), RCT(0, 6), L0); \
    P1 = CO_MUL(YO(25), g1a); \
    g2a = CO_MUL(YO(13), RCT(0, 1)); \
    L1 = CO_FMA(YO(2), RCT(0, 0), L1); \
    g2a = CO_FMA(YO(11), RCT(0, 3), g2a); \
    L0 = CO_FMA(YO(3), RCT(0, 2), L0); \
    P0 = CO_FMA(YO(10), g2a, P0); \
    TM_WAIT(1, 4); \
    TM_LD2(0, 0, 332, 108); \
    TM_LD2(0, 1, 404, 127); \
    TM_LD2(0, 2, 444, 110); \
    TM_LD2(0, 3, 500, 140); \
    P1 = CO_FMA((YO(16) * YO(3)), RCT(1, 2), P1); \
    L1 = CO_FMA(YO(2), RCT(1, 3), L1); \
    P0 = CO_FMA((YO(13) * YO(8)), RCT(1, 7), P0); \
    L0 = CO_ADD(L0, RCT(1, 6)); \
    CO_WAIT_Y(0); \
    CO_GET(0, 19, 1, 1); \
    CO_GET(1, 20, 0, 1); \
    CO_GET(2, 21, 1, 1); \
    v0 = G0a; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    P0 = CO_MUL((YO(16) * YO(6)), RCT(1, 4)); \
    L0 = CO_MUL(YO(4), RCT(1, 5)); \
    v3 = P0; \
    v4 = L0; \
    CO_PUT(2, v1, v0); \
    CO_PUT(3, v2, v3); \
    CO_PUT(4, v4, 0.0); \
    CO_ARRIVE_P(0); \
    G0a = RCT(1, 0); \
    L0 = CO_MUL(YO(2), RCT(1, 1)); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 224, 113, 115); \
    TM_LD2(1, 2, 368, 112); \
    TM_LD2(1, 3, 440, 105); \
    G0a = CO_FMA(YO(4), RCT(0, 6), G0a); \
    L1 = CO_MUL(YO(5), RCT(0, 7)); \
    g0a = CO_MUL(YO(28), RCT(0, 3)); \
    L0 = CO_FMA(YO(4), RCT(0, 2), L0); \
    g0a = CO_FMA(YO(18), RCT(0, 5), g0a); \
    L1 = CO_FMA(YO(13), RCT(0, 4), L1); \
    P0 = CO_MUL(YO(8), g0a); \
    P1 = CO_MUL((YO(14) * YO(9)), RCT(0, 1)); \
    L0 = CO_FMA(YO(3), RCT(0, 0), L0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 376, 117, 119); \
    TM_LD2(0, 2, 372, 114); \
    TM_LD2(0, 3, 448, 111); \
    P0 = CO_FMA((YO(21) * YO(4)), RCT(1, 6), P0); \
    L1 = CO_FMA(YO(2), RCT(1, 7), L1); \
    const double2 s69 = RCS2(30); \
    P1 = CO_FMA((YO(1) * YO(37)), s69.x, P1); \
    L0 = CO_FMA(YO(10), s69.y, L0); \
    CO_WAIT_Y(1); \
    CO_GET(3, 22, 0, 1); \
    v0 = G0a; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    CO_PUT(9, v1, v0); \
    CO_PUT(10, v2, 0.0); \
    CO_ARRIVE_P(1); \
    g0a = CO_MUL((YOS(6) * YO(2)), RCT(1, 1)); \
    L0 = CO_MUL(YO(3), RCT(1, 0)); \
    g0a = CO_FMA((YO(9) * YO(2)), RCT(1, 3), g0a); \
    L1 = CO_MUL(YO(1), RCT(1, 2)); \
    g0a = CO_FMA((YO(10) * YO(2)), RCT(1, 5), g0a); \
    L0 = CO_FMA(YO(4), RCT(1, 4), L0); \
    TM_WAIT(0, 4); \
    TM_LD8(1, 0, 160, 128, 132, 133, 134); \
    g0a = CO_FMA((YOS(6) * YO(4)), RCT(0, 5), g0a); \
    L1 = CO_FMA(YO(1), RCT(0, 4), L1); \
    g0a = CO_FMA(YO(15), RCT(0, 7), g0a); \
    L0 = CO_FMA(YO(2), RCT(0, 6), L0); \
    P0 = CO_MUL(YO(8), g0a); \
    const double2 s70 = RCS2(26); \
    P1 = CO_MUL((YO(3) * YO(36)), s70.x); \
    L1 = CO_FMA(YO(13), s70.y, L1); \
    CO_WAIT_Y(0); \
    CO_GET(0, 23, 1, 1); \
    CO_GET(1, 24, 0, 1); \
    v0 = CO_ADD(P0, P1); \
    v1 = CO_ADD(L0, L1); \
    CO_PUT(2, v0, v1); \
    CO_ARRIVE_P(0); \
    g0a = CO_MUL(YO(8), RCT(0, 1)); \
    L0 = CO_MUL(YO(3), RCT(0, 0)); \
    g0a = CO_FMA(YO(9), RCT(0, 3), g0a); \
    L0 = CO_FMA(YO(1), RCT(0, 2), L0); \
    P0 = CO_MUL(YO(20), g0a); \
    CO_WAIT_Y(1); \
    CO_GET(3, 25, 1, 1); \
    v0 = P0; \
    v1 = L0; \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 384, 121, 123); \
    TM_LD2(0, 2, 404, 127); \
    TM_LD2(0, 3, 452, 125); \
    g0a = CO_MUL(YO(4), RCT(1, 0)); \
    L0 = CO_MUL(YO(5), RCT(1, 1)); \
    g0a = CO_FMA(YO(3), RCT(1, 2), g0a); \
    L1 = CO_MUL(YO(4), RCT(1, 3)); \
    g0a = CO_FMA(YO(6), RCT(1, 4), g0a); \
    L0 = CO_FMA(YO(7), RCT(1, 5), L0); \
    g0a = CO_FMA(YO(1), RCT(1, 6), g0a); \
    L1 = CO_FMA(YO(6), RCT(1, 7), L1); \
    P0 = CO_MUL(YO(29), g0a); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 160, 128, 132); \
    TM_LD2(1, 2, 472, 159); \
    TM_LD2(1, 3, 496, 126); \
    g1a = CO_MUL(YO(0), RCT(0, 1)); \
    L0 = CO_FMA(YO(2), RCT(0, 0), L0); \
    g1a = CO_FMA(YO(5), RCT(0, 3), g1a); \
    L1 = CO_FMA(YO(4), RCT(0, 2), L1); \
    g1a = CO_FMA(YO(2), RCT(0, 7), g1a); \
    L0 = CO_ADD(L0, RCT(0, 6)); \
    P1 = CO_MUL(YO(11), g1a); \
    P0 = CO_FMA((YO(25) * YO(4)), RCT(0, 4), P0); \
    L1 = CO_FMA(YO(8), RCT(0, 5), L1); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 168, 133, 134); \
    TM_LD4(0, 2, 456, 131, 135); \
    P1 = CO_FMA(YO(30), RCT(1, 4), P1); \
    L0 = CO_FMA(YO(13), RCT(1, 5), L0); \
    P0 = CO_FMA(YO(17), RCT(1, 6), P0); \
    L1 = CO_ADD(L1, RCT(1, 7)); \
    const double2 s71 = RCS2(20); \
    P1 = CO_FMA((YO(2) * YO(32)), s71.x, P1); \
    L0 = CO_FMA(YO(13), s71.y, L0); \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    CO_PUT(10, v0, v1); \
    CO_PUT(11, v2, v3); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(5), RCT(1, 1)); \
    L0 = CO_MUL(YO(4), RCT(1, 0)); \
    G0a = CO_FMA(YO(4), RCT(1, 3), G0a); \
    L1 = CO_MUL(YO(3), RCT(1, 2)); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 16, 161, 162); \
    TM_LD2(1, 2, 192, 163); \
    TM_LD2(1, 3, 472, 159); \
    G0a = CO_FMA(YO(7), RCT(0, 1), G0a); \
    L0 = CO_FMA(YO(6), RCT(0, 0), L0); \
    G0a = CO_FMA(YO(6), RCT(0, 3), G0a); \
    L1 = CO_FMA(YO(1), RCT(0, 2), L1); \
    P0 = CO_MUL((YO(17) * YO(0)), RCT(0, 5)); \
    L0 = CO_FMA(YO(2), RCT(0, 4), L0); \
    P1 = CO_MUL((YO(13) * YO(4)), RCT(0, 7)); \
    L1 = CO_ADD(L1, RCT(0, 6)); \
    CO_WAIT_Y(0); \
    CO_GET(0, 26, 0, 1); \
    v0 = G0a; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 8, 164, 165); \
    TM_LD2(0, 2, 196, 166); \
    TM_LD2(0, 3, 476, 160); \
    G0a = CO_MUL(YO(13), RCT(1, 7)); \
    L0 = RCT(1, 6); \
    g0a = CO_MUL(YO(33), RCT(1, 1)); \
    L1 = CO_MUL(YO(4), RCT(1, 0)); \
    g0a = CO_FMA(YO(32), RCT(1, 3), g0a); \
    L0 = CO_FMA(YO(4), RCT(1, 2), L0); \
    g0a = CO_FMA(YO(35), RCT(1, 5), g0a); \
    L1 = CO_FMA(YO(4), RCT(1, 4), L1); \
    TM_WAIT(0, 4); \
    TM_LD2(1, 0, 28, 148); \
    TM_LD2(1, 1, 204, 158); \
    TM_LD2(1, 2, 392, 152); \
    TM_LD2(1, 3, 508, 167); \
    g0a = CO_FMA(YO(16), RCT(0, 7), g0a); \
    L0 = CO_ADD(L0, RCT(0, 6)); \
    P0 = CO_MUL(YO(5), g0a); \
    g1a = CO_MUL(YO(33), RCT(0, 1)); \
    L1 = CO_FMA(YO(2), RCT(0, 0), L1); \
    g1a = CO_FMA(YO(32), RCT(0, 3), g1a); \
    L0 = CO_FMA(YO(2), RCT(0, 2), L0); \
    g1a = CO_FMA(YO(35), RCT(0, 5), g1a); \
    L1 = CO_FMA(YO(2), RCT(0, 4), L1); \
    P1 = CO_MUL(YO(0), g1a); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 176, 144, 151); \
    TM_LD2(0, 2, 396, 156); \
    TM_LD2(0, 3, 504, 154); \
    P0 = CO_FMA((YO(4) * YO(33)), RCT(1, 7), P0); \
    L0 = CO_FMA(YO(3), RCT(1, 6), L0); \
    v3 = G0a; \
    v4 = CO_ADD(P0, P1); \
    v5 = CO_ADD(L0, L1); \
    CO_PUT(3, v1, v0); \
    CO_PUT(4, v2, v4); \
    CO_PUT(5, v3, v5); \
    CO_ARRIVE_P(0); \
    g0a = CO_MUL(YO(5), RCT(1, 1)); \
    L0 = CO_MUL(YO(4), RCT(1, 0)); \
    g0a = CO_FMA(YO(6), RCT(1, 3), g0a); \
    L1 = CO_MUL(YO(1), RCT(1, 2)); \
    g0a = CO_FMA(YO(0), RCT(1, 5), g0a); \
    L0 = CO_FMA(YO(2), RCT(1, 4), L0); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 184, 149, 153); \
    TM_LD2(1, 2, 12, 165); \
    TM_LD2(1, 3, 468, 146); \
    g0a = CO_FMA(YO(7), RCT(0, 5), g0a); \
    L1 = CO_FMA(YO(6), RCT(0, 4), L1); \
    g0a = CO_FMA(YO(12), RCT(0, 7), g0a); \
    L0 = CO_FMA(YO(13), RCT(0, 6), L0); \
    P0 = CO_MUL(YO(34), g0a); \
    g1a = CO_MUL(YO(6), RCT(0, 0)); \
    L1 = CO_FMA(YO(1), RCT(0, 1), L1); \
    g1a = CO_FMA(YO(4), RCT(0, 3), g1a); \
    L0 = CO_FMA(YO(3), RCT(0, 2), L0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 16, 161, 162); \
    TM_LD2(0, 2, 8, 164); \
    TM_LD2(0, 3, 508, 167); \
    g1a = CO_FMA(YO(5), RCT(1, 1), g1a); \
    L1 = CO_FMA(YO(4), RCT(1, 0), L1); \
    g1a = CO_FMA(YO(0), RCT(1, 3), g1a); \
    L0 = CO_FMA(YO(2), RCT(1, 2), L0); \
    P1 = CO_MUL(YO(23), g1a); \
    const double2 s72 = RCS2(18); \
    g2a = CO_MUL(YO(3), s72.x); \
    L1 = CO_FMA(YO(4), s72.y, L1); \
    const double2 s73 = RCS2(22); \
    g2a = CO_FMA(YO(4), s73.x, g2a); \
    L0 = CO_FMA(YO(5), s73.y, L0); \
    P0 = CO_FMA(YO(32), g2a, P0); \
    P1 = CO_FMA((YO(13) * YO(10)), RCT(1, 7), P1); \
    L1 = CO_ADD(L1, RCT(1, 6)); \
    const double2 s74 = RCS2(23); \
    P0 = CO_FMA(YO(32), s74.x, P0); \
    L0 = CO_FMA(YO(2), s74.y, L0); \
    CO_WAIT_Y(1); \
    CO_GET(3, 27, 1, 1); \
    CO_GET(4, 28, 0, 1); \
    v0 = CO_ADD(P0, P1); \
    v1 = CO_ADD(L0, L1); \
    CO_PUT(8, v0, v1); \
    CO_ARRIVE_P(1); \
    e30a = CO_MUL(YO(2), RCT(1, 4)); \
    L0 = CO_MUL(YO(0), RCT(1, 5)); \
    TM_WAIT(0, 4); \
    TM_LD4(1, 0, 392, 152, 156); \
    TM_LD2(1, 2, 28, 148); \
    TM_LD2(1, 3, 204, 158); \
    e30a = CO_FMA(YO(4), RCT(0, 2), e30a); \
    L0 = CO_FMA(YO(5), RCT(0, 3), L0); \
    const double2 s75 = RCS2(19); \
    P0 = CO_MUL((YO(16) * YO(5)), s75.y); \
    L0 = CO_FMA(YO(2), s75.x, L0); \
    const double2 s76 = RCS2(20); \
    P0 = CO_FMA((YO(28) * YO(13)), s76.y, P0); \
    L0 = CO_FMA(YO(2), s76.x, L0); \
    CO_WAIT_Y(0); \
    CO_GET(0, 29, 1, 1); \
    CO_GET(1, 30, 0, 1); \
    P0 = CO_FMA(YO(30), e30a, P0); \
    v0 = P0; \
    v1 = L0; \
    g0a = CO_MUL(YO(2), RCT(0, 4)); \
    L0 = CO_MUL(YO(0), RCT(0, 5)); \
    g0a = CO_FMA(YO(4), RCT(0, 0), g0a); \
    L1 = CO_MUL(YO(5), RCT(0, 1)); \
    g0a = CO_FMA(YO(3), RCT(0, 6), g0a); \
    L0 = CO_FMA(YO(4), RCT(0, 7), L0); \
    const double2 s77 = RCS2(2); \
    g0a = CO_FMA(YO(13), s77.x, g0a); \
    L1 = CO_FMA(YO(12), s77.y, L1); \
    const double2 s78 = RCS2(6); \
    g0a = CO_FMA(YO(6), s78.x, g0a); \
    L0 = CO_FMA(YO(7), s78.y, L0); \
    P0 = CO_MUL(YO(30), g0a); \
    const double2 s79 = RCS2(8); \
    P1 = CO_MUL((YO(16) * YO(4)), s79.x); \
    L1 = CO_ADD(L1, s79.y); \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    CO_PUT(2, v0, v1); \
    CO_PUT(3, v2, v3); \
    CO_ARRIVE_P(0); \
    TM_WAIT(1, 4); \
    TM_LD4(0, 0, 192, 163, 166); \
    TM_LD2(0, 2, 200, 147); \
    TM_LD2(0, 3, 504, 154); \
    e31a = CO_MUL(YO(4), RCT(1, 4)); \
    L0 = CO_MUL(YO(5), RCT(1, 5)); \
    e31a = CO_FMA(YO(1), RCT(1, 6), e31a); \
    L1 = CO_MUL(YO(6), RCT(1, 7)); \
    e31a = CO_FMA(YO(2), RCT(1, 0), e31a); \
    L0 = CO_FMA(YO(0), RCT(1, 1), L0); \
    e31a = CO_FMA(YO(6), RCT(1, 2), e31a); \
    L1 = CO_FMA(YO(7), RCT(1, 3), L1); \
    TM_WAIT(0, 4); \
    e31a = CO_FMA(YO(13), RCT(0, 6), e31a); \
    L0 = CO_FMA(YO(12), RCT(0, 7), L0); \
    P1 = CO_MUL((YO(13) * YO(8)), RCT(0, 5)); \
    L1 = CO_ADD(L1, RCT(0, 4)); \
    CO_WAIT_Y(1); \
    CO_GET(3, 31, 1, 1); \
    P0 = CO_MUL(YO(31), e31a); \
    v0 = CO_ADD(P0, P1); \
    v1 = CO_ADD(L0, L1); \
    g0a = CO_MUL(YO(4), RCT(0, 0)); \
    L0 = CO_MUL(YO(5), RCT(0, 1)); \
    g0a = CO_FMA(YO(2), RCT(0, 2), g0a); \
    L1 = CO_MUL(YO(0), RCT(0, 3)); \
    const double2 s80 = RCS2(1); \
    g0a = CO_FMA(YO(3), s80.x, g0a); \
    L0 = CO_FMA(YO(4), s80.y, L0); \
    const double2 s81 = RCS2(4); \
    g0a = CO_FMA(YO(13), s81.x, g0a); \
    L1 = CO_FMA(YO(12), s81.y, L1); \
    const double2 s82 = RCS2(7); \
    g0a = CO_FMA(YO(6), s82.x, g0a); \
    L0 = CO_FMA(YO(7), s82.y, L0); \
    P0 = CO_MUL(YO(30), g0a); \
    const double2 s83 = RCS2(12); \
    g1a = CO_MUL(YO(6), s83.y); \
    L1 = CO_FMA(YO(1), s83.x, L1); \
    const double2 s84 = RCS2(16); \
    g1a = CO_FMA(YO(5), s84.y, g1a); \
    L0 = CO_FMA(YO(4), s84.x, L0); \
    P1 = CO_MUL(YO(31), g1a); \
    const double2 s85 = RCS2(14); \
    P0 = CO_FMA((YO(28) * YO(13)), s85.y, P0); \
    L1 = CO_FMA(YO(2), s85.x, L1); \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    const double2 s86 = RCS2(27); \
    g0a = CO_MUL(YO(2), s86.x); \
    L0 = s86.y; \
    const double2 s87 = RCS2(28); \
    g0a = CO_FMA(YO(6), s87.x, g0a); \
    L1 = CO_MUL(YO(1), s87.y); \
    const double2 s88 = RCS2(29); \
    g0a = CO_FMA(YO(5), s88.y, g0a); \
    L0 = CO_FMA(YO(4), s88.x, L0); \
    const double2 s89 = RCS2(37); \
    g0a = CO_FMA(YO(10), s89.x, g0a); \
    L1 = CO_FMA(YO(8), s89.y, L1); \
    P0 = CO_MUL(YO(37), g0a); \
    const double2 s90 = RCS2(33); \
    g1a = CO_MUL(YO(1), s90.x); \
    L0 = CO_FMA(YO(6), s90.y, L0); \
    const double2 s91 = RCS2(36); \
    g1a = CO_FMA(YO(4), s91.x, g1a); \
    L1 = CO_FMA(YO(5), s91.y, L1); \
    P1 = CO_MUL(YO(38), g1a); \
    const double2 s92 = RCS2(26); \
    P0 = CO_FMA((YO(26) * YO(13)), s92.y, P0); \
    L0 = CO_FMA(YO(3), s92.x, L0); \
    const double2 s93 = RCS2(76); \
    P1 = CO_FMA(YO(45), s93.x, P1); \
    L1 = CO_FMA(YO(16), s93.y, L1); \
    v4 = CO_ADD(P0, P1); \
    v5 = CO_ADD(L0, L1); \
    CO_PUT(10, v0, v1); \
    CO_PUT(11, v2, v3); \
    CO_PUT(12, v4, v5); \
    CO_ARRIVE_P(1); \
    const double2 s94 = RCS2(27); \
    G0a = s94.y; \
    L0 = CO_MUL(YO(2), s94.x); \
    const double2 s95 = RCS2(28); \
    G0a = CO_FMA(YO(1), s95.y, G0a); \
    L1 = CO_MUL(YO(6), s95.x); \
    const double2 s96 = RCS2(29); \
    G0a = CO_FMA(YO(4), s96.x, G0a); \
    L0 = CO_FMA(YO(5), s96.y, L0); \
    const double2 s97 = RCS2(37); \
    G0a = CO_FMA(YO(8), s97.y, G0a); \
    L1 = CO_FMA(YO(10), s97.x, L1); \
    const double2 s98 = RCS2(30); \
    P0 = CO_MUL((YO(25) * YO(10)), s98.y); \
    L0 = CO_FMA(YO(1), s98.x, L0); \
    const double2 s99 = RCS2(38); \
    P1 = CO_MUL(((YO(22) * YO(4)) * YO(8)), s99.y); \
    L1 = CO_FMA(YO(6), s99.x, L1); \
    const double2 s100 = RCS2(74); \
    P0 = CO_FMA(YO(43), s100.y, P0); \
    L0 = CO_FMA(YO(13), s100.x, L0); \
    CO_WAIT_Y(0); \
    CO_GET(0, 32, 0, 1); \
    CO_GET(1, 33, 1, 1); \
    v0 = G0a; \
    v1 = CO_ADD(P0, P1); \
    v2 = CO_ADD(L0, L1); \
    const double2 s101 = RCS2(36); \
    G0a = CO_MUL(YO(5), s101.y); \
    L0 = CO_MUL(YO(4), s101.x); \
    const double2 s102 = RCS2(46); \
    g0a = CO_MUL((YO(22) * YO(11)), s102.y); \
    L1 = CO_MUL(YO(6), s102.x); \
    const double2 s103 = RCS2(72); \
    g0a = CO_FMA(YO(43), s103.x, g0a); \
    L0 = CO_FMA((YO(44) * YO(2)), s103.y, L0); \
    P0 = CO_MUL(YO(4), g0a); \
    const double2 s104 = RCS2(35); \
    g1a = CO_MUL(YO(21), s104.x); \
    L1 = CO_ADD(L1, s104.y); \
    const double2 s105 = RCS2(49); \
    g1a = CO_FMA(YO(22), s105.x, g1a); \
    L0 = CO_FMA(YO(2), s105.y, L0); \
    P1 = CO_MUL(YO(13), g1a); \
    const double2 s106 = RCS2(43); \
    P0 = CO_FMA((YO(2) * YO(39)), s106.x, P0); \
    L1 = CO_FMA(YO(0), s106.y, L1); \
    const double2 s107 = RCS2(78); \
    P1 = CO_FMA((YO(1) * YO(45)), s107.x, P1); \
    L0 = CO_FMA((YO(21) * YO(6)), s107.y, L0); \
    const double2 s108 = RCS2(91); \
    P0 = CO_FMA(YO(48), s108.x, P0); \
    L1 = CO_FMA(YO(18), s108.y, L1); \
    const double2 s109 = RCS2(99); \
    P1 = CO_FMA(YO(47), s109.x, P1); \
    L0 = CO_FMA(YO(13), s109.y, L0); \
    v3 = G0a; \
    v4 = CO_ADD(P0, P1); \
    v5 = CO_ADD(L0, L1); \
    CO_PUT(2, v1, v0); \
    CO_PUT(3, v2, v4); \
    CO_PUT(4, v3, v5); \
    CO_ARRIVE_P(0); \
    const double2 s110 = RCS2(42); \
    g0a = CO_MUL((YO(25) * YO(13)), s110.y); \
    L0 = CO_MUL(YO(3), s110.x); \
    const double2 s111 = RCS2(83); \
    g0a = CO_FMA(YO(46), s111.x, g0a); \
    const double2 s112 = RCS2(94); \
    g0a = CO_FMA(YO(48), s112.x, g0a); \
    P0 = CO_MUL(YO(2), g0a); \
    const double2 s113 = RCS2(63); \
    g1a = CO_MUL(YO(41), s113.x); \
    L1 = CO_MUL(YO(6), s113.y); \
    const double2 s114 = RCS2(66); \
    g1a = CO_FMA(YO(42), s114.x, g1a); \
    L0 = CO_FMA(YO(6), s114.y, L0); \
    P1 = CO_MUL(YO(1), g1a); \
    const double2 s115 = RCS2(89); \
    g2a = CO_MUL(YO(46), s115.x); \
    const double2 s116 = RCS2(93); \
    g2a = CO_FMA(YO(48), s116.x, g2a); \
    P0 = CO_FMA(YO(4), g2a, P0); \
    const double2 s117 = RCS2(47); \
    g0a = CO_MUL(YO(22), s117.x); \
    L1 = CO_ADD(L1, s117.y); \
    const double2 s118 = RCS2(48); \
    g0a = CO_FMA(YO(16), s118.y, g0a); \
    L0 = CO_FMA(YO(2), s118.x, L0); \
    P1 = CO_FMA(YO(13), g0a, P1); \
    g1a = CO_MUL(YO(5), s116.y); \
    const double2 s119 = RCS2(94); \
    g1a = CO_FMA(YO(0), s119.y, g1a); \
    L1 = CO_FMA(YO(22), g1a, L1); \
    const double2 s120 = RCS2(40); \
    P0 = CO_FMA((YO(18) * YO(10)), s120.y, P0); \
    L0 = CO_FMA(YO(3), s120.x, L0); \
    const double2 s121 = RCS2(62); \
    P1 = CO_FMA(YO(41), s121.y, P1); \
    L1 = CO_FMA(YO(2), s121.x, L1); \
    const double2 s122 = RCS2(75); \
    P0 = CO_FMA(YO(45), s122.x, P0); \
    L0 = CO_FMA(YO(21), s122.y, L0); \
    CO_WAIT_Y(1); \
    CO_GET(3, 34, 0, 1); \
    CO_GET(4, 35, 1, 1); \
    CO_GET(5, 36, 0, 1); \
    v0 = CO_ADD(P0, P1); \
    v1 = CO_ADD(L0, L1); \
    const double2 s123 = RCS2(51); \
    g0a = CO_MUL(YO(6), s123.y); \
    L0 = CO_MUL(YO(1), s123.x); \
    const double2 s124 = RCS2(53); \
    g0a = CO_FMA(YO(0), s124.y, g0a); \
    L1 = CO_MUL(YO(2), s124.x); \
    const double2 s125 = RCS2(59); \
    g0a = CO_FMA(YO(7), s125.y, g0a); \
    L0 = CO_FMA(YO(6), s125.x, L0); \
    P0 = CO_MUL(YO(41), g0a); \
    const double2 s126 = RCS2(52); \
    g1a = CO_MUL(YO(6), s126.y); \
    L1 = CO_FMA(YO(1), s126.x, L1); \
    const double2 s127 = RCS2(57); \
    g1a = CO_FMA(YO(5), s127.y, g1a); \
    L0 = CO_FMA(YO(4), s127.x, L0); \
    const double2 s128 = RCS2(60); \
    g1a = CO_FMA(YO(7), s128.y, g1a); \
    L1 = CO_FMA(YO(6), s128.x, L1); \
    P1 = CO_MUL(YO(42), g1a); \
    const double2 s129 = RCS2(50); \
    P0 = CO_FMA((YO(18) * YO(13)), s129.y, P0); \
    L0 = CO_ADD(L0, s129.x); \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    CO_PUT(10, v0, v1); \
    CO_PUT(11, v2, v3); \
    CO_ARRIVE_P(1); \
    const double2 s130 = RCS2(51); \
    G0a = CO_MUL(YO(1), s130.x); \
    L0 = CO_MUL(YO(6), s130.y); \
    const double2 s131 = RCS2(53); \
    G0a = CO_FMA(YO(2), s131.x, G0a); \
    L0 = CO_FMA(YO(0), s131.y, L0); \
    const double2 s132 = RCS2(55); \
    G0a = CO_FMA(YO(3), s132.x, G0a); \
    L0 = CO_FMA(YO(4), s132.y, L0); \
    const double2 s133 = RCS2(58); \
    G0a = CO_FMA(YO(4), s133.x, G0a); \
    L0 = CO_FMA(YO(5), s133.y, L0); \
    const double2 s134 = RCS2(59); \
    G0a = CO_FMA(YO(6), s134.x, G0a); \
    L0 = CO_FMA(YO(7), s134.y, L0); \
    CO_WAIT_Y(0); \
    CO_GET(0, 37, 1, 1); \
    CO_GET(1, 38, 0, 1); \
    v0 = G0a; \
    v1 = L0; \
    CO_PUT(2, v0, v1); \
    CO_ARRIVE_P(0); \
    const double2 s135 = RCS2(61); \
    G0a = s135.x; \
    L0 = s135.y; \
    const double2 s136 = RCS2(52); \
    e40a = CO_MUL(YO(1), s136.x); \
    L0 = CO_FMA(YO(6), s136.y, L0); \
    const double2 s137 = RCS2(54); \
    e40a = CO_FMA(YO(2), s137.x, e40a); \
    L0 = CO_FMA(YO(0), s137.y, L0); \
    const double2 s138 = RCS2(56); \
    e40a = CO_FMA(YO(3), s138.x, e40a); \
    L0 = CO_FMA(YO(4), s138.y, L0); \
    const double2 s139 = RCS2(57); \
    e40a = CO_FMA(YO(4), s139.x, e40a); \
    L0 = CO_FMA(YO(5), s139.y, L0); \
    CO_WAIT_Y(1); \
    CO_GET(3, 39, 1, 1); \
    CO_GET(4, 40, 0, 1); \
    P0 = CO_MUL(YO(40), e40a); \
    v0 = G0a; \
    v1 = P0; \
    v2 = L0; \
    const double2 s140 = RCS2(67); \
    g0a = CO_MUL((YO(21) * YO(2)), s140.y); \
    L0 = s140.x; \
    const double2 s141 = RCS2(68); \
    g0a = CO_FMA(YOS(7), s141.y, g0a); \
    L1 = s141.x; \
    const double2 s142 = RCS2(69); \
    g0a = CO_FMA(YOS(7), s142.x, g0a); \
    L0 = CO_ADD(L0, s142.y); \
    const double2 s143 = RCS2(71); \
    g0a = CO_FMA((YO(0) * YO(21)), s143.y, g0a); \
    L1 = CO_FMA(YO(2), s143.x, L1); \
    const double2 s144 = RCS2(73); \
    g0a = CO_FMA((YO(12) * YO(21)), s144.y, g0a); \
    L0 = CO_FMA(YO(13), s144.x, L0); \
    P0 = CO_MUL(YO(22), g0a); \
    const double2 s145 = RCS2(72); \
    P1 = CO_MUL(((YO(38) * YO(44)) * YO(2)), s145.y); \
    L1 = CO_FMA(YO(4), s145.x, L1); \
    const double2 s146 = RCS2(74); \
    P0 = CO_FMA((YO(37) * YO(13)), s146.x, P0); \
    L0 = CO_ADD(L0, s146.y); \
    v3 = CO_ADD(P0, P1); \
    v4 = CO_ADD(L0, L1); \
    CO_PUT(9, v1, v0); \
    CO_PUT(10, v2, v3); \
    CO_PUT(11, v4, 0.0); \
    CO_ARRIVE_P(1); \
    G0a = CO_MUL(YO(4), s145.x); \
    L0 = CO_MUL((YO(2) * YO(38)), s145.y); \
    CO_WAIT_Y(0); \
    CO_GET(0, 41, 1, 1); \
    v0 = G0a; \
    v1 = L0; \
    const double2 s147 = RCS2(75); \
    g0a = CO_MUL(YO(39), s147.y); \
    L0 = s147.x; \
    const double2 s148 = RCS2(78); \
    g0a = CO_FMA((YO(38) * YO(6)), s148.y, g0a); \
    L1 = CO_MUL(YO(1), s148.x); \
    const double2 s149 = RCS2(80); \
    g0a = CO_FMA((YO(38) * YO(7)), s149.y, g0a); \
    L0 = CO_FMA(YO(6), s149.x, L0); \
    P0 = CO_MUL(YO(21), g0a); \
    const double2 s150 = RCS2(76); \
    g1a = CO_MUL(YO(16), s150.y); \
    L1 = CO_ADD(L1, s150.x); \
    const double2 s151 = RCS2(79); \
    g1a = CO_FMA((YO(22) * YO(6)), s151.y, g1a); \
    L0 = CO_FMA(YO(1), s151.x, L0); \
    const double2 s152 = RCS2(81); \
    g1a = CO_FMA((YO(22) * YO(7)), s152.y, g1a); \
    L1 = CO_FMA(YO(6), s152.x, L1); \
    P1 = CO_MUL(YO(36), g1a); \
    v2 = CO_ADD(P0, P1); \
    v3 = CO_ADD(L0, L1); \
    const double2 s153 = RCS2(88); \
    L0 = CO_MUL(YO(4), s153.x); \
    const double2 s154 = RCS2(89); \
    L0 = CO_FMA(YO(4), s154.x, L0); \
    const double2 s155 = RCS2(90); \
    L0 = CO_FMA(YO(4), s155.x, L0); \
    v4 = L0; \
    CO_PUT(2, v0, v1); \
    CO_PUT(3, v2, v3); \
    CO_PUT(4, v4, 0.0); \
    CO_ARRIVE_P(0); \
    const double2 s156 = RCS2(84); \
    G0a = CO_MUL(YO(2), s156.x); \
    G0a = CO_FMA(YO(4), s153.x, G0a); \
    const double2 s157 = RCS2(101); \
    P0 = CO_MUL((YO(39) * YO(13)), s157.y); \
    L0 = CO_MUL(YO(2), s157.x); \
    CO_WAIT_Y(1); \
    CO_GET(3, 42, 0, 1); \
    CO_GET(4, 43, 1, 1); \
    v0 = G0a; \
    v1 = P0; \
    v2 = L0; \
    const double2 s158 = RCS2(86); \
    G0a = CO_MUL(YO(2), s158.x); \
    const double2 s159 = RCS2(87); \
    G0a = CO_FMA(YO(4), s159.x, G0a); \
    const double2 s160 = RCS2(92); \
    g0a = CO_MUL(YO(39), s160.y); \
    L0 = s160.x; \
    const double2 s161 = RCS2(95); \
    g0a = CO_FMA((YOS(4) * YO(13)), s161.y, g0a); \
    L1 = CO_MUL(YO(2), s161.x); \
    const double2 s162 = RCS2(97); \
    g0a = CO_FMA((YO(38) * YO(0)), s162.y, g0a); \
    L0 = CO_FMA(YO(2), s162.x, L0); \
    P0 = CO_MUL(YO(16), g0a); \
    const double2 s163 = RCS2(93); \
    g1a = CO_MUL((YO(39) * YO(5)), s163.y); \
    L1 = CO_FMA(YO(4), s163.x, L1); \
    const double2 s164 = RCS2(94); \
    g1a = CO_FMA((YO(39) * YO(0)), s164.y, g1a); \
    L0 = CO_FMA(YO(2), s164.x, L0); \
    P1 = CO_MUL(YO(22), g1a); \
    const double2 s165 = RCS2(86); \
    g2a = CO_MUL(YO(0), s165.y); \
    const double2 s166 = RCS2(87); \
    g2a = CO_FMA(YO(5), s166.y, g2a); \
    L1 = CO_FMA(YO(18), g2a, L1); \
    v3 = G0a; \
    v4 = CO_ADD(P0, P1); \
    v5 = CO_ADD(L0, L1); \
    CO_PUT(9, v1, v0); \
    CO_PUT(10, v2, v4); \
    CO_PUT(11, v3, v5); \
    CO_ARRIVE_P(1); \
    CO_WAIT_Y(0); \
    CO_GET(0, 44, 0, 1); \
    CO_GET(1, 45, 1, 1); \
    CO_GET(2, 46, 0, 1); \
} while (0)
#define UC_CO_CLOSE() do { \
    double n0, n1, n2, d0, d1, d2, q0, q1, q2, fnew, rest, t00, t01, t02, t03, t04, t05, t06, t10, t11, t12, t13, t14, t15, t16, x00, x01, x02, x03, x10, x11, x12, x13, y00, y01, y02, y03, y10, y11, y12, y13; \
    CO_PF(0, 0); \
    CO_PF(1, 1); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x10, y10); \
    t00 = CO_ADD(y00, y10); \
    t01 = CO_ADD(x00, x10); \
    CO_CHECK(); \
    CO_PF(2, 2); \
    n0 = (CO_FMA(DTW(0), CO_FMA(SOUR(0), YO(21), t01), RY0(0)) - FNS(0)) * sor1; \
    d0 = CO_FMA(DTW(0), t00, rho - FSS(0)); \
    q0 = CO_QUOT(n0, d0); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x10, y10); \
    CO_TAKE(9, x11, y11); \
    t10 = y11; \
    t11 = CO_ADD(y00, x11); \
    t12 = y10; \
    t13 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(0), q0); \
    rsd += fabs(YO(0) - fnew); \
    CO_TAIL(0); \
    CO_GIVE(0, 0); \
    CO_ARRIVE_Y(0); \
    CO_PF(3, 3); \
    n1 = (CO_FMA(DTW(1), CO_FMA(YO(0), t12, t13), RY0(1)) - FNS(1)) * sor1; \
    d1 = CO_FMA(DTW(1), CO_ADD(CO_FMA(YO(0), t10, t11), (0.5 * SOUR(2))), rho - FSS(1)); \
    q1 = CO_QUOT(n1, d1); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x10, y10); \
    CO_TAKE(3, x11, y11); \
    t00 = y11; \
    t01 = CO_ADD(x01, x11); \
    t02 = CO_ADD(y00, y10); \
    t03 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(1), q1); \
    rsd += fabs(YO(1) - fnew); \
    CO_TAIL(1); \
    CO_GIVE(3, 1); \
    CO_ARRIVE_Y(1); \
    CO_PF(4, 4); \
    n2 = (CO_FMA(DTW(2), CO_FMA(SOUR(3), YO(4), CO_FMA(YO(1), t02, t03)), RY0(2)) - FNS(2)) * sor1; \
    d2 = CO_FMA(DTW(2), CO_FMA(YO(1), t00, t01), rho - FSS(2)); \
    q2 = CO_QUOT(n2, d2); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x01, y01); \
    CO_TAKE(9, x10, y10); \
    CO_TAKE(10, x11, y11); \
    t10 = y11; \
    t11 = CO_ADD(x01, x11); \
    t12 = CO_ADD(y00, y10); \
    t13 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(2), q2); \
    rsd += fabs(YO(2) - fnew); \
    CO_TAIL(2); \
    CO_GIVE(0, 2); \
    CO_ARRIVE_Y(0); \
    CO_PF(5, 5); \
    n0 = (CO_FMA(DTW(3), CO_FMA(YO(2), t12, t13), RY0(3)) - FNS(3)) * sor1; \
    d0 = CO_FMA(DTW(3), CO_ADD(CO_FMA(YO(2), t10, t11), SOUR(4)), rho - FSS(3)); \
    q0 = CO_QUOT(n0, d0); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x10, y10); \
    CO_TAKE(3, x11, y11); \
    t00 = CO_ADD(y01, y11); \
    t01 = CO_ADD(x01, x11); \
    t02 = CO_ADD(y00, y10); \
    t03 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(3), q0); \
    rsd += fabs(YO(3) - fnew); \
    CO_TAIL(3); \
    CO_GIVE(3, 3); \
    CO_ARRIVE_Y(1); \
    CO_PF(6, 6); \
    n1 = (CO_FMA(DTW(4), CO_FMA(YO(3), t02, t03), RY0(4)) - FNS(4)) * sor1; \
    d1 = CO_FMA(DTW(4), CO_ADD(CO_FMA(YO(3), t00, t01), SOUR(3)), rho - FSS(4)); \
    q1 = CO_QUOT(n1, d1); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x01, y01); \
    CO_TAKE(9, x10, y10); \
    CO_TAKE(10, x11, y11); \
    t10 = y11; \
    t11 = CO_ADD(x01, x11); \
    t12 = CO_ADD(y00, y10); \
    t13 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(4), q1); \
    rsd += fabs(YO(4) - fnew); \
    CO_TAIL(4); \
    CO_GIVE(0, 4); \
    CO_ARRIVE_Y(0); \
    CO_PF(0, 7); \
    n2 = (CO_FMA(DTW(5), CO_FMA(YO(4), t12, t13), RY0(5)) - FNS(5)) * sor1; \
    d2 = CO_FMA(DTW(5), CO_FMA(YO(4), t10, t11), rho - FSS(5)); \
    q2 = CO_QUOT(n2, d2); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x10, y10); \
    CO_TAKE(3, x11, y11); \
    t00 = x01; \
    t01 = CO_ADD(y00, x11); \
    t02 = y10; \
    t03 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(5), q2); \
    rsd += fabs(YO(5) - fnew); \
    CO_TAIL(5); \
    CO_GIVE(3, 5); \
    CO_ARRIVE_Y(1); \
    CO_PF(1, 8); \
    n0 = (CO_FMA(DTW(6), CO_FMA(YO(5), t02, t03), RY0(6)) - FNS(6)) * sor1; \
    d0 = CO_FMA(DTW(6), CO_FMA(YO(5), t00, t01), rho - FSS(6)); \
    q0 = CO_QUOT(n0, d0); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x10, y10); \
    CO_TAKE(9, x11, y11); \
    t10 = CO_ADD(y00, x11); \
    t11 = CO_ADD(x00, y10); \
    t12 = x10; \
    fnew = CO_FMA(sor2, YO(6), q0); \
    rsd += fabs(YO(6) - fnew); \
    CO_TAIL(6); \
    CO_GIVE(0, 6); \
    CO_ARRIVE_Y(0); \
    CO_PF(2, 9); \
    n1 = (CO_FMA(DTW(7), CO_FMA(YO(6), t11, t12), RY0(7)) - FNS(0)) * sor1; \
    d1 = CO_FMA(DTW(7), t10, rho - FSS(0)); \
    q1 = CO_QUOT(n1, d1); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x10, y10); \
    t00 = x01; \
    t01 = CO_ADD(y00, y10); \
    t02 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(7), q1); \
    rsd += fabs(YO(7) - fnew); \
    CO_TAIL(7); \
    CO_GIVE(3, 7); \
    CO_ARRIVE_Y(1); \
    CO_PF(3, 10); \
    n2 = (CO_FMA(DTW(8), CO_FMA(SOUR(4), YO(3), CO_FMA(SOUR(3), YO(4), CO_FMA((0.5 * SOUR(2)), YO(1), t02))), RY0(8)) - FNS(1)) * sor1; \
    d2 = CO_FMA(DTW(8), CO_FMA(YO(7), t00, t01), rho - FSS(1)); \
    q2 = CO_QUOT(n2, d2); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x01, y01); \
    CO_TAKE(9, x10, y10); \
    CO_TAKE(10, x11, y11); \
    t10 = y11; \
    t11 = CO_ADD(x01, x11); \
    t12 = CO_ADD(y00, y10); \
    t13 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(8), q2); \
    rsd += fabs(YO(8) - fnew); \
    CO_TAIL(8); \
    CO_GIVE(0, 8); \
    CO_ARRIVE_Y(0); \
    CO_PF(4, 11); \
    CO_PF(5, 12); \
    n0 = (CO_FMA(DTW(9), CO_FMA(YO(8), t12, t13), RY0(9)) - FNS(2)) * sor1; \
    d0 = CO_FMA(DTW(9), CO_FMA(YO(8), t10, t11), rho - FSS(2)); \
    q0 = CO_QUOT(n0, d0); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x10, y10); \
    t00 = CO_ADD(x01, y10); \
    t01 = y00; \
    t02 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(9), q0); \
    rsd += fabs(YO(9) - fnew); \
    CO_TAIL(9); \
    CO_GIVE(3, 9); \
    CO_ARRIVE_Y(1); \
    CO_PF(6, 13); \
    n1 = (CO_FMA(DTW(10), CO_FMA(YO(9), t01, t02), RY0(10)) - FNS(3)) * sor1; \
    d1 = CO_FMA(DTW(10), t00, rho - FSS(3)); \
    q1 = CO_QUOT(n1, d1); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x01, y01); \
    CO_TAKE(9, x02, y02); \
    CO_TAKE(10, x03, y03); \
    CO_TAKE(11, x10, y10); \
    CO_TAKE(12, x11, y11); \
    CO_TAKE(13, x12, y12); \
    t10 = CO_ADD(y01, y11); \
    t11 = CO_ADD(x01, x11); \
    t12 = CO_ADD(y00, y10); \
    t13 = CO_ADD(x00, x10); \
    t14 = CO_ADD(x03, y12); \
    t15 = y02; \
    t16 = CO_ADD(x02, x12); \
    fnew = CO_FMA(sor2, YO(10), q1); \
    rsd += fabs(YO(10) - fnew); \
    CO_TAIL(10); \
    CO_GIVE(0, 10); \
    CO_ARRIVE_Y(0); \
    CO_PF(0, 14); \
    n2 = (CO_FMA(DTW(11), CO_FMA(YO(10), t12, t13), RY0(11)) - FNS(4)) * sor1; \
    d2 = CO_FMA(DTW(11), CO_FMA(YO(10), t10, t11), rho - FSS(4)); \
    n0 = (CO_FMA(DTW(12), CO_FMA(YO(10), t15, t16), RY0(12)) - FNS(5)) * sor1; \
    d0 = CO_FMA(DTW(12), t14, rho - FSS(5)); \
    q2 = CO_QUOT(n2, d2); \
    q0 = CO_QUOT(n0, d0); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x10, y10); \
    CO_TAKE(3, x11, y11); \
    CO_TAKE(4, x12, y12); \
    t00 = x12; \
    t01 = CO_ADD(x01, y11); \
    t02 = y10; \
    t03 = CO_ADD(y00, x11); \
    t04 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(11), q2); \
    rsd += fabs(YO(11) - fnew); \
    CO_TAIL(11); \
    CO_GIVE(3, 11); \
    fnew = CO_FMA(sor2, YO(12), q0); \
    rsd += fabs(YO(12) - fnew); \
    CO_TAIL(12); \
    CO_GIVE(4, 12); \
    CO_ARRIVE_Y(1); \
    CO_PF(1, 15); \
    CO_PF(2, 16); \
    n1 = (CO_FMA(DTW(13), CO_FMA(YO(12), t03, CO_FMA(YO(11), t02, t04)), RY0(13)) - FNS(6)) * sor1; \
    d1 = CO_FMA(DTW(13), CO_FMA(YO(11), t00, t01), rho - FSS(6)); \
    q1 = CO_QUOT(n1, d1); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x10, y10); \
    CO_TAKE(9, x11, y11); \
    t10 = y11; \
    t11 = CO_ADD(y00, x11); \
    t12 = y10; \
    t13 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(13), q1); \
    rsd += fabs(YO(13) - fnew); \
    CO_TAIL(13); \
    CO_GIVE(0, 13); \
    CO_ARRIVE_Y(0); \
    CO_PF(3, 17); \
    CO_PF(4, 18); \
    n2 = (CO_FMA(DTW(14), CO_FMA(YO(13), t12, t13), RY0(14)) - FNS(0)) * sor1; \
    d2 = CO_FMA(DTW(14), CO_FMA(YO(13), t10, t11), rho - FSS(0)); \
    q2 = CO_QUOT(n2, d2); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x10, y10); \
    CO_TAKE(3, x11, y11); \
    CO_TAKE(4, x12, y12); \
    t00 = CO_ADD(y00, x11); \
    t01 = y10; \
    t02 = CO_ADD(x00, x10); \
    t03 = CO_ADD(y01, y12); \
    t04 = x12; \
    t05 = CO_ADD(x01, y11); \
    fnew = CO_FMA(sor2, YO(14), q2); \
    rsd += fabs(YO(14) - fnew); \
    CO_TAIL(14); \
    CO_GIVE(3, 14); \
    CO_ARRIVE_Y(1); \
    CO_PF(5, 19); \
    CO_PF(6, 20); \
    CO_PF(0, 21); \
    n0 = (CO_FMA(DTW(15), CO_FMA(YO(14), t01, t02), RY0(15)) - FNS(1)) * sor1; \
    d0 = CO_FMA(DTW(15), t00, rho - FSS(1)); \
    n1 = (CO_FMA(DTW(16), CO_FMA(YO(14), t04, t05), RY0(16)) - FNS(2)) * sor1; \
    d1 = CO_FMA(DTW(16), t03, rho - FSS(2)); \
    q0 = CO_QUOT(n0, d0); \
    q1 = CO_QUOT(n1, d1); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x01, y01); \
    CO_TAKE(9, x02, y02); \
    CO_TAKE(10, x10, y10); \
    CO_TAKE(11, x11, y11); \
    CO_TAKE(12, x12, y12); \
    t10 = CO_ADD(y00, x11); \
    t11 = y10; \
    t12 = CO_ADD(x00, x10); \
    t13 = x02; \
    t14 = CO_ADD(y01, y12); \
    t15 = x12; \
    t16 = CO_ADD(x01, y11); \
    fnew = CO_FMA(sor2, YO(15), q0); \
    rsd += fabs(YO(15) - fnew); \
    CO_TAIL(15); \
    CO_GIVE(0, 15); \
    fnew = CO_FMA(sor2, YO(16), q1); \
    rsd += fabs(YO(16) - fnew); \
    CO_TAIL(16); \
    CO_GIVE(1, 16); \
    CO_ARRIVE_Y(0); \
    CO_PF(1, 22); \
    n2 = (CO_FMA(DTW(17), CO_FMA(YO(15), t11, t12), RY0(17)) - FNS(3)) * sor1; \
    d2 = CO_FMA(DTW(17), t10, rho - FSS(3)); \
    n0 = (CO_FMA(DTW(18), CO_FMA(YO(16), t15, t16), RY0(18)) - FNS(4)) * sor1; \
    d0 = CO_FMA(DTW(18), CO_FMA(YO(16), t13, t14), rho - FSS(4)); \
    q2 = CO_QUOT(n2, d2); \
    q0 = CO_QUOT(n0, d0); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x02, y02); \
    CO_TAKE(3, x10, y10); \
    CO_TAKE(4, x11, y11); \
    CO_TAKE(5, x12, y12); \
    CO_TAKE(6, x13, y13); \
    t00 = CO_ADD(y00, x11); \
    t01 = CO_ADD(x00, y10); \
    t02 = x10; \
    t03 = CO_ADD(y01, x12); \
    t04 = CO_ADD(x01, y11); \
    t05 = CO_ADD(y02, x13); \
    t06 = CO_ADD(x02, y12); \
    fnew = CO_FMA(sor2, YO(17), q2); \
    rsd += fabs(YO(17) - fnew); \
    CO_TAIL(17); \
    CO_GIVE(3, 17); \
    fnew = CO_FMA(sor2, YO(18), q0); \
    rsd += fabs(YO(18) - fnew); \
    CO_TAIL(18); \
    CO_GIVE(4, 18); \
    CO_ARRIVE_Y(1); \
    CO_PF(2, 23); \
    CO_PF(3, 24); \
    n1 = (CO_FMA(DTW(19), CO_FMA(YO(18), t01, t02), RY0(19)) - FNS(5)) * sor1; \
    d1 = CO_FMA(DTW(19), t00, rho - FSS(5)); \
    n2 = (CO_FMA(DTW(20), t04, RY0(20)) - FNS(6)) * sor1; \
    d2 = CO_FMA(DTW(20), t03, rho - FSS(6)); \
    n0 = (CO_FMA(DTW(21), t06, RY0(21)) - FNS(0)) * sor1; \
    d0 = CO_FMA(DTW(21), CO_ADD(t05, SOUR(0)), rho - FSS(0)); \
    q1 = CO_QUOT(n1, d1); \
    q2 = CO_QUOT(n2, d2); \
    q0 = CO_QUOT(n0, d0); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x01, y01); \
    CO_TAKE(9, x10, y10); \
    CO_TAKE(10, x11, y11); \
    t10 = x01; \
    t11 = CO_ADD(y00, x11); \
    t12 = y10; \
    t13 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(19), q1); \
    rsd += fabs(YO(19) - fnew); \
    CO_TAIL(19); \
    CO_GIVE(0, 19); \
    fnew = CO_FMA(sor2, YO(20), q2); \
    rsd += fabs(YO(20) - fnew); \
    CO_TAIL(20); \
    CO_GIVE(1, 20); \
    fnew = CO_FMA(sor2, YO(21), q0); \
    rsd += fabs(YO(21) - fnew); \
    CO_TAIL(21); \
    CO_GIVE(2, 21); \
    CO_ARRIVE_Y(0); \
    CO_PF(4, 25); \
    n1 = (CO_FMA(DTW(22), CO_FMA(YO(21), t12, t13), RY0(22)) - FNS(1)) * sor1; \
    d1 = CO_FMA(DTW(22), CO_FMA(YO(21), t10, t11), rho - FSS(1)); \
    q1 = CO_QUOT(n1, d1); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x10, y10); \
    CO_TAKE(3, x11, y11); \
    CO_TAKE(4, x12, y12); \
    t00 = CO_ADD(y00, x11); \
    t01 = y10; \
    t02 = CO_ADD(x00, x10); \
    t03 = CO_ADD(y01, x12); \
    t04 = CO_ADD(x01, y11); \
    fnew = CO_FMA(sor2, YO(22), q1); \
    rsd += fabs(YO(22) - fnew); \
    CO_TAIL(22); \
    CO_GIVE(3, 22); \
    CO_ARRIVE_Y(1); \
    CO_PF(5, 26); \
    n2 = (CO_FMA(DTW(23), CO_FMA(YO(22), t01, t02), RY0(23)) - FNS(2)) * sor1; \
    d2 = CO_FMA(DTW(23), t00, rho - FSS(2)); \
    n0 = (CO_FMA(DTW(24), t04, RY0(24)) - FNS(3)) * sor1; \
    d0 = CO_FMA(DTW(24), t03, rho - FSS(3)); \
    q2 = CO_QUOT(n2, d2); \
    q0 = CO_QUOT(n0, d0); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x01, y01); \
    CO_TAKE(9, x10, y10); \
    CO_TAKE(10, x11, y11); \
    t10 = CO_ADD(x01, x11); \
    t11 = CO_ADD(y00, y10); \
    t12 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(23), q2); \
    rsd += fabs(YO(23) - fnew); \
    CO_TAIL(23); \
    CO_GIVE(0, 23); \
    fnew = CO_FMA(sor2, YO(24), q0); \
    rsd += fabs(YO(24) - fnew); \
    CO_TAIL(24); \
    CO_GIVE(1, 24); \
    CO_ARRIVE_Y(0); \
    CO_PF(6, 27); \
    CO_PF(0, 28); \
    n1 = (CO_FMA(DTW(25), CO_FMA(YO(23), t11, t12), RY0(25)) - FNS(4)) * sor1; \
    d1 = CO_FMA(DTW(25), t10, rho - FSS(4)); \
    q1 = CO_QUOT(n1, d1); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x10, y10); \
    t00 = CO_ADD(x01, y10); \
    t01 = y00; \
    t02 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(25), q1); \
    rsd += fabs(YO(25) - fnew); \
    CO_TAIL(25); \
    CO_GIVE(3, 25); \
    CO_ARRIVE_Y(1); \
    CO_PF(1, 29); \
    CO_PF(2, 30); \
    n2 = (CO_FMA(DTW(26), CO_FMA(YO(25), t01, t02), RY0(26)) - FNS(5)) * sor1; \
    d2 = CO_FMA(DTW(26), t00, rho - FSS(5)); \
    q2 = CO_QUOT(n2, d2); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x01, y01); \
    CO_TAKE(9, x02, y02); \
    CO_TAKE(10, x10, y10); \
    CO_TAKE(11, x11, y11); \
    t10 = CO_ADD(x01, y10); \
    t11 = y00; \
    t12 = CO_ADD(x00, x10); \
    t13 = CO_ADD(x02, y11); \
    t14 = CO_ADD(y01, x11); \
    fnew = CO_FMA(sor2, YO(26), q2); \
    rsd += fabs(YO(26) - fnew); \
    CO_TAIL(26); \
    CO_GIVE(0, 26); \
    CO_ARRIVE_Y(0); \
    CO_PF(3, 31); \
    n0 = (CO_FMA(DTW(27), CO_FMA(YO(26), t11, t12), RY0(27)) - FNS(6)) * sor1; \
    d0 = CO_FMA(DTW(27), t10, rho - FSS(6)); \
    n1 = (CO_FMA(DTW(28), t14, RY0(28)) - FNS(0)) * sor1; \
    d1 = CO_FMA(DTW(28), t13, rho - FSS(0)); \
    q0 = CO_QUOT(n0, d0); \
    q1 = CO_QUOT(n1, d1); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x02, y02); \
    CO_TAKE(3, x10, y10); \
    CO_TAKE(4, x11, y11); \
    CO_TAKE(5, x12, y12); \
    t00 = CO_ADD(x01, x11); \
    t01 = CO_ADD(y00, y10); \
    t02 = CO_ADD(x00, x10); \
    t03 = CO_ADD(x02, y12); \
    t04 = x12; \
    t05 = CO_ADD(y01, y11); \
    fnew = CO_FMA(sor2, YO(27), q0); \
    rsd += fabs(YO(27) - fnew); \
    CO_TAIL(27); \
    CO_GIVE(3, 27); \
    fnew = CO_FMA(sor2, YO(28), q1); \
    rsd += fabs(YO(28) - fnew); \
    CO_TAIL(28); \
    CO_GIVE(4, 28); \
    CO_ARRIVE_Y(1); \
    CO_PF(4, 32); \
    CO_PF(5, 33); \
    n2 = (CO_FMA(DTW(29), CO_FMA(YO(28), t01, t02), RY0(29)) - FNS(1)) * sor1; \
    d2 = CO_FMA(DTW(29), t00, rho - FSS(1)); \
    n0 = (CO_FMA(DTW(30), CO_FMA(YO(28), t04, t05), RY0(30)) - FNS(2)) * sor1; \
    d0 = CO_FMA(DTW(30), t03, rho - FSS(2)); \
    q2 = CO_QUOT(n2, d2); \
    q0 = CO_QUOT(n0, d0); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x10, y10); \
    t10 = CO_ADD(y00, y10); \
    t11 = CO_ADD(x00, x10); \
    fnew = CO_FMA(sor2, YO(29), q2); \
    rsd += fabs(YO(29) - fnew); \
    CO_TAIL(29); \
    CO_GIVE(0, 29); \
    fnew = CO_FMA(sor2, YO(30), q0); \
    rsd += fabs(YO(30) - fnew); \
    CO_TAIL(30); \
    CO_GIVE(1, 30); \
    CO_ARRIVE_Y(0); \
    CO_PF(6, 34); \
    CO_PF(0, 35); \
    CO_PF(1, 36); \
    n1 = (CO_FMA(DTW(31), t11, RY0(31)) - FNS(3)) * sor1; \
    d1 = CO_FMA(DTW(31), t10, rho - FSS(3)); \
    q1 = CO_QUOT(n1, d1); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x10, y10); \
    CO_TAKE(3, x11, y11); \
    t00 = CO_ADD(x01, y10); \
    t01 = y00; \
    t02 = CO_ADD(x00, x10); \
    t03 = y11; \
    t04 = x11; \
    fnew = CO_FMA(sor2, YO(31), q1); \
    rsd += fabs(YO(31) - fnew); \
    CO_TAIL(31); \
    CO_GIVE(3, 31); \
    CO_ARRIVE_Y(1); \
    CO_PF(2, 37); \
    CO_PF(3, 38); \
    n2 = (CO_FMA(DTW(32), CO_FMA(YO(31), t01, t02), RY0(32)) - FNS(4)) * sor1; \
    d2 = CO_FMA(DTW(32), t00, rho - FSS(4)); \
    n0 = (CO_FMA(DTW(33), t04, RY0(33)) - FNS(5)) * sor1; \
    d0 = CO_FMA(DTW(33), t03, rho - FSS(5)); \
    q2 = CO_QUOT(n2, d2); \
    q0 = CO_QUOT(n0, d0); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x01, y01); \
    CO_TAKE(9, x02, y02); \
    CO_TAKE(10, x10, y10); \
    CO_TAKE(11, x11, y11); \
    CO_TAKE(12, x12, y12); \
    t10 = CO_ADD(y00, y10); \
    t11 = CO_ADD(x00, x10); \
    t12 = CO_ADD(y01, y11); \
    t13 = CO_ADD(x01, x11); \
    t14 = CO_ADD(y02, y12); \
    t15 = CO_ADD(x02, x12); \
    fnew = CO_FMA(sor2, YO(32), q2); \
    rsd += fabs(YO(32) - fnew); \
    CO_TAIL(32); \
    CO_GIVE(0, 32); \
    fnew = CO_FMA(sor2, YO(33), q0); \
    rsd += fabs(YO(33) - fnew); \
    CO_TAIL(33); \
    CO_GIVE(1, 33); \
    CO_ARRIVE_Y(0); \
    CO_PF(4, 39); \
    CO_PF(5, 40); \
    n1 = (CO_FMA(DTW(34), t11, RY0(34)) - FNS(6)) * sor1; \
    d1 = CO_FMA(DTW(34), t10, rho - FSS(6)); \
    n2 = (CO_FMA(DTW(35), t13, RY0(35)) - FNS(0)) * sor1; \
    d2 = CO_FMA(DTW(35), t12, rho - FSS(0)); \
    n0 = (CO_FMA(DTW(36), t15, RY0(36)) - FNS(1)) * sor1; \
    d0 = CO_FMA(DTW(36), t14, rho - FSS(1)); \
    q1 = CO_QUOT(n1, d1); \
    q2 = CO_QUOT(n2, d2); \
    q0 = CO_QUOT(n0, d0); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x10, y10); \
    CO_TAKE(3, x11, y11); \
    CO_TAKE(4, x12, y12); \
    t00 = x11; \
    t01 = y10; \
    t02 = x10; \
    t03 = CO_ADD(x01, y12); \
    t04 = CO_ADD(y00, x12); \
    t05 = CO_ADD(x00, y11); \
    fnew = CO_FMA(sor2, YO(34), q1); \
    rsd += fabs(YO(34) - fnew); \
    CO_TAIL(34); \
    CO_GIVE(3, 34); \
    fnew = CO_FMA(sor2, YO(35), q2); \
    rsd += fabs(YO(35) - fnew); \
    CO_TAIL(35); \
    CO_GIVE(4, 35); \
    fnew = CO_FMA(sor2, YO(36), q0); \
    rsd += fabs(YO(36) - fnew); \
    CO_TAIL(36); \
    CO_GIVE(5, 36); \
    CO_ARRIVE_Y(1); \
    CO_PF(6, 41); \
    n1 = (CO_FMA(DTW(37), CO_FMA(YO(36), t01, t02), RY0(37)) - FNS(2)) * sor1; \
    d1 = CO_FMA(DTW(37), t00, rho - FSS(2)); \
    n2 = (CO_FMA(DTW(38), CO_FMA(YO(36), t04, t05), RY0(38)) - FNS(3)) * sor1; \
    d2 = CO_FMA(DTW(38), t03, rho - FSS(3)); \
    q1 = CO_QUOT(n1, d1); \
    q2 = CO_QUOT(n2, d2); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x01, y01); \
    CO_TAKE(9, x02, y02); \
    CO_TAKE(10, x10, y10); \
    CO_TAKE(11, x11, y11); \
    t10 = CO_ADD(x01, y10); \
    t11 = y00; \
    t12 = CO_ADD(x00, x10); \
    t13 = CO_ADD(x02, y11); \
    t14 = CO_ADD(y01, x11); \
    fnew = CO_FMA(sor2, YO(37), q1); \
    rsd += fabs(YO(37) - fnew); \
    CO_TAIL(37); \
    CO_GIVE(0, 37); \
    fnew = CO_FMA(sor2, YO(38), q2); \
    rsd += fabs(YO(38) - fnew); \
    CO_TAIL(38); \
    CO_GIVE(1, 38); \
    CO_ARRIVE_Y(0); \
    CO_PF(0, 42); \
    CO_PF(1, 43); \
    n0 = (CO_FMA(DTW(39), CO_FMA(YO(38), t11, t12), RY0(39)) - FNS(4)) * sor1; \
    d0 = CO_FMA(DTW(39), t10, rho - FSS(4)); \
    n1 = (CO_FMA(DTW(40), t14, RY0(40)) - FNS(5)) * sor1; \
    d1 = CO_FMA(DTW(40), t13, rho - FSS(5)); \
    q0 = CO_QUOT(n0, d0); \
    q1 = CO_QUOT(n1, d1); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x10, y10); \
    t00 = CO_ADD(x01, y10); \
    t01 = y00; \
    t02 = x10; \
    t03 = x00; \
    fnew = CO_FMA(sor2, YO(39), q0); \
    rsd += fabs(YO(39) - fnew); \
    CO_TAIL(39); \
    CO_GIVE(3, 39); \
    fnew = CO_FMA(sor2, YO(40), q1); \
    rsd += fabs(YO(40) - fnew); \
    CO_TAIL(40); \
    CO_GIVE(4, 40); \
    CO_ARRIVE_Y(1); \
    CO_PF(2, 44); \
    CO_PF(3, 45); \
    CO_PF(4, 46); \
    n2 = (CO_FMA(DTW(41), CO_FMA(YO(40), t02, CO_FMA(YO(39), t01, t03)), RY0(41)) - FNS(6)) * sor1; \
    d2 = CO_FMA(DTW(41), t00, rho - FSS(6)); \
    q2 = CO_QUOT(n2, d2); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x01, y01); \
    CO_TAKE(9, x10, y10); \
    CO_TAKE(10, x11, y11); \
    CO_TAKE(11, x12, y12); \
    t10 = CO_ADD(y00, x11); \
    t11 = y10; \
    t12 = CO_ADD(x00, x10); \
    t13 = CO_ADD(y01, x12); \
    t14 = CO_ADD(x01, y11); \
    fnew = CO_FMA(sor2, YO(41), q2); \
    rsd += fabs(YO(41) - fnew); \
    CO_TAIL(41); \
    CO_GIVE(0, 41); \
    CO_ARRIVE_Y(0); \
    CO_PF(5, 47); \
    CO_PF(6, 48); \
    n0 = (CO_FMA(DTW(42), CO_FMA(YO(41), t11, t12), RY0(42)) - FNS(0)) * sor1; \
    d0 = CO_FMA(DTW(42), t10, rho - FSS(0)); \
    n1 = (CO_FMA(DTW(43), t14, RY0(43)) - FNS(1)) * sor1; \
    d1 = CO_FMA(DTW(43), t13, rho - FSS(1)); \
    q0 = CO_QUOT(n0, d0); \
    q1 = CO_QUOT(n1, d1); \
    CO_WAIT_P(0); \
    CO_TAKE(0, x00, y00); \
    CO_TAKE(1, x01, y01); \
    CO_TAKE(2, x10, y10); \
    CO_TAKE(3, x11, y11); \
    CO_TAKE(4, x12, y12); \
    t00 = y10; \
    t01 = x10; \
    t02 = CO_ADD(y00, y11); \
    t03 = CO_ADD(x00, x11); \
    t04 = CO_ADD(y01, x12); \
    t05 = x01; \
    fnew = CO_FMA(sor2, YO(42), q0); \
    rsd += fabs(YO(42) - fnew); \
    CO_TAIL(42); \
    CO_GIVE(3, 42); \
    fnew = CO_FMA(sor2, YO(43), q1); \
    rsd += fabs(YO(43) - fnew); \
    CO_TAIL(43); \
    CO_GIVE(4, 43); \
    CO_ARRIVE_Y(1); \
    CO_PF(0, 49); \
    CO_PF(1, 50); \
    n2 = (CO_FMA(DTW(44), CO_MUL(YO(43), t01), RY0(44)) - FNS(2)) * sor1; \
    d2 = CO_FMA(DTW(44), t00, rho - FSS(2)); \
    n0 = (CO_FMA(DTW(45), t03, RY0(45)) - FNS(3)) * sor1; \
    d0 = CO_FMA(DTW(45), t02, rho - FSS(3)); \
    n1 = (CO_FMA(DTW(46), t05, RY0(46)) - FNS(4)) * sor1; \
    d1 = CO_FMA(DTW(46), t04, rho - FSS(4)); \
    q2 = CO_QUOT(n2, d2); \
    q0 = CO_QUOT(n0, d0); \
    q1 = CO_QUOT(n1, d1); \
    CO_WAIT_P(1); \
    CO_TAKE(7, x00, y00); \
    CO_TAKE(8, x01, y01); \
    CO_TAKE(9, x10, y10); \
    CO_TAKE(10, x11, y11); \
    CO_TAKE(11, x12, y12); \
    t10 = CO_ADD(y00, x11); \
    t11 = y10; \
    t12 = CO_ADD(x00, x10); \
    t13 = CO_ADD(y01, y12); \
    t14 = x12; \
    t15 = CO_ADD(x01, y11); \
    fnew = CO_FMA(sor2, YO(44), q2); \
    rsd += fabs(YO(44) - fnew); \
    CO_TAIL(44); \
    CO_GIVE(0, 44); \
    fnew = CO_FMA(sor2, YO(45), q0); \
    rsd += fabs(YO(45) - fnew); \
    CO_TAIL(45); \
    CO_GIVE(1, 45); \
    fnew = CO_FMA(sor2, YO(46), q1); \
    rsd += fabs(YO(46) - fnew); \
    CO_TAIL(46); \
    CO_GIVE(2, 46); \
    CO_ARRIVE_Y(0); \
    n2 = (CO_FMA(DTW(47), CO_FMA(YO(46), t11, t12), RY0(47)) - FNS(5)) * sor1; \
    d2 = CO_FMA(DTW(47), t10, rho - FSS(5)); \
    rest = CO_FMA(YO(46), t14, t15); \
    n0 = (CO_FMA(DTW(48), rest, RY0(48)) - FNS(6)) * sor1; \
    d0 = CO_FMA(DTW(48), t13, rho - FSS(6)); \
    q2 = CO_QUOT(n2, d2); \
    q0 = CO_QUOT(n0, d0); \
    fnew = CO_FMA(sor2, YO(47), q2); \
    rsd += fabs(YO(47) - fnew); \
    CO_TAIL(47); \
    CO_GIVE(3, 47); \
    fnew = CO_FMA(sor2, YO(48), q0); \
    rsd += fabs(YO(48) - fnew); \
    CO_TAIL(48); \
    CO_GIVE(4, 48); \
    CO_ARRIVE_Y(1); \
    n1 = (CO_FMA(DTW(49), rest, RY0(49)) - FNS(0)) * sor1; \
    d1 = rho - FSS(0); \
    q1 = CO_QUOT(n1, d1); \
    fnew = CO_FMA(sor2, YO(49), q1); \
    rsd += fabs(YO(49) - fnew); \
    CO_TAIL(49); \
    n2 = (CO_FMA(DTW(50), rest, RY0(50)) - FNS(1)) * sor1; \
    d2 = rho - FSS(1); \
    q2 = CO_QUOT(n2, d2); \
    fnew = CO_FMA(sor2, YO(50), q2); \
    rsd += fabs(YO(50) - fnew); \
    CO_TAIL(50); \
} while (0)
#ifdef __CUDACC__
static __constant__ int16_t uc_co_pairs_0[40] = {6, 8, 19, 23, 26, 27, 30, 35, 37, 40, 41, 49, 56, 58, 60, 61, 64, 69, 72, 76, 94, 102, 103, 106, 107, 109, 116, 118, 120, 122, 124, 129, 130, 138, 141, 142, 143, 150, 155, 157};
static __constant__ int16_t uc_co_cols_0[40] = {24, 72, 8, 16, 80, 152, 88, 32, 92, 36, 128, 20, 48, 96, 136, 56, 60, 52, 0, 100, 132, 104, 140, 12, 64, 84, 108, 28, 112, 144, 40, 4, 44, 156, 116, 68, 76, 148, 120, 124};
static __constant__ int16_t uc_co_pairs_1[128] = {0, 1, 2, 3, 4, 5, 7, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18, 20, 21, 22, 24, 25, 28, 29, 31, 32, 33, 34, 36, 38, 39, 42, 43, 44, 45, 46, 47, 48, 50, 51, 52, 53, 54, 55, 57, 59, 62, 63, 65, 66, 67, 68, 70, 71, 73, 74, 75, 77, 78, 79, 80, 81, 82, 83, 84, 85, 86, 87, 88, 89, 90, 91, 92, 93, 95, 96, 97, 98, 99, 100, 101, 104, 105, 108, 110, 111, 112, 113, 114, 115, 117, 119, 121, 123, 125, 126, 127, 128, 131, 132, 133, 134, 135, 136, 137, 139, 140, 144, 145, 146, 147, 148, 149, 151, 152, 153, 154, 156, 158, 159, 160, 161, 162, 163, 164, 165, 166, 167};
static __constant__ int16_t uc_co_cols_1[128] = {32, 0, 4, 232, 208, 48, 52, 212, 40, 240, 64, 88, 236, 400, 248, 256, 36, 260, 44, 80, 216, 264, 24, 252, 220, 268, 272, 96, 100, 280, 276, 288, 112, 296, 68, 304, 84, 312, 408, 308, 56, 136, 320, 316, 480, 324, 328, 412, 416, 72, 336, 344, 116, 348, 424, 484, 428, 128, 300, 284, 140, 132, 120, 352, 488, 356, 432, 124, 360, 292, 76, 364, 244, 92, 436, 420, 144, 152, 340, 492, 148, 156, 440, 332, 444, 448, 368, 224, 372, 228, 376, 380, 384, 388, 452, 496, 404, 160, 456, 164, 168, 172, 460, 60, 104, 108, 500, 176, 464, 468, 200, 28, 184, 180, 392, 188, 504, 396, 204, 472, 476, 16, 20, 192, 8, 12, 196, 508};
#else
static const short uc_co_pairs_0[40] = {6, 8, 19, 23, 26, 27, 30, 35, 37, 40, 41, 49, 56, 58, 60, 61, 64, 69, 72, 76, 94, 102, 103, 106, 107, 109, 116, 118, 120, 122, 124, 129, 130, 138, 141, 142, 143, 150, 155, 157};
static const short uc_co_cols_0[40] = {24, 72, 8, 16, 80, 152, 88, 32, 92, 36, 128, 20, 48, 96, 136, 56, 60, 52, 0, 100, 132, 104, 140, 12, 64, 84, 108, 28, 112, 144, 40, 4, 44, 156, 116, 68, 76, 148, 120, 124};
static const short uc_co_pairs_1[128] = {0, 1, 2, 3, 4, 5, 7, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18, 20, 21, 22, 24, 25, 28, 29, 31, 32, 33, 34, 36, 38, 39, 42, 43, 44, 45, 46, 47, 48, 50, 51, 52, 53, 54, 55, 57, 59, 62, 63, 65, 66, 67, 68, 70, 71, 73, 74, 75, 77, 78, 79, 80, 81, 82, 83, 84, 85, 86, 87, 88, 89, 90, 91, 92, 93, 95, 96, 97, 98, 99, 100, 101, 104, 105, 108, 110, 111, 112, 113, 114, 115, 117, 119, 121, 123, 125, 126, 127, 128, 131, 132, 133, 134, 135, 136, 137, 139, 140, 144, 145, 146, 147, 148, 149, 151, 152, 153, 154, 156, 158, 159, 160, 161, 162, 163, 164, 165, 166, 167};
static const short uc_co_cols_1[128] = {32, 0, 4, 232, 208, 48, 52, 212, 40, 240, 64, 88, 236, 400, 248, 256, 36, 260, 44, 80, 216, 264, 24, 252, 220, 268, 272, 96, 100, 280, 276, 288, 112, 296, 68, 304, 84, 312, 408, 308, 56, 136, 320, 316, 480, 324, 328, 412, 416, 72, 336, 344, 116, 348, 424, 484, 428, 128, 300, 284, 140, 132, 120, 352, 488, 356, 432, 124, 360, 292, 76, 364, 244, 92, 436, 420, 144, 152, 340, 492, 148, 156, 440, 332, 444, 448, 368, 224, 372, 228, 376, 380, 384, 388, 452, 496, 404, 160, 456, 164, 168, 172, 460, 60, 104, 108, 500, 176, 464, 468, 200, 28, 184, 180, 392, 188, 504, 396, 204, 472, 476, 16, 20, 192, 8, 12, 196, 508};
#endif
