// What the prepared tables of the rate kernels hold, and that the mechanism's data fits: regenerated data that
// does not ends the build here instead of giving wrong rates.
#pragma once
#include "generated/mech_tables.h"

constexpr int FALL_MAX = 24;             // entries of the fall-off table
constexpr int KC_MIN = 3, KC_MAX = 6;    // factors of an equilibrium constant (the kernel multiplies three at least)
constexpr int RC_Y_MAX = 1;              // mass fractions that are factors of one RC slot
constexpr int RC_POST_MAX = 4, TB_MAX = 10;
constexpr int RATE_WARPS = 16;           // warps of the rate kernel
constexpr int WARP_ITEMS = 25;           // reaction pairs (or the soot sources) of one of them

static_assert(UC_FALLOFF <= FALL_MAX, "more fall-off pairs than the table holds");
static_assert(UC_QMIN >= KC_MIN && UC_QMAX <= KC_MAX, "an equilibrium constant with too few or too many factors");
static_assert(UC_RC_YMAX <= RC_Y_MAX, "an RC slot with more than one mass fraction as a factor");
static_assert(UC_PMAX <= RC_POST_MAX, "an RC slot with more factors than its record holds");
static_assert(UC_NTB <= TB_MAX, "more third-body groups than the tile has rows for");
static_assert(UC_NPAIR + 1 <= RATE_WARPS * WARP_ITEMS, "more reaction pairs than the warps' lists hold");
