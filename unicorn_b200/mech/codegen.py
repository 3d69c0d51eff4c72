"""Generate the device-side mechanism tables and the species-update program.

Build-time tool: reads ``sandiego52.json`` (written by ``extract.py``) and
writes ``unicorn_b200/csrc/generated/mech_tables.h`` and
``unicorn_b200/csrc/generated/update_program.cuh``.

The species update of the reference (``src/lib/solvesp.f:85-2806``) keeps
544 scalar "A-terms" per cell that are recomputed with one species factored
out, multiplied by the freshly updated mass fraction, and reused by later
species. On a GPU, 544 doubles per cell do not fit on chip, so the generator
executes that statement sequence symbolically: every A-term becomes an
expression tree over three kinds of leaves, RC(r), Y_j as it was at the
start of the pass (``yo``) and Y_j after its own update in this pass
(``yn``). Each production and loss term of each species is then emitted as
that tree, with the reference's operand order, so the device code needs only
RC, the old and the new Y of the cell.
"""
from __future__ import annotations

import json
from pathlib import Path

LSP, LRX = 52, 544
HERE = Path(__file__).resolve().parent
MECH = HERE / "sandiego52.json"
GEN = HERE.parent / "csrc" / "generated"


# ------------------------------------------------------------------ symbolic update

class Leaf:
    __slots__ = ("kind", "idx", "val")

    def __init__(self, kind, idx=0, val=0.0):
        self.kind, self.idx, self.val = kind, idx, val

    def c(self, ctx) -> str:
        if self.kind == "RC":
            return ctx.rc(self.idx)
        if self.kind == "yo":
            return ctx.yo(self.idx) if hasattr(ctx, "yo") else f"YO({self.idx})"
        if self.kind == "yn":
            return f"YN({self.idx})"
        if self.kind == "y0":
            return f"Y0({self.idx})"
        if self.kind == "SOUR":
            return f"SOUR({self.idx})"
        if self.kind == "num":
            return repr(float(self.val))
        raise ValueError(self.kind)


class Mul:
    __slots__ = ("a", "b")

    def __init__(self, a, b):
        self.a, self.b = a, b

    def c(self, ctx) -> str:
        return f"({self.a.c(ctx)} * {self.b.c(ctx)})"


def leaves(e, out):
    if isinstance(e, Mul):
        leaves(e.a, out)
        leaves(e.b, out)
    else:
        out.append(e)
    return out


def resolve_update(mech: dict) -> list[dict]:
    """Symbolic execution of the per-cell update program.

    Returns one dict per species block k (0-based) with expression trees for
    the production sum (list of (sign, tree) or None = reuse the previous
    block's value), the extra sum, and the loss sum (None = 0)."""
    A: dict[int, object] = {}
    updated: set[int] = set()

    def yleaf(k0):
        return Leaf("yn" if k0 in updated else "yo", k0)

    def chain_tree(factors):
        t = None
        for f in factors:
            kind = f[0]
            if kind == "num":
                x = Leaf("num", val=f[1])
            elif kind == "Y":
                x = yleaf(f[1] - 1)
            elif kind == "Y0":
                x = Leaf("y0", f[1] - 1)
            elif kind == "RC":
                x = Leaf("RC", f[1] - 1)
            elif kind == "SOUR":
                x = Leaf("SOUR", f[1] - 1)
            elif kind == "A":
                x = A[f[1]]
            else:
                raise ValueError(kind)
            t = x if t is None else Mul(t, x)
        return t

    out = []
    for b in mech["update"]["blocks"]:
        k0 = b["species"] - 1
        for r, fac in b["recompute"]:
            A[r] = chain_tree(fac)
        blk = {"species": k0}
        blk["prod"] = None if b["prod"] is None else [(s, chain_tree(f)) for s, f in b["prod"]]
        blk["extra"] = [(s, chain_tree(f)) for s, f in b["extra"]]
        blk["loss"] = None if b["loss"] is None else [(s, chain_tree(f)) for s, f in b["loss"]]
        out.append(blk)
        updated.add(k0)
        for r in b["multiply"]:
            A[r] = Mul(Leaf("yn", k0), A[r])
    return out


def emit_sum(terms, ctx, acc: str) -> list[str]:
    lines = []
    for i, (s, t) in enumerate(terms):
        v = t.c(ctx)
        if i == 0:
            lines.append(f"{acc} = {'' if s > 0 else '-'}{v};")
        else:
            lines.append(f"{acc} = {acc} {'+' if s > 0 else '-'} {v};")
    return lines


class _Ctx:
    """Emission context: the last use of each RC(r) in a pass is emitted as
    RC_LAST(r), so the device code can tell L2 that the line will not be
    needed again this pass."""

    def __init__(self, last_use: dict | None = None):
        self.last_use = last_use or {}
        self.count: dict[int, int] = {}

    def rc(self, r0: int) -> str:
        self.count[r0] = self.count.get(r0, 0) + 1
        if self.last_use.get(r0) == self.count[r0]:
            return f"RC_LAST({r0})"
        return f"RC({r0})"


def gen_update_program(mech: dict) -> str:
    blocks = resolve_update(mech)
    uses: dict[int, int] = {}
    for b in blocks:
        for key in ("prod", "extra", "loss"):
            for _, t in (b[key] or []):
                for leaf in leaves(t, []):
                    if leaf.kind == "RC":
                        uses[leaf.idx] = uses.get(leaf.idx, 0) + 1
    ctx = _Ctx(uses)
    # RC rows each species block reads, in first-use order (for L2 prefetch)
    rows, offs = [], []
    for b in blocks:
        offs.append(len(rows))
        seen = []
        for key in ("prod", "extra", "loss"):
            for _, t in (b[key] or []):
                for leaf in leaves(t, []):
                    if leaf.kind == "RC" and leaf.idx not in seen:
                        seen.append(leaf.idx)
        rows.extend(seen)
    offs.append(len(rows))
    L = ["// Generated by unicorn_b200/mech/codegen.py from the update program of",
         "// src/lib/solvesp.f:85-2806 (one block per species, in the reference's order).",
         "// Requires accessor macros RC(r) (0-based reaction slot; RC_LAST(r) marks its",
         "// last use in a pass), YO(k) (Y at the",
         "// start of the pass), YN(k) (Y after its own update), Y0(k) (old time level),",
         "// SOUR(m), WM(k), FACE_SUM(k), FACE_NBR(k); scalars rho, dt, sor1, sor2, rsd;",
         "// and UC_UPDATE_TAIL(k), which clips fnew and stores it as YN(k);",
         "// UC_UPDATE_SYNC() runs after every species (a barrier, or nothing);",
         "// UC_UPDATE_BLOCK_BEGIN(b) runs before species block b (e.g. to prefetch).",
         "#pragma once",
         "#define UC_UPDATE_PROGRAM() do { \\",
         "    double prod = 0.0, extra, loss, rhs1, rhs2, ppp, fnew; \\"]
    nterms = 0
    for bi, b in enumerate(blocks):
        k = b["species"]
        body = [f"UC_UPDATE_BLOCK_BEGIN({bi});"]
        if b["prod"] is not None:
            body += emit_sum(b["prod"], ctx, "prod")
            nterms += len(b["prod"])
        body += emit_sum(b["extra"], ctx, "extra")
        nterms += len(b["extra"])
        body.append(f"rhs1 = rho * Y0({k}) + dt * WM({k}) * (prod + extra);")
        if b["loss"] is None:
            body.append("rhs2 = 0.0;")
        else:
            body += emit_sum(b["loss"], ctx, "loss")
            nterms += len(b["loss"])
            body.append(f"rhs2 = -(dt * WM({k}) * loss);")
        body.append(f"ppp = rho - FACE_SUM({k});")
        body.append(f"fnew = sor2 * YO({k}) + (rhs1 - FACE_NBR({k})) * sor1 / (ppp - rhs2);")
        body.append(f"rsd += fabs(YO({k}) - fnew);")
        body.append(f"UC_UPDATE_TAIL({k});")
        body.append("UC_UPDATE_SYNC();")
        L.append(f"    /* species {k + 1} */ \\")
        L.extend("    " + x + " \\" for x in body)
    L.append("} while (0)")
    L.insert(6, f"// {nterms} production/extra/loss terms per cell and pass")
    L.append("")
    L.append(f"#define UC_UPD_NBLOCKS {len(blocks)}")
    L.append("#ifdef __CUDACC__")
    L.append("// RC rows read by each species block (first-use order): rows [off[b], off[b+1]).")
    L.append(f"static __device__ const int16_t uc_upd_row_off[{len(offs)}] = {{{', '.join(map(str, offs))}}};")
    L.append(f"static __device__ const int16_t uc_upd_rows[{len(rows)}] = {{{', '.join(map(str, rows))}}};")
    L.append("#endif")
    return "\n".join(L) + "\n\n" + gen_inplace_program(blocks, uses)


# ------------------------------------------------------------------ in-place form

class _InPlaceCtx(_Ctx):
    """Emission context of the in-place program: one Y array per tile, each
    species overwritten by its own update. A species' start-of-pass value read
    after its update (through an A-term built before it) comes from a shadow
    copy YOS(m) the tile keeps for those few species."""

    def __init__(self, last_use: dict):
        super().__init__(last_use)
        self.updated: set[int] = set()
        self.shadow: list[int] = []

    def yo(self, k: int) -> str:
        if k not in self.updated:
            return f"YO({k})"
        if k not in self.shadow:
            self.shadow.append(k)
        return f"YOS({self.shadow.index(k)})"


def gen_inplace_program(blocks, uses: dict) -> str:
    ctx = _InPlaceCtx(uses)
    body = []
    for b in blocks:
        k = b["species"]
        if b["prod"] is not None:
            body += emit_sum(b["prod"], ctx, "prod")
        body += emit_sum(b["extra"], ctx, "extra")
        body.append(f"rhs1 = rho * Y0({k}) + dt * WM({k}) * (prod + extra);")
        if b["loss"] is None:
            body.append("rhs2 = 0.0;")
        else:
            body += emit_sum(b["loss"], ctx, "loss")
            body.append(f"rhs2 = -(dt * WM({k}) * loss);")
        body.append(f"ppp = rho - FACE_SUM({k});")
        body.append(f"fnew = sor2 * YO({k}) + (rhs1 - FACE_NBR({k})) * sor1 / (ppp - rhs2);")
        body.append(f"rsd += fabs(YO({k}) - fnew);")
        body.append(f"UC_UPDATE_TAIL({k});")
        ctx.updated.add(k)
    L = ["// In-place form of the same program: YO(k) and YN(k) name one array; YOS(m)",
         "// is the start-of-pass value of species uc_ip_shadow[m], read after that",
         "// species' own update.",
         f"#define UC_IP_NSHADOW {len(ctx.shadow)}",
         f"#define UC_IP_SHADOW_LIST {{{', '.join(map(str, ctx.shadow or [0]))}}}",
         "#define UC_UPDATE_PROGRAM_IP() do { \\",
         "    double prod = 0.0, extra, loss, rhs1, rhs2, ppp, fnew; \\"]
    L.extend("    " + x + " \\" for x in body)
    L.append("} while (0)")
    L.append("#ifdef __CUDACC__")
    L.append(f"static __constant__ int8_t uc_ip_shadow[{max(1, len(ctx.shadow))}] = UC_IP_SHADOW_LIST;")
    L.append("#endif")
    gen_inplace_program.shadow = list(ctx.shadow)
    return "\n".join(L) + "\n"


# ------------------------------------------------------------------ tile-resident form

TR_NTMEM, TR_SEG = 256, 12


class _TRCtx(_InPlaceCtx):
    """Emission context of the tile-resident program: RC(r) becomes a token
    that is later bound to a shared-memory row or a tensor-memory register."""

    def rc(self, r0: int) -> str:
        return f"@{r0}@"


def gen_tr_program(blocks, uses: dict, shadow: list[int]) -> str:
    """The in-place program for a tile whose RC block lives on chip: the RC rows
    used least often (TR_NTMEM of them) in tensor memory, two 32-bit columns
    each, the others in shared memory. Tensor-memory operands are loaded into
    registers ahead of use in segments of at most TR_SEG values, alternating
    between two register banks: the loads of segment s+1 are issued before the
    statements of segment s run and waited for after them, so their latency is
    hidden behind segment s. The arithmetic, its operands and their order are
    those of the in-place program. The kernels run the grouped form below (gen_co_program); this one, whose
    arithmetic is the two-array program's bit for bit, is run by the host test of the generated programs."""
    import re
    ctx = _TRCtx(uses)
    body = [f"UC_TR_PF(0, {blocks[0]['species']});"]
    for bi, b in enumerate(blocks):
        k = b["species"]
        slot = bi % 2
        if bi + 1 < len(blocks):
            # old time level and face terms of the next species, one block ahead of their use
            body.append(f"UC_TR_PF({(bi + 1) % 2}, {blocks[bi + 1]['species']});")
        # the production, extra and loss sums are independent of each other: their statements are
        # interleaved (each sum keeps its own order) so that two or three chains are in flight
        sums = [emit_sum(b["prod"], ctx, "prod") if b["prod"] is not None else [],
                emit_sum(b["extra"], ctx, "extra"),
                emit_sum(b["loss"], ctx, "loss") if b["loss"] is not None else []]
        for i in range(max(len(x) for x in sums)):
            body += [x[i] for x in sums if i < len(x)]
        body.append(f"rhs1 = rho * Y0S({slot}) + dt * WM({k}) * (prod + extra);")
        body.append("rhs2 = 0.0;" if b["loss"] is None else f"rhs2 = -(dt * WM({k}) * loss);")
        body.append(f"ppp = rho - FSS({slot});")
        body.append(f"fnew = sor2 * YO({k}) + (rhs1 - FNS({slot})) * sor1 / (ppp - rhs2);")
        body.append(f"rsd += fabs(YO({k}) - fnew);")
        body.append(f"UC_UPDATE_TAIL({k});")
        body.append("UC_TR_SYNC();")
        ctx.updated.add(k)
    assert ctx.shadow == shadow, "the tile-resident and in-place programs must shadow the same species"
    tok = re.compile(r"@(\d+)@")
    # by slot number: slots [0, TR_NTMEM) in tensor memory, the rest in shared memory, so that each
    # part is one contiguous range of the RC plane's rows and is staged by a few tiled bulk copies
    trow = list(range(TR_NTMEM))
    srow = list(range(TR_NTMEM, LRX))
    tcol = {r: i for i, r in enumerate(trow)}
    scol = {r: i for i, r in enumerate(srow)}
    # segments: runs of statements with at most TR_SEG distinct tensor-memory rows
    segs = []          # (statements, tensor-memory rows in first-use order)
    cur, cur_rows = [], []
    for st in body:
        need = [int(x) for x in tok.findall(st) if int(x) in tcol]
        new = [r for r in dict.fromkeys(need) if r not in cur_rows]
        if cur and len(cur_rows) + len(new) > TR_SEG:
            segs.append((cur, cur_rows))
            cur, cur_rows = [], []
            new = list(dict.fromkeys(need))
        cur.append(st)
        cur_rows += new
    segs.append((cur, cur_rows))
    out = []

    def loads(si):
        bank = si % 2
        return [f"TM_LD({bank}, {q}, {2 * tcol[r]});" for q, r in enumerate(segs[si][1])]

    out += loads(0)
    out.append("TM_WAIT(0);")
    for si, (stmts, trs) in enumerate(segs):
        bank = si % 2
        slot = {r: q for q, r in enumerate(trs)}
        if si + 1 < len(segs):
            out += loads(si + 1)

        def bind(m, slot=slot, bank=bank):
            r = int(m.group(1))
            return f"RCT({bank}, {slot[r]})" if r in tcol else f"RCS({scol[r]})"
        out += [tok.sub(bind, st) for st in stmts]
        if si + 1 < len(segs):
            out.append(f"TM_WAIT({(si + 1) % 2});")
    nld = sum(len(t) for _, t in segs)

    def muls(t):
        return 1 + muls(t.a) + muls(t.b) if isinstance(t, Mul) else 0
    # floating-point operations per cell and pass: the multiplications of each term and its addition
    # into the sum, and the 16 of each species' closing statements (rhs1 5, rhs2 2, ppp 1, fnew 6 with
    # the division as one, the residual 2); the two soot scalars 19
    flops = sum(muls(t) + 1 for b in blocks for key in ("prod", "extra", "loss") for _, t in (b[key] or [])) + \
        16 * len(blocks) + 19
    L = ["// Generated by unicorn_b200/mech/codegen.py: the in-place species-update program",
         "// (src/lib/solvesp.f:85-2806) for a tile whose RC block is held on chip.",
         "// Run by the host test of the generated programs; the kernels run update_program_co.cuh.",
         f"// RC slots 0..{len(trow) - 1} in tensor memory (slot i in columns 2i, 2i+1: low and high",
         f"// word), slots {len(trow)}..{LRX - 1} in shared memory. Requires RCS(i) (shared-memory row i of the",
         "// cell), TM_LD(bank, q, col) (load the double at column col into slot q of a",
         "// register bank), TM_WAIT(bank) (wait for the loads of that bank), RCT(bank, q),",
         "// UC_TR_PF(slot, k) (fetch Y0, FACE_SUM and FACE_NBR of species k into register slot 0",
         "// or 1; read as Y0S, FSS, FNS), UC_TR_SYNC() (after every species: a barrier or nothing)",
         "// and the accessors of the in-place program (YO, YN, YOS, SOUR, WM, UC_UPDATE_TAIL;",
         "// scalars rho, dt, sor1, sor2, rsd). The production, extra and loss statements of a",
         "// species are interleaved; each sum keeps the reference's order.",
         f"// {len(segs)} segments and {nld} tensor-memory loads per cell and pass.",
         "#pragma once",
         f"#define UC_TR_NT {len(trow)}",
         f"#define UC_TR_NS {len(srow)}",
         f"#define UC_TR_SEG {TR_SEG}",
         f"#define UC_UPDATE_FLOPS_PER_CELL_PASS {flops}",
         "#define UC_TR_SHADOW_SAVE() do { " + " ".join(f"YOS({m}) = YO({k});" for m, k in enumerate(shadow)) + " } while (0)",
         "#define UC_UPDATE_PROGRAM_TR() do { \\",
         "    double prod = 0.0, extra, loss, rhs1, rhs2, ppp, fnew; \\"]
    L.extend("    " + x + " \\" for x in out)
    L.append("} while (0)")
    L.append("#ifdef __CUDACC__")
    L.append(f"static __constant__ int16_t uc_tr_trow[{len(trow)}] = {{{', '.join(map(str, trow))}}};")
    L.append(f"static __constant__ int16_t uc_tr_srow[{len(srow)}] = {{{', '.join(map(str, srow))}}};")
    L.append("#else")
    L.append(f"static const short uc_tr_trow[{len(trow)}] = {{{', '.join(map(str, trow))}}};")
    L.append(f"static const short uc_tr_srow[{len(srow)}] = {{{', '.join(map(str, srow))}}};")
    L.append("#endif")
    return "\n".join(L) + "\n"


# ------------------------------------------------------------------ grouped form, three warps per tile

CO_NT, CO_PIECE = 336, 168       # rows in tensor memory, staged in pieces of CO_PIECE rows
CO_PAIRS = (20, 64)              # row pairs of each piece that each of the summing warps holds
CO_SHARE = (0.40, 0.60)          # of the work (the first ones of an SM's three tiles run on one scheduler)
CO_SUMS = len(CO_PAIRS)
CO_SEG = 4                       # row pairs per register bank of tensor-memory operands
CO_REUSE = 10                    # statements over which a row pair read from shared memory stays in registers
CO_LAST = 48                     # the last species whose sums have terms (argon and helium follow)
CO_LONG = 6                      # terms from which a sum has two accumulators
CO_NEWSUM = 4.0                  # see _share_out
CO_RUN, CO_VALUES = 3, 7         # species closed in one step, and the partial sums a warp hands over for them


def _grouped_sums(blocks):
    """Per species block the terms of (production and extra, loss) as (coefficient, operand, Y leaves): the
    operand is ("RC", r), ("SOUR", m) or None. Terms that are the literal zero are dropped."""
    out = []
    for b in blocks:
        d = []
        for keys in (("prod", "extra"), ("loss",)):
            ts = []
            for key in keys:
                for s, t in b[key] or []:
                    coef, op, ys = float(s), None, []
                    for x in leaves(t, []):
                        if x.kind == "num":
                            coef *= x.val
                        elif x.kind in ("RC", "SOUR"):
                            assert op is None
                            op = (x.kind, x.idx)
                        else:
                            assert x.kind in ("yo", "yn"), x.kind
                            ys.append((x.kind, x.idx))
                    if op is None and not ys and coef == 0.0:
                        continue
                    ts.append((coef, op, ys))
            d.append(ts)
        out.append(d)
    return out


def _runs(sums):
    """The species in runs that are closed together: no species of a run is a factor, with its new value, of
    another's sums in the same run. The fewest runs (an even number, so that the two sets of exchange buffers
    alternate over the passes), at most CO_RUN species and CO_VALUES partial sums each."""
    nb = CO_LAST + 1
    dep = [{y[1] for side in sums[b] for _, _, ys in side for y in ys if y[0] == "yn"} for b in range(nb)]
    best = {(0, 0, 0): (0, None)}                      # (species done, length of the last run, parity)
    for e in range(1, nb + 1):
        for m in range(1, min(CO_RUN, e) + 1):
            run = range(e - m, e)
            if any(dep[b] & set(run) for b in run):
                continue
            for m0 in range(CO_RUN + 1):
                for par in range(2):
                    if (e - m, m0, par) not in best:
                        continue
                    if len(_values(sums, run, range(e - m - m0, e - m))) > CO_VALUES:
                        continue
                    n = best[(e - m, m0, par)][0] + 1
                    if n < best.get((e, m, 1 - par), (10 ** 9,))[0]:
                        best[(e, m, 1 - par)] = (n, (e - m, m0, par))
    at = min(((nb, m, 0) for m in range(1, CO_RUN + 1) if (nb, m, 0) in best), key=lambda k: best[k][0])
    out = []
    while at[0]:
        out.append(list(range(at[0] - at[1], at[0])))
        at = best[at][1]
    return out[::-1]


def _values(sums, run, prev):
    """The partial sums of a run: (species, 'P' or 'L', factor of the run before or None)."""
    out = []
    for b in run:
        for side, nm in enumerate("PL"):
            ks = sorted({y[1] for _, _, ys in sums[b][side] for y in ys if y[0] == "yn" and y[1] in prev})
            out += [(b, nm, None)] + [(b, nm, k) for k in ks]
    return out


def _pair(t):
    return t[1][1] // 2


def _share_out(sums, runs):
    """Which of the summing warps takes which row pair of each run. A pair in tensor memory belongs to
    one warp; a pair in shared memory may be read by any. The measure is the sum over the runs of the
    largest share, since the warps meet after every run; found by a descent over swaps of tensor-memory
    pairs from a fixed start."""
    import random
    ntp, nr = CO_NT // 2, len(runs)
    cost = [dict() for _ in range(nr)]                # per run: pair -> statements and loads
    for r, run in enumerate(runs):
        for b in run:
            for side in sums[b]:
                for t in side:
                    p = _pair(t)
                    cost[r][p] = cost[r].get(p, 1.0) + 1.0 + 0.3 * max(0, len(t[2]) - 1)
    where = [[(r, cost[r][p]) for r in range(nr) if p in cost[r]] for p in range(ntp)]
    free = [sum(c for p, c in cost[r].items() if p >= ntp) for r in range(nr)]

    def level(load, r):
        """Time of run r, by the slowest warp, with the free pairs dealt out evenly."""
        return max(sum(load[r]) + free[r], *[x / f for x, f in zip(load[r], CO_SHARE)])

    owner, load = [0] * ntp, [[0.0] * CO_SUMS for _ in range(nr)]
    for piece in range(CO_NT // CO_PIECE):
        lo = piece * CO_PIECE // 2
        left = list(CO_PAIRS)
        for p in sorted(range(lo, lo + CO_PIECE // 2), key=lambda p: -sum(c for _, c in where[p])):
            w = min((w for w in range(CO_SUMS) if left[w]),
                    key=lambda w: (sum(max(0.0, load[r][w] + c - max(load[r])) for r, c in where[p]), -left[w]))
            owner[p] = w
            left[w] -= 1
            for r, c in where[p]:
                load[r][w] += c
    rng = random.Random(1)
    for _ in range(60000):
        p = rng.randrange(ntp)
        q = p // (CO_PIECE // 2) * (CO_PIECE // 2) + rng.randrange(CO_PIECE // 2)
        if owner[p] == owner[q]:
            continue
        touched = sorted({r for r, _ in where[p]} | {r for r, _ in where[q]})
        before = sum(level(load, r) for r in touched)

        def swap():
            for r, c in where[p]:
                load[r][owner[p]] -= c
                load[r][owner[q]] += c
            for r, c in where[q]:
                load[r][owner[q]] -= c
                load[r][owner[p]] += c
            owner[p], owner[q] = owner[q], owner[p]
        swap()
        if sum(level(load, r) for r in touched) > before + 1e-9:
            swap()
    # the free pairs: onto the least loaded warp, where a partial sum that the warp does not form yet counts as
    # CO_NEWSUM statements (it has to be handed over and read)
    share = []                                         # per run: pair -> warp
    for r, run in enumerate(runs):
        prev = set(runs[r - 1]) if r else set()
        keys: dict = {}
        for b in run:
            for side, nm in enumerate("PL"):
                for t in sums[b][side]:
                    f = [y[1] for y in t[2] if y[0] == "yn" and y[1] in prev]
                    keys.setdefault(_pair(t), set()).add((b, nm, f[0] if f else None))
        mine = {p: owner[p] for p in cost[r] if p < ntp}
        has = [set().union(*[keys[p] for p in mine if mine[p] == w]) for w in range(CO_SUMS)]
        now = list(load[r])
        for p in sorted((p for p in cost[r] if p >= ntp), key=lambda p: (-cost[r][p], p)):
            w = min(range(CO_SUMS), key=lambda w: (now[w] + cost[r][p] + CO_NEWSUM * len(keys[p] - has[w])) / CO_SHARE[w])
            mine[p] = w
            has[w] |= keys[p]
            now[w] += cost[r][p]
        share.append(mine)
    return owner, share


def _added(parts) -> str:
    """The sum of the parts from left to right, as CO_ADD."""
    e = parts[0]
    for x in parts[1:]:
        e = f"CO_ADD({e}, {x})"
    return e


class _COEmit:
    """Statements of one summing warp. RC(r) is the token @r@, bound later."""

    def __init__(self, place=None):
        self.updated: set[int] = set()
        self.shadow: list[int] = []
        self.place = place or {}           # pair -> tensor-memory column: pairs that are loaded together side by side

    def key(self, t):
        p = _pair(t)
        return (0, self.place[p]) if p in self.place else (1, p)

    def y(self, leaf) -> str:
        kind, k = leaf
        if kind == "yo" and k in self.updated:
            if k not in self.shadow:
                self.shadow.append(k)
            return f"YOS({self.shadow.index(k)})"
        return f"YO({k})"

    def product(self, coef, op, ys) -> tuple:
        """coef * op * ys as two factors (the second None where there is one)."""
        parts = [self.y(v) for v in ys]
        if op is not None:
            parts.append(f"@{op[1]}@" if op[0] == "RC" else f"SOUR({op[1]})")
        if coef != 1.0:
            parts.insert(0, repr(coef))
        e = parts[0]
        for x in parts[1:-1]:
            e = f"({e} * {x})"
        return (e, None) if len(parts) == 1 else (e, parts[-1])

    def sums(self, b, prod, loss, prev, fresh):
        """Statements that form, of the given terms of species b, P and L (without the species of `prev`, the
        run being closed, whose new values are not known yet) and what each species of prev multiplies in
        them. `fresh`: the run before that, whose values arrive meanwhile. Returns the statements that need
        no fresh value, those that do, and {(b, 'P' or 'L', factor or None): expression}."""
        pre: list[tuple] = []              # (accumulator, its sum's number, addend)
        post: list[tuple] = []
        turn: dict[str, int] = {}
        number = [0]

        def add(st, var, expr, sum_=0):
            st.append((var, sum_, expr))

        # two accumulators, in turn, for a sum long enough that its chain of additions would be waited for
        long_ = {"P": len(prod) >= CO_LONG, "L": len(loss) >= CO_LONG}

        def alternate(name):
            turn[name] = turn.get(name, -1) + 1
            return f"{name}{turn[name] & 1 if long_[name] else 0}"

        def is_fresh(t):
            return any(y[1] in fresh for y in t[2])

        def split(terms):
            """({species of prev: terms without it}, [(factor, terms without it)], single terms)"""
            mine, many, single = {}, [], []
            for c, op, ys in terms:
                f = [y for y in ys if y[0] == "yn" and y[1] in prev]
                assert len(f) <= 1
                if f:
                    ys = list(ys)
                    ys.remove(f[0])
                    mine.setdefault(f[0][1], []).append((c, op, ys))
                else:
                    (many if len(ys) >= 2 else single).append((c, op, ys))
            groups = []
            while many:
                cnt: dict = {}
                for _, _, ys in many:
                    for v in set(ys):
                        cnt[v] = cnt.get(v, 0) + 1
                # a fresh factor first: what it multiplies can be summed before it arrives
                f = max(cnt, key=lambda v: (v[1] in fresh, cnt[v], v[0], -v[1]))
                if cnt[f] < 2 and f[1] not in fresh:
                    break
                g = []
                for t in [t for t in many if f in t[2]]:
                    many.remove(t)
                    ys = list(t[2])
                    ys.remove(f)
                    g.append((t[0], t[1], ys))
                groups.append((f, g))
            return mine, groups, single + many

        pm, pg, ps = split(prod)
        lm, lg, ls = split(loss)
        have = {}
        waiting = sorted([("L", t) for t in ls] + [(f"H{i}", t) for i, k in enumerate(sorted(lm)) for t in lm[k]],
                         key=lambda q: self.key(q[1]))

        def put(q):
            waiting.remove(q)
            add(post if is_fresh(q[1]) else pre, alternate(q[0]) if q[0] == "L" else q[0], self.product(*q[1]))

        def loss_of(pair):
            for q in [q for q in waiting if _pair(q[1]) == pair and not is_fresh(q[1])]:
                put(q)

        def inner(g, name):
            """A group's sum as an expression: two accumulators where it is long; (expression, fresh or not)"""
            ways = 2 if len(g) >= CO_LONG else 1
            var = [name + "ab"[w] for w in range(ways)]
            number[0] += 1
            me = number[0]
            now = [t for t in sorted(g, key=self.key) if not is_fresh(t)]
            later = [t for t in sorted(g, key=self.key) if is_fresh(t)]
            for i, t in enumerate(now + later):
                add(pre if i < len(now) else post, var[i % ways], self.product(*t), me)
                loss_of(_pair(t))
            return var[0] if ways == 1 else f"CO_ADD({var[0]}, {var[1]})", bool(later)

        for i, k in enumerate(sorted(pm)):
            have[(b, "P", k)] = inner(pm[k], f"G{i}")[0]
        n = 0
        for sums_, groups in (("P", pg), ("L", lg)):
            for f, g in groups:
                late = f[1] in fresh
                e, deep = inner(g, f"{'ef'[sums_ == 'L']}{f[1]}" if late else f"g{n % 3}")
                assert not deep or late
                n += not late
                add(post if late else pre, alternate(sums_), (self.y(f), e))
        for t in sorted(ps, key=self.key):
            add(post if is_fresh(t) else pre, alternate("P"), self.product(*t))
            loss_of(_pair(t))
        for q in list(waiting):
            put(q)
        for i, k in enumerate(sorted(lm)):
            have[(b, "L", k)] = f"H{i}"
        started: set[tuple] = set()

        def text(st):
            out = []
            for var, sum_, (x, y) in st:
                if (var, sum_) in started:
                    out.append(f"{var} = CO_ADD({var}, {x});" if y is None else f"{var} = CO_FMA({x}, {y}, {var});")
                else:
                    out.append(f"{var} = {x};" if y is None else f"{var} = CO_MUL({x}, {y});")
                started.add((var, sum_))
            return out
        pre, post = text(pre), text(post)
        for nm in "PL":
            v = [x for x in (nm + "0", nm + "1") if (x, 0) in started]
            if v:
                have[(b, nm, None)] = _added(v)
        return pre, post, have


def _segments(body, mine):
    """The statements in segments of at most CO_SEG row pairs in tensor memory."""
    import re
    tok = re.compile(r"@(\d+)@")
    segs, cur, rows = [], [], []
    for st in body:
        need = list(dict.fromkeys(int(x) // 2 for x in tok.findall(st) if int(x) // 2 in mine))
        new = [r for r in need if r not in rows]
        if cur and len(rows) + len(new) > CO_SEG:
            segs.append((cur, rows))
            cur, rows, new = [], [], need
        cur.append(st)
        rows = rows + new
    return segs + [(cur, rows)]


def _place(segs, mine):
    """Tensor-memory columns of a warp's pairs: pairs that are loaded in the same segments side by side (in
    twos, and the twos in twos), heaviest first, so that one wide load brings them."""
    groups = [(p,) for p in sorted(mine)]
    for _ in range(2):
        at = {p: i for i, g in enumerate(groups) for p in g}
        weight: dict = {}
        for _, rows in segs:
            have = sorted({at[p] for p in rows if all(q in rows for q in groups[at[p]])})
            for i, x in enumerate(have):
                for y in have[i + 1:]:
                    weight[(x, y)] = weight.get((x, y), 0) + 1
        taken, merged = set(), []
        for (x, y), _w in sorted(weight.items(), key=lambda q: (-q[1], q[0])):
            if x not in taken and y not in taken and len(groups[x]) == len(groups[y]):
                taken |= {x, y}
                merged.append(groups[x] + groups[y])
        left = [g for i, g in enumerate(groups) if i not in taken]
        full = max(len(g) for g in groups)
        ones = [g for g in left if len(g) < full]
        left = [g for g in left if len(g) == full]
        while len(left) > 1:
            merged.append(left.pop(0) + left.pop(0))
        groups = merged + left + ones
    return {p: 4 * i for i, p in enumerate(p for g in sorted(groups, key=len, reverse=True) for p in g)}


def _bind(body, slots, first=None, shared="RCS2"):
    """Bind the row pairs of a warp's statements: those in `slots` (pair -> tensor-memory column) through two
    register banks, loaded one segment ahead, the others from shared memory. Returns (statements, segments,
    tensor-memory loads, shared-memory loads)."""
    import re
    tok = re.compile(r"@(\d+)@")
    first = CO_NT // 2 if first is None else first     # row pair of the first shared-memory row
    segs = _segments(body, slots)
    out, live, name, nlds, ns, ntm = [], {}, {}, 0, 0, 0
    places = []
    for _, rows in segs:
        # aligned neighbours in one load: four pairs, two pairs, one
        cols = {slots[r]: r for r in rows}
        order, lds = [], []
        for n in (4, 2, 1):
            for c in sorted(cols):
                if c in cols and c % (4 * n) == 0 and all(c + 4 * i in cols for i in range(n)):
                    lds.append((n, len(order), c, [cols[c + 4 * i] for i in range(n)]))
                    order += [cols.pop(c + 4 * i) for i in range(n)]
        places.append((order, lds))

    def loads(si):
        nonlocal ntm
        ntm += len(places[si][1])
        return [f"TM_LD{2 * n}({si % 2}, {q}, {c}, {', '.join(map(str, ps))});" for n, q, c, ps in places[si][1]]
    def wait(si):
        n = len(segs[si][1])
        return [f"TM_WAIT({si % 2}, {n});"] if n else []
    out += loads(0) + wait(0)
    for si, (stmts, rows) in enumerate(segs):
        slot = {r: q for q, r in enumerate(places[si][0])}
        if si + 1 < len(segs):
            out += loads(si + 1)
        for st in stmts:
            ns += 1
            for x in tok.findall(st):
                pr = int(x) // 2
                if pr in slots:
                    continue
                if pr not in live or ns - live[pr] > CO_REUSE:
                    name[pr] = f"s{nlds}"
                    out.append(f"const double2 s{nlds} = {shared}({pr - first});")
                    nlds += 1
                live[pr] = ns

            def bind(m):
                r = int(m.group(1))
                if r // 2 in slots:
                    return f"RCT({si % 2}, {2 * slot[r // 2] + r % 2})"
                return f"{name[r // 2]}.{'xy'[r % 2]}"
            out.append(tok.sub(bind, st))
        if si + 1 < len(segs):
            out += wait(si + 1)
    return out, len(segs), ntm, nlds


def gen_co_program(blocks) -> str:
    """The species update with three warps per tile: two form the sums of the species, each from the terms
    of its own row pairs, and the third closes them. The sums are grouped: terms that share a mass fraction
    are added before they are multiplied by it, so that a term costs one fused multiply-add. Species that do
    not enter one another's sums are closed together, in runs. While the closing warp forms a run, the others
    already sum the next one: what a species of the run multiplies there is summed apart and waits for it in
    one multiply-add. Terms, factors and the order of the species are those of the in-place program; only the
    order of the additions and multiplications within a sum differs."""
    import re
    full = _grouped_sums(blocks)
    assert [b["species"] for b in blocks] == list(range(LSP - 1))
    assert all(not any(s) for s in full[CO_LAST + 1:]) and all(b["prod"] is None for b in blocks[CO_LAST + 1:])
    assert len(full[CO_LAST][0]) == len(blocks[CO_LAST]["prod"])      # no extra terms in the sum they reuse
    # the few soot-source terms are the closing warp's
    sour = [[[t for t in side if t[1] is not None and t[1][0] == "SOUR"] for side in s] for s in full]
    sums = [[[t for t in side if t[1] is not None and t[1][0] == "RC"] for side in s] for s in full]
    assert all(len(a) + len(c) == len(d) for x, y, z in zip(sums, sour, full) for a, c, d in zip(x, y, z))
    runs = _runs(sums)
    nr = len(runs)
    owner, share = _share_out(sums, runs)
    macros, stats = [], []
    flops = 19                                         # the two soot scalars

    def operations(stmts):
        return sum(st.count(" * ") + st.count(" + ") + st.count(" - ") + 2 * st.count("CO_FMA(") + st.count("CO_ADD(") +
                   st.count("CO_MUL(") + st.count("CO_QUOT(") for st in stmts)

    shadow_max = 1
    handed = [[None] * CO_SUMS for _ in range(nr)]           # per run and warp: values in the order of its slots
    slots_of = [0, 0]                                  # pair rows of each set of exchange buffers
    base = [[0] * CO_SUMS for _ in range(nr)]

    def program(w, place):
        """Statements of summing warp w; place: tensor-memory columns of its pairs."""
        em = _COEmit(place)
        body: list[str] = []

        def take(r, now):
            return [f"CO_WAIT_Y({r & 1});"] + [f"CO_GET({3 * (r & 1) + i}, {k}, {int(k % CO_SUMS == w)}, {now});"
                                             for i, k in enumerate(runs[r])]

        def run_sums(r, before_post):
            """The partial sums of run r; before_post: statements that bring the fresh values."""
            prev = set(runs[r - 1]) if r > 0 else set()
            fresh = set(runs[r - 2]) if r > 1 else set(runs[nr - 1]) if r == 0 else set()
            st, vals, waited = [], {}, False
            for b in runs[r]:
                mine = [[t for t in side if share[r][_pair(t)] == w] for side in sums[b]]
                pre, post, hv = em.sums(b, mine[0], mine[1], prev, fresh if not waited else set())
                st += pre
                if not waited:
                    st += before_post
                    waited = True
                st += post
                # the value's own variable, since the next species of the run uses the accumulators again
                for key, e in hv.items():
                    v = f"v{len(vals)}"
                    st.append(f"{v} = {e};")
                    vals[key] = v
            keys = [k for k in _values(sums, runs[r], prev) if k in vals]
            handed[r][w] = keys
            for i in range(0, len(keys), 2):
                st.append(f"CO_PUT(@@{r},{w},{i // 2}@@, {vals[keys[i]]}, {vals[keys[i + 1]] if i + 1 < len(keys) else '0.0'});")
            return st + [f"CO_ARRIVE_P({r & 1});"]

        # (the species of the last run are known from the pass before)
        body += run_sums(0, take(nr - 1, 0))
        body.append("CO_CHECK();")
        for r in range(1, nr):
            em.updated |= set(runs[r - 1])             # being closed now: an old value is the copy
            body += run_sums(r, take(r - 2, 1) if r > 1 else [])
        body += take(nr - 2, 1)
        first = next(i for i, x in enumerate(body) if x == "CO_CHECK();")
        body[first:first] = [f"YOS({m}) = YO({k});" for m, k in enumerate(em.shadow)]
        return body, len(em.shadow)
    bodies, places = [], []
    for w in range(CO_SUMS):
        mine = {p for p, v in enumerate(owner) if v == w}
        place = {p: 4 * i for i, p in enumerate(sorted(mine))}
        for _ in range(3):                             # places from the segments, statements in the places' order
            body, n = program(w, place)
            place = _place(_segments(body, mine), mine)
        body, n = program(w, place)
        shadow_max = max(shadow_max, n)
        bodies.append(body)
        places.append(place)
    for r in range(nr):
        n = 0
        for w in range(CO_SUMS):
            base[r][w] = n
            n += (len(handed[r][w]) + 1) // 2
        slots_of[r & 1] = max(slots_of[r & 1], n)

    def slot(m):
        r, w, i = (int(x) for x in m.group(1).split(","))
        return str((slots_of[0] if r & 1 else 0) + base[r][w] + i)
    mark = re.compile(r"@@(\d+,\d+,\d+)@@")
    for w in range(CO_SUMS):
        body = [mark.sub(slot, st) for st in bodies[w]]
        flops += operations(body)
        out, nseg, nt, ns = _bind(body, places[w])
        stats.append((nseg, nt, ns, operations(body)))
        names = sorted({m for st in body for m in re.findall(r"\b([PLvGHgef]\d+[ab]?)\b", st)})
        macros.append(["#define UC_CO_SUMS_%d() do { \\" % w, f"    double {', '.join(names)}; \\"] +
                      ["    " + x + " \\" for x in out] + ["} while (0)"])
    # ---- the closing warp
    close: list[str] = []
    names = {"rest"}

    def fetch(r):
        """The partial sums of run r, added up over the warps."""
        st, parts = [f"CO_WAIT_P({r & 1});"], {}
        for w in range(CO_SUMS):
            keys = handed[r][w]
            for i in range(0, len(keys), 2):
                x, y = f"x{w}{i // 2}", f"y{w}{i // 2}"
                names.update((x, y))
                st.append(f"CO_TAKE({(slots_of[0] if r & 1 else 0) + base[r][w] + i // 2}, {x}, {y});")
                parts.setdefault(keys[i], []).append(x)
                if i + 1 < len(keys):
                    parts.setdefault(keys[i + 1], []).append(y)
        total = {}
        for j, (key, vs) in enumerate(sorted(parts.items(), key=lambda q: str(q[0]))):
            v = f"t{r & 1}{j}"
            names.add(v)
            st.append(f"{v} = {_added(vs)};")
            total[key] = v
        return st, total

    def faces(r):
        return [f"CO_PF({k % window}, {k});" for k in (runs[r] if r < nr else range(CO_LAST + 1, LSP - 1) if r == nr else [])]
    spans = [len(x) for x in runs] + [2]
    window = max(sum(spans[i:i + 3]) for i in range(len(spans)))

    def finish(k):
        return [f"fnew = CO_FMA(sor2, YO({k}), q{k % 3});", f"rsd += fabs(YO({k}) - fnew);", f"CO_TAIL({k});"]
    close += faces(0) + faces(1)
    st, total = fetch(0)
    close += st + ["CO_CHECK();"]
    for r, run in enumerate(runs):
        close += faces(r + 2)
        for k in run:
            e = {}
            for side, nm in enumerate("PL"):
                x = total.get((k, nm, None), "")
                more = [(f"YO({key[2]})", v) for key, v in sorted(total.items(), key=lambda q: str(q[0]))
                        if key[0] == k and key[1] == nm and key[2] is not None]
                for c, op, ys in sour[k][side]:
                    assert all(y[0] == "yn" or y[1] >= k for y in ys) and len(ys) <= 1
                    more.append((f"SOUR({op[1]})" if c == 1.0 else f"({c!r} * SOUR({op[1]}))", f"YO({ys[0][1]})" if ys else None))
                for f, v in more:
                    if v is None:
                        x = f"CO_ADD({x}, {f})" if x else f
                    else:
                        x = f"CO_FMA({f}, {v}, {x})" if x else f"CO_MUL({f}, {v})"
                e[nm] = x
            if k == CO_LAST:
                close.append(f"rest = {e['P']};")      # argon and helium reuse the last production sum
                e["P"] = "rest"
            num = f"CO_FMA(DTW({k}), {e['P']}, RY0({k}))" if e["P"] else f"RY0({k})"
            den = f"rho - FSS({k % window})"
            close.append(f"n{k % 3} = ({num} - FNS({k % window})) * sor1;")
            close.append(f"d{k % 3} = " + (f"CO_FMA(DTW({k}), {e['L']}, {den});" if e["L"] else f"{den};"))
        # the next run's partial sums are fetched while the quotients are on their way
        st, total = fetch(r + 1) if r + 1 < nr else ([], {})
        close += [f"q{k % 3} = CO_QUOT(n{k % 3}, d{k % 3});" for k in run] + st
        for i, k in enumerate(run):
            close += finish(k) + [f"CO_GIVE({3 * (r & 1) + i}, {k});"]
        close.append(f"CO_ARRIVE_Y({r & 1});")
    for k in range(CO_LAST + 1, LSP - 1):
        close.append(f"n{k % 3} = (CO_FMA(DTW({k}), rest, RY0({k})) - FNS({k % window})) * sor1;")
        close.append(f"d{k % 3} = rho - FSS({k % window});")
        close.append(f"q{k % 3} = CO_QUOT(n{k % 3}, d{k % 3});")
        close += finish(k)
    flops += operations(close)
    macros.append(["#define UC_CO_CLOSE() do { \\", f"    double n0, n1, n2, d0, d1, d2, q0, q1, q2, fnew, {', '.join(sorted(names))}; \\"] +
                  ["    " + x + " \\" for x in close] + ["} while (0)"])
    # in the order of staging: (pair, column)
    rows = [[(p, places[w][p]) for p in sorted(places[w])] for w in range(CO_SUMS)]
    L = ["// Generated by unicorn_b200/mech/codegen.py: the species update (src/lib/solvesp.f:85-2806) with three",
         "// warps per 32-cell tile. UC_CO_SUMS_0 and _1 are a pass of the two summing warps, UC_CO_CLOSE one of the",
         f"// closing warp. RC slots 0..{CO_NT - 1} lie in tensor memory, each pair of slots (2p, 2p + 1) with the one",
         "// summing warp that uses it (uc_co_pairs_w: the pairs in row order; uc_co_cols_w: the first of the four",
         "// 32-bit columns of each); the others lie in shared memory as rows of pairs, RCS2(i). Accessors: TM_LD2(bank,",
         "// q, col, p) loads pair p (column col) into slots 2q, 2q + 1 of a register bank, TM_LD4 and TM_LD8 two and four",
         "// pairs in neighbouring columns, TM_WAIT(bank, n) waits for the loads of its n pairs, RCT(bank, i); CO_PUT",
         "// (slot, a, b) publishes two partial sums, CO_TAKE(slot, a, b) reads them; CO_GIVE(buf, k) publishes the",
         "// new Y of species k, CO_GET(buf, k, mine, now) takes it into YO(k) (mine: this warp also stores it; now: of",
         "// this pass, else of the pass before). Even and odd runs use sets 0 and 1 of the buffers and barriers:",
         "// CO_ARRIVE_P(set) by the summing warps, CO_WAIT_P(set) by the closing one, CO_ARRIVE_Y, CO_WAIT_Y the other way;",
         "// CO_CHECK() may leave the program (no more passes). CO_PF(slot, k) fetches the face terms of species k",
         "// (FSS, FNS); RY0(k) is rho times the old level's Y; DTW(k) is dt * WM(k); CO_QUOT(n, d) is the quotient;",
         "// CO_FMA(a, b, c) = a * b + c, CO_MUL and CO_ADD are rounded as they stand, so that every kernel that runs the",
         "// program computes a cell bit for bit the same.",
         f"// {nr} runs: {' '.join('-'.join(map(str, sorted({x[0], x[-1]}))) for x in runs)}",
         "// Per summing warp: " + "; ".join(f"{a} segments, {b} tensor-memory loads, {c} shared-memory pair loads, {d} "
                                          "operations" for a, b, c, d in stats) + ".",
         "#pragma once",
         f"#define UC_CO_NT {CO_NT}", f"#define UC_CO_NS {LRX - CO_NT}", f"#define UC_CO_PIECE {CO_PIECE}",
         f"#define UC_CO_SEG {CO_SEG}", f"#define UC_CO_SUMS {CO_SUMS}", f"#define UC_CO_NSHADOW {shadow_max}", f"#define UC_CO_LAST {CO_LAST}",
         f"#define UC_CO_SLOTS {sum(slots_of)}", f"#define UC_CO_WINDOW {window}",
         "// the last run: its species' buffers hold their values when a pass begins, handed over through the set",
         f"#define UC_CO_LAST_SET {(nr - 1) & 1}", "#define UC_CO_LAST_RUN() do { " +
         " ".join(f"CO_LAST_SPECIES({3 * ((nr - 1) & 1) + i}, {k});" for i, k in enumerate(runs[-1])) + " } while (0)",
         "// operations per cell and pass (a multiply-add is two, a quotient one), the exchange between the warps included",
         f"#define UC_UPDATE_FLOPS_PER_CELL_PASS {flops}"]
    for w in range(CO_SUMS):
        L.append(f"#define UC_CO_PAIRS_{w} {CO_PAIRS[w]}")
    for m in macros:
        L += m
    for kind, guard in (("static __constant__ int16_t", "#ifdef __CUDACC__"), ("static const short", "#else")):
        L.append(guard)
        for w in range(CO_SUMS):
            for i, nm in enumerate(("pairs", "cols")):
                L.append(f"{kind} uc_co_{nm}_{w}[{len(rows[w])}] = {{{', '.join(str(x[i]) for x in rows[w])}}};")
    L.append("#endif")
    return "\n".join(L) + "\n"


# ------------------------------------------------------------------ species source terms

OM_WARPS = 16


def gen_omega_program(mech: dict) -> str:
    """The gain sum P_k and the loss sum L_k (the loss terms with one Y_k factored out, so that the production
    is P_k - Y_k L_k and d(omega_k)/dY_k is -L_k) of every species from the PRD lists of
    src/lib/solveh.f:677-1133, as straight-line code for the warps of a tile: each sum is one warp's, longest
    first onto the least loaded. Terms that share a mass fraction are added before they are multiplied by it."""
    import re
    units = []
    for key, terms in mech["prd"].items():
        k = int(key) - 1
        gain, loss = [], []
        for s, fac in terms or []:
            if fac[-1][0] == "SRA":
                continue                               # SRA(i) = 0.0 (src/lib/solveh.f:671-676)
            assert fac[-1][0] == "RA" and all(f[0] == "num" for f in fac[:-1])
            r = fac[-1][1] - 1
            if mech["ra"][str(r + 1)] is None:
                continue                               # a slot that is never written: its RC is zero
            ys = [("yo", x - 1) for x in mech["ra"][str(r + 1)]]
            coef = 1.0
            for f in fac[:-1]:
                coef *= f[1]
            if s > 0:
                gain.append((coef, ("RC", r), ys))
            else:
                ys.remove(("yo", k))
                loss.append((coef, ("RC", r), ys))
        units += [(k, "P", gain), (k, "L", loss)]
    load = [0.0] * OM_WARPS
    mine: list[list] = [[] for _ in range(OM_WARPS)]
    for u in sorted(units, key=lambda u: (-len(u[2]), u[0], u[1])):
        w = min(range(OM_WARPS), key=lambda w: load[w])
        mine[w].append(u)
        load[w] += 2.0 + 1.6 * len(u[2])
    tok = re.compile(r"@(\d+)@")
    L = ["// Generated by unicorn_b200/mech/codegen.py: the species' gain and loss sums from the PRD lists of",
         "// src/lib/solveh.f:677-1133, shared out over the warps of a tile: UC_OMEGA_w() is warp w's part.",
         "// Requires RCP(p), the pair (RC(2p), RC(2p + 1)) of the cell as a double2, YO(k), and OM_PUT(k, v) and",
         "// OM_PUT(52 + k, v), which store P_k and L_k; CO_FMA, CO_MUL, CO_ADD as in the species update.",
         "#pragma once", f"#define UC_OM_WARPS {OM_WARPS}"]
    for w, us in enumerate(mine):
        em, body = _COEmit(), []
        for k, nm, terms in us:
            pre, post, have = em.sums(k, terms if nm == "P" else [], terms if nm == "L" else [], set(), set())
            assert not post
            body += pre + [f"OM_PUT({k + (LSP if nm == 'L' else 0)}, {have.get((k, nm, None), '0.0')});"]
        out, _, _, _ = _bind(body, {}, 0, "RCP")
        names = sorted({m for st in body for m in re.findall(r"\b([PLvGHgef]\d+[ab]?)\b", st)})
        L += ["#define UC_OMEGA_%d() do { \\" % w, f"    double {', '.join(names)}; \\"] + ["    " + x + " \\" for x in out] + ["} while (0)"]
    return "\n".join(L) + "\n"


# ------------------------------------------------------------------ tables

def fmt(v: float) -> str:
    return repr(float(v)) if v == v else "0.0"


def arr(name, ctype, vals, per_line=8) -> str:
    vals = list(vals)
    rows = []
    for i in range(0, len(vals), per_line):
        rows.append("    " + ", ".join(vals[i:i + per_line]))
    return f"static const {ctype} {name}[{len(vals)}] = {{\n" + ",\n".join(rows) + "\n};\n"


def element_counts(names) -> list[list[int]]:
    import re
    out = []
    for nm in names:
        base = re.sub(r"^[A-Z]-", "", nm)
        c = {"C": 0, "H": 0, "O": 0}
        if base not in ("AR", "HE", "N2"):
            assert re.fullmatch(r"([CHO]\d*)+", base), nm
            for el, cnt in re.findall(r"([CHO])(\d*)", base):
                c[el] += int(cnt) if cnt else 1
        out.append([c["C"], c["H"], c["O"]])
    return out


def gen_tables(mech: dict) -> str:
    R = mech["reactions"]
    out = ["// Generated by unicorn_b200/mech/codegen.py from sandiego52.json (the",
           "// San Diego mechanism as UNICORN encodes it: src/lib/DATA.f, src/lib/ckrates.f,",
           "// src/lib/solveh.f, src/unicornd-mild-sd-5.f:76-113). Do not edit.",
           "#pragma once", "#include <stdint.h>",
           f"#define UC_LSP {LSP}", f"#define UC_LRX {LRX}", f"#define UC_NPAIR {LRX // 2}",
           f"#define UC_TPOL1 {fmt(mech['tpol'][0])}", f"#define UC_TPOL2 {fmt(mech['tpol'][1])}"]
    out.append(arr("uc_wsp", "double", map(fmt, mech["wsp"])))
    # atoms of C, H and O per species, read from the species names (T-, S-, I-, N- are isomer prefixes;
    # AR, HE and N2 carry none of the three): every reaction conserves them, so the exact omega does
    out.append(arr("uc_elem_cho", "int8_t", (str(v) for row in element_counts(mech["species"]) for v in row), 3))
    out.append(arr("uc_cdia", "double", map(fmt, mech["cdia"])))
    out.append(arr("uc_tlj", "double", map(fmt, mech["tlj"])))
    out.append(arr("uc_poly", "double", (fmt(v) for row in mech["poly"] for v in row)))
    out.append(arr("uc_om22", "double", (fmt(v) for row in mech["omega22"] for v in row)))
    out.append(arr("uc_ci11", "double", (fmt(v) for row in mech["ci11"] for v in row)))
    for k in ("akf", "alf", "exaf", "aklow", "allow", "ealow"):
        out.append(arr(f"uc_raw_{k}", "double", (fmt(x[k]) for x in R)))
    out.append(arr("uc_raw_troe", "double", (fmt(v) for x in R for v in x["troe"])))
    # reverse formulas: per even slot (0-based odd index r0), rut and q chain (<= 6 factors)
    QMAX = max(len(v["q"]) for v in mech["reverse"].values())
    rev_has, rev_rut, rev_len = [0] * LRX, [0] * LRX, [0] * LRX
    rev_sp = [0] * (LRX * QMAX)
    rev_div = [0] * (LRX * QMAX)
    for key, rv in mech["reverse"].items():
        r0 = int(key) - 1
        rev_has[r0], rev_rut[r0], rev_len[r0] = 1, rv["rut"], len(rv["q"])
        for t, (op, sp) in enumerate(rv["q"]):
            rev_sp[r0 * QMAX + t] = sp - 1
            rev_div[r0 * QMAX + t] = 1 if op == "/" else 0
    out.append(f"#define UC_QMAX {QMAX}")
    out.append(f"#define UC_QMIN {min(len(v['q']) for v in mech['reverse'].values())}")
    # fall-off pairs: a negative AKF of the forward slot marks them (src/unicornd-mild-sd-5.f:364-413)
    out.append(f"#define UC_FALLOFF {sum(x['akf'] < 0 and x['aklow'] != 0 for x in R[::2])}")
    out.append(arr("uc_rev_has", "int8_t", map(str, rev_has), 32))
    out.append(arr("uc_rev_rut", "int8_t", map(str, rev_rut), 32))
    out.append(arr("uc_rev_len", "int8_t", map(str, rev_len), 32))
    out.append(arr("uc_rev_sp", "int8_t", map(str, rev_sp), 32))
    out.append(arr("uc_rev_div", "int8_t", map(str, rev_div), 32))
    # third-body groups 1..10: TBODY + sum sign*coef*Y/W
    tbn = [0] * 11
    tbo = [0] * 11
    tsp, tsg, tco, thc = [], [], [], []
    for g in range(1, 11):
        terms = mech["tb"][f"TB{g:03d}"][1:]
        tbo[g], tbn[g] = len(tsp), len(terms)
        for s, k, c in terms:
            tsp.append(k - 1)
            tsg.append(s)
            tco.append(0.0 if c is None else c)
            thc.append(0 if c is None else 1)
    out.append(f"#define UC_NTB {len(mech['tb']) - 1}")
    out.append(arr("uc_tb_off", "int16_t", map(str, tbo), 16))
    out.append(arr("uc_tb_len", "int16_t", map(str, tbn), 16))
    out.append(arr("uc_tb_sp", "int8_t", map(str, tsp), 32))
    out.append(arr("uc_tb_sign", "int8_t", map(str, tsg), 32))
    out.append(arr("uc_tb_coef", "double", map(fmt, tco)))
    out.append(arr("uc_tb_hascoef", "int8_t", map(str, thc), 32))
    dm = [0] * LRX
    for key, g in mech["dmole"].items():
        dm[int(key) - 1] = int(g[2:])
    out.append(arr("uc_dmole_grp", "int8_t", map(str, dm), 32))
    # RC assembly: order (0 = never written), tb (-1 none, 0 TBODY, g), post ops <= 4
    PMAX = max(len(v["post"]) for v in mech["rc"].values())
    rc_order, rc_tb, rc_len = [0] * LRX, [-1] * LRX, [0] * LRX
    rc_kind = [0] * (LRX * PMAX)
    rc_idx = [0] * (LRX * PMAX)
    for key, rc in mech["rc"].items():
        r0 = int(key) - 1
        rc_order[r0] = rc["order"]
        rc_tb[r0] = -1 if rc["tb"] is None else (0 if rc["tb"] == "TBODY" else int(rc["tb"][2:]))
        rc_len[r0] = len(rc["post"])
        for t, (op, kind, idx) in enumerate(rc["post"]):
            rc_kind[r0 * PMAX + t] = 1 if kind == "Y" else 0   # 1: *Y_idx, 0: /W_idx
            rc_idx[r0 * PMAX + t] = idx - 1
    out.append(f"#define UC_PMAX {PMAX}")
    out.append(f"#define UC_RC_YMAX {max(sum(kind == 'Y' for _, kind, _ in v['post']) for v in mech['rc'].values())}")
    out.append(arr("uc_rc_order", "int8_t", map(str, rc_order), 32))
    out.append(arr("uc_rc_tb", "int8_t", map(str, rc_tb), 32))
    out.append(arr("uc_rc_len", "int8_t", map(str, rc_len), 32))
    out.append(arr("uc_rc_kind", "int8_t", map(str, rc_kind), 32))
    out.append(arr("uc_rc_idx", "int8_t", map(str, rc_idx), 32))
    # RA reactant lists (<= 3), 0 = slot never written
    ra_len = [0] * LRX
    ra_sp = [0] * (LRX * 3)
    for key, sps in mech["ra"].items():
        r0 = int(key) - 1
        if sps is None:
            continue
        ra_len[r0] = len(sps)
        for t, s in enumerate(sps):
            ra_sp[r0 * 3 + t] = s - 1
    out.append(arr("uc_ra_len", "int8_t", map(str, ra_len), 32))
    out.append(arr("uc_ra_sp", "int8_t", map(str, ra_sp), 32))
    # PRD term lists per species: packed (r0 | sign<<15 | coef_flag<<14), coef is 1.000 or SRA(0)
    prd_off, prd_len, prd_term, prd_coef = [0] * LSP, [0] * LSP, [], []
    loss_off, loss_len, loss_term = [0] * LSP, [0] * LSP, []
    for key, terms in mech["prd"].items():
        k0 = int(key) - 1
        if not terms:
            continue
        prd_off[k0] = len(prd_term)
        loss_off[k0] = len(loss_term)
        for s, fac in terms:
            kinds = [f[0] for f in fac]
            if kinds == ["SRA"]:
                # SRA(i) = 0.0 (src/lib/solveh.f:671-676): a zero term
                prd_term.append((LRX) | ((1 if s < 0 else 0) << 15) | (1 << 13))
                prd_coef.append(0.0)
                continue
            if kinds == ["RA"]:
                coef, r = None, fac[0][1]
            else:
                assert kinds == ["num", "RA"], fac
                coef, r = fac[0][1], fac[1][1]
            prd_term.append((r - 1) | ((1 if s < 0 else 0) << 15) | ((1 if coef is not None else 0) << 14))
            prd_coef.append(0.0 if coef is None else coef)
            if s < 0:
                assert coef is None, "loss terms carry no coefficient in this mechanism"
                loss_term.append(r - 1)
        prd_len[k0] = len(prd_term) - prd_off[k0]
        loss_len[k0] = len(loss_term) - loss_off[k0]
    out.append(arr("uc_prd_off", "int16_t", map(str, prd_off), 16))
    out.append(arr("uc_prd_len", "int16_t", map(str, prd_len), 16))
    out.append(arr("uc_prd_term", "uint16_t", map(str, prd_term), 16))
    out.append(arr("uc_prd_coef", "double", map(fmt, prd_coef)))
    out.append(arr("uc_loss_off", "int16_t", map(str, loss_off), 16))
    out.append(arr("uc_loss_len", "int16_t", map(str, loss_len), 16))
    out.append(arr("uc_loss_term", "uint16_t", map(str, loss_term), 16))
    out.append(f"#define UC_NPRD_TERMS {len(prd_term)}")
    out.append(f"#define UC_NLOSS_TERMS {len(loss_term)}")
    return "\n".join(out) + "\n"


def main():
    mech = json.loads(MECH.read_text())
    GEN.mkdir(parents=True, exist_ok=True)
    (GEN / "mech_tables.h").write_text(gen_tables(mech))
    (GEN / "update_program.cuh").write_text(gen_update_program(mech))
    blocks = resolve_update(mech)
    uses: dict[int, int] = {}
    for b in blocks:
        for key in ("prod", "extra", "loss"):
            for _, t in (b[key] or []):
                for leaf in leaves(t, []):
                    if leaf.kind == "RC":
                        uses[leaf.idx] = uses.get(leaf.idx, 0) + 1
    (GEN / "update_program_tr.cuh").write_text(gen_tr_program(blocks, uses, gen_inplace_program.shadow))
    (GEN / "update_program_co.cuh").write_text(gen_co_program(blocks))
    (GEN / "omega_program.cuh").write_text(gen_omega_program(mech))
    print("wrote", ", ".join(str(GEN / f) for f in ("mech_tables.h", "update_program.cuh", "update_program_tr.cuh",
                                                   "update_program_co.cuh", "omega_program.cuh")))


if __name__ == "__main__":
    main()
