"""Lane schedules of the cooperative kernels (a warp's lanes integrate one cell in shared memory).

A routine of the cell's solver (rates, right-hand side, Jacobian, factorisation, triangular
solves) is written down as the sequence of its scalar operations, every one of the form
``acc = +-x[a] * x[b] + c`` or ``x[d] = 1 / x[d]``, in the order of the generated sequential
code.  `schedule` deals these operations out to W lanes, row by row: a row is one operation
per lane, and an operation is placed as soon as the values that it reads are there, longest
remaining chain first.  No operation is changed and no sum is reordered: each element of the
cell's state goes through the same operations on the same values as in the sequential
routine, so the results have the same bits.

The kernel (csrc/coop.cuh) loads the operands of row t + 2 before it stores the results of
row t, so a value is read at the earliest three rows after the one that computed it, unless
the same lane goes on with it in its accumulator.  The kernel goes through UNROLL rows
without a branch (a test for reciprocals in each row took 50 of its 165 cycles); a row of
reciprocals takes the place of such a block.

Tables are made from the mechanism's manifest alone:

    python -m cmaq_gb300.mechgen.coop
"""
from __future__ import annotations

import json
from dataclasses import dataclass, field
from pathlib import Path

from .emit_common import c_double
from .emit_cuda import _jac_terms
from .fortran_tables import Mechanism
from .sparse import SparseMech, build_sparse

PKG = Path(__file__).resolve().parents[1]
VISIBLE = 3          # rows from the one that computes a value to the first that may load it
CHUNK = 28           # rows of a table that are fetched together (more would cost CRACMM2 a cell)
AHEAD = 3            # rows past a chunk's end whose words the kernel may look at
UNROLL = 4           # rows that the kernel goes through without a branch: a row of reciprocals
                     # comes only after a multiple of it, in a block of its own
SLACK = 3            # how much shorter a reciprocal's chain may be than the longest one
SMEM_MAX = 227 * 1024
TABLE_SMEM = 2 * (CHUNK + AHEAD) * 32 * 8 + 64   # two chunks in flight, each with rows of zeros, and their barriers

# where an operation's addend comes from: the element itself, the lane's accumulator, -0.0
# (the exact identity of an addition: a product alone); MULACC: acc * x[b]
LOAD, KEEP, NEG0, MULACC = range(4)
# encoding: word 0 = offset of a | offset of b << 16, word 1 = offset of d, and flags.
# Offsets are bytes (multiples of 8) into the cell's state; b may be a constant's offset.
A_RECIP, C_LOAD, C_KEEP, C_MULACC = 1, 1, 2, 4
D_STORE, B_CONST, A_NEG = 1 << 16, 1 << 17, 1 << 31
ADDEND = {LOAD: C_LOAD, KEEP: C_KEEP, NEG0: 0, MULACC: C_MULACC}


@dataclass
class Program:
    """Operations in sequential order: ("F", d, a, b, negate a, addend) or ("D", d).  Elements are
    names or ("c", value) constants."""
    ops: list = field(default_factory=list)

    def fma(self, d, a, b, neg=False, init=LOAD):
        self.ops.append(("F", d, a, b, neg, init))

    def recip(self, d):
        self.ops.append(("D", d, d, None, False, LOAD))


def dependencies(ops) -> list[list[tuple[int, str]]]:
    """Per operation its predecessors: "R" reads a value it wrote, "C" goes on with its sum,
    "W" reads what this one overwrites, "O" wrote the same element before."""
    last, readers, preds = {}, {}, []
    for i, (kind, d, a, b, _, init) in enumerate(ops):
        p = []
        scaled = kind == "F" and init == NEG0 and a == d      # d = d * x[b]
        reads = [d] if kind == "D" else ([b] if init == MULACC or scaled else [a, b])
        for e in reads:
            if isinstance(e, tuple):
                continue
            if e in last:
                p.append((last[e], "R"))
            readers.setdefault(e, []).append(i)
        if kind == "F" and (init in (LOAD, MULACC) or scaled):
            if d in last:
                p.append((last[d], "C"))
            elif init == MULACC:
                raise ValueError(f"{d} multiplied before it was formed")
            readers.setdefault(d, []).append(i)
        p += [(r, "W") for r in readers.get(d, []) if r != i]
        if d in last:
            p.append((last[d], "O"))
        readers[d] = []
        last[d] = i
        preds.append(p)
    return preds


@dataclass
class Schedule:
    rows: list          # ("F", [operation or None per lane]) or ("D", [operation or None per lane])
    kind: list          # addend kind of each operation as placed (LOAD may have become KEEP)
    store: list         # whether the operation's result goes to its element


def schedule(ops, width: int, recip_cost: int = 3) -> Schedule:
    """List scheduling, the longest remaining dependence chain first."""
    n = len(ops)
    preds = dependencies(ops)
    succ = [[] for _ in range(n)]
    chain = [None] * n
    for i, ps in enumerate(preds):
        for p, k in ps:
            succ[p].append((i, k))
            if k == "C":
                chain[i] = p

    def latency(p, k, i):
        if k in "WO":
            return 0
        if ops[p][0] == "D" or ops[i][0] == "D":
            return 1
        return VISIBLE

    prio = [0] * n
    for i in range(n - 1, -1, -1):
        own = recip_cost if ops[i][0] == "D" else 1
        best = own
        for j, k in succ[i]:
            step = 0 if k == "W" else own + (VISIBLE - 1 if k == "R" and ops[i][0] == "F" else 0)
            best = max(best, step + prio[j])
        prio[i] = best
    open_preds = [len(p) for p in preds]
    when, lane_of = [-1] * n, [-1] * n
    waiting = {i for i in range(n) if not open_preds[i]}
    lane_acc = [None] * width            # the operation whose result a lane's accumulator holds
    product = [None] * width             # the MULACC that waits for it
    read = [any(k == "R" for _, k in s) for s in succ]   # others load the result
    kind = [op[5] for op in ops]
    store = [True] * n
    rows, t, done = [], 0, 0

    def earliest(i, skip_chain=False):
        e = 0
        for p, k in preds[i]:
            if not (skip_chain and k == "C"):
                e = max(e, when[p] + latency(p, k, i))
        return e

    ready_at = {i: 0 for i in waiting}
    while done < n:
        ready = [i for i in waiting if ready_at[i] <= t]
        recips = sorted((i for i in ready if ops[i][0] == "D"), key=lambda i: (-prio[i], i))[:width]
        # operations that a lane can go on with in its accumulator
        goes_on = {i for i in waiting if chain[i] is not None and ops[i][0] == ops[chain[i]][0] == "F"
                   and lane_acc[lane_of[chain[i]]] == chain[i] and earliest(i, skip_chain=True) <= t}
        cand = sorted(goes_on.union(i for i in ready if ops[i][0] == "F" and ops[i][5] != MULACC),
                      key=lambda i: (-prio[i], i))
        if recips and t % UNROLL == 0 and (not cand or prio[recips[0]] >= prio[cand[0]] - SLACK):
            rows.append(("D", recips + [None] * (width - len(recips))))
            for lane, i in enumerate(recips):
                when[i], lane_of[i] = t - 1, lane
            placed = recips
        else:
            lanes, fresh = [None] * width, []
            for i in goes_on:            # a product's accumulator waits for it
                if ops[i][5] == MULACC:
                    lanes[lane_of[chain[i]]] = i
            room = sum(lanes[ln] is None and product[ln] is None for ln in range(width))
            for i in cand:
                if not room:
                    break
                if ops[i][5] == MULACC:
                    continue
                ln = lane_of[chain[i]] if i in goes_on else None
                if ln is not None and lanes[ln] is None and product[ln] is None:
                    lanes[ln] = i
                    room -= 1
                    kind[i] = KEEP if kind[i] == LOAD else MULACC
                elif ready_at[i] <= t:
                    fresh.append(i)
                    room -= 1
            free = [ln for ln in range(width) if lanes[ln] is None and product[ln] is None]
            for i, ln in zip(fresh, free):
                lanes[ln] = i
            for ln, i in enumerate(lanes):
                if i is not None:
                    if kind[i] in (KEEP, MULACC) and not read[chain[i]]:
                        store[chain[i]] = False
                    lane_acc[ln], when[i], lane_of[i] = i, t, ln
                    product[ln] = next((j for j, k in succ[i] if k == "C" and ops[j][5] == MULACC), None)
            rows.append(("F", lanes))
            placed = [i for i in lanes if i is not None]
        done += len(placed)
        waiting.difference_update(placed)
        for i in placed:
            for j, _ in succ[i]:
                open_preds[j] -= 1
                if not open_preds[j]:
                    waiting.add(j)
                    ready_at[j] = earliest(j)
        if rows[-1][0] == "F":
            t += 1
    return Schedule(rows, kind, store)


def encode(ops, sch: Schedule, offset, const_offset, zero: int) -> list[list[tuple[int, int]]]:
    """Rows of (word 0, word 1) per lane; `offset` and `const_offset` give bytes."""
    idle = (zero | zero << 16, zero | C_KEEP | A_NEG)   # acc = -0 * 0 + acc
    out = []
    for what, lanes in sch.rows:
        row = []
        for i in lanes:
            if what == "D":
                row.append((zero | A_RECIP | zero << 16, zero if i is None else offset(ops[i][1]) | D_STORE))
                continue
            if i is None:
                row.append(idle)
                continue
            _, d, a, b, neg, _ = ops[i]
            k = sch.kind[i]
            const = isinstance(b, tuple)
            w0 = (zero if k == MULACC else offset(a)) | (const_offset(b[1]) if const else offset(b)) << 16
            w1 = (offset(d) | ADDEND[k]) + (D_STORE if sch.store[i] else 0)
            row.append((w0, w1 + (B_CONST if const else 0) + (A_NEG if neg else 0)))
        out.append(row)
        if what == "D":
            out += [[idle] * len(lanes)] * (UNROLL - 1)
    width = len(sch.rows[0][1])
    while len(out) % UNROLL:
        out.append([idle] * width)
    return out


# ----------------------------------------------------------------------------- a mechanism's programs

def mechanism(mech: str) -> tuple[Mechanism, SparseMech]:
    """The reactions of a manifest and the sparse structure they give."""
    d = json.loads((PKG / "mechs" / mech / "manifest.json").read_text())
    mx = d["mxprd"]
    m = Mechanism(mech, d["nspec"], d["nrxns"], mxprd=mx)
    for r in d["reactions"]:
        m.irr.append([s + 1 for s in r["reactants"]] + [0] * (3 - r["nreact"])
                     + [s + 1 for s in r["products"]] + [0] * (mx - r["nprdct"]))
        m.sc.append(list(r["sc"]) + [0.0] * (mx - len(r["sc"])))
        m.nreact.append(r["nreact"])
        m.nprdct.append(r["nprdct"])
        m.irxbits.append(2 if r["photolytic"] else 0)
    sp = build_sparse(m)
    if sp.active != d["active"] or sp.iarray != d["iarray"] or sp.inew2old != d["inew2old"]:
        raise ValueError(f"{mech}: the manifest's structure is not its reactions'")
    return m, sp


def rates(P: Program, m, sp, src: str):
    """X_r = RKI_r times the reactants' concentrations (rbfeval.F:88-127)."""
    for r in sp.active[0]:
        P.fma(f"X{r}", f"R{r}", f"{src}{sp.irm2[r][0]}", init=NEG0)
        for q in range(1, m.nreact[r]):
            P.fma(f"X{r}", None, f"{src}{sp.irm2[r][q]}", init=MULACC)


def tendency(P: Program, m, sp, dst: str):
    """Each species' loss and production terms in reaction order (rbfeval.F:129-151)."""
    terms: dict[int, list] = {}
    for r in sp.active[0]:
        for q in range(m.nreact[r]):
            terms.setdefault(sp.irm2[r][q], []).append((r, -1.0))
        for p in range(m.nprdct[r]):
            terms.setdefault(sp.irm2[r][3 + p], []).append((r, m.sc[r][p]))
    for s in range(sp.ischan):
        if s not in terms:
            P.fma(f"{dst}{s}", "Z", ("c", 1.0), init=NEG0)
        for t, (r, c) in enumerate(terms.get(s, [])):
            P.fma(f"{dst}{s}", f"X{r}", ("c", c), init=NEG0 if t == 0 else LOAD)


def partials(P: Program, m, sp):
    """Partial-derivative products of 2- and 3-reactant reactions (rbjacob.F:112-143)."""
    for r in sp.active[0]:
        y = [f"Y{sp.irm2[r][q]}" for q in range(m.nreact[r])]
        if m.nreact[r] == 2:
            P.fma(f"E{r}_0", f"R{r}", y[1], init=NEG0)
            P.fma(f"E{r}_1", f"R{r}", y[0], init=NEG0)
        elif m.nreact[r] == 3:
            for q, (u, v) in enumerate(((1, 2), (0, 2), (1, 0))):
                P.fma(f"E{r}_{q}", f"R{r}", y[u], init=NEG0)
                P.fma(f"E{r}_{q}", None, y[v], init=MULACC)


def iteration_matrix(P: Program, m, sp):
    """J - I/(gamma h) and its LU factors, row by row (rbjacob.F, rbdecomp.F); the reciprocal of
    a pivot takes its place.  An entry without terms starts at -0.0 (the sequential routine's
    0.0: only the sign of a zero product could tell them apart)."""
    jpt, terms = sp.jarraypt[0], _jac_terms(m, sp, 0)
    for i in range(sp.ischan):
        cols = [st for st, _ in sp.lower[0][i]] + [jpt[(i, i)]] + [st for st, _ in sp.upper[0][i]]
        empty = set()
        for st in cols:
            tl = terms.get(st, [])
            for q, (r, ial, coef, sign) in enumerate(tl):
                a = f"R{r}" if m.nreact[r] == 1 else f"E{r}_{ial}"
                P.fma(f"A{st}", a, ("c", -1.0 if sign < 0 else 1.0 if coef is None else coef),
                      init=NEG0 if q == 0 else LOAD)
            if not tl:
                empty.add(st)

        def first(st):
            if st in empty:
                empty.discard(st)
                return NEG0
            return LOAD
        di = jpt[(i, i)]
        P.fma(f"A{di}", "G", ("c", -1.0), init=first(di))
        for st, k in sp.lower[0][i]:
            if st in empty:
                raise ValueError("an entry of L without terms or updates")
            P.fma(f"A{st}", f"A{st}", f"A{jpt[(k, k)]}", init=NEG0)
            for st_kj, j in sp.upper[0][k]:
                o = jpt[(i, j)]
                P.fma(f"A{o}", f"A{st}", f"A{st_kj}", neg=True, init=first(o))
        if empty:
            raise ValueError("an entry of U without terms or updates")
        P.recip(f"A{di}")


def substitution(P: Program, m, sp, v: str):
    """Forward and backward substitution (rbsolve.F)."""
    for i in range(sp.ischan):
        for st, j in sp.lower[0][i]:
            P.fma(f"{v}{i}", f"A{st}", f"{v}{j}", neg=True)
    for i in range(sp.ischan - 1, -1, -1):
        terms = sp.upper[0][i]
        for st, j in terms:
            P.fma(f"{v}{i}", f"A{st}", f"{v}{j}", neg=True)
        P.fma(f"{v}{i}", f"{v}{i}", f"A{sp.jarraypt[0][(i, i)]}", init=NEG0)


def ros3_programs(m, sp) -> dict[str, Program]:
    """Of one ROS3 attempt: stage1 (f(Y), the iteration matrix, its factors and the first solve,
    in V, for the right-hand side f(Y): -K1), rhs (T = f(T)) and solve (V)."""
    p = {"stage1": Program(), "rhs": Program(), "solve": Program()}
    rates(p["stage1"], m, sp, "Y")
    tendency(p["stage1"], m, sp, "V")
    partials(p["stage1"], m, sp)
    iteration_matrix(p["stage1"], m, sp)
    substitution(p["stage1"], m, sp, "V")
    rates(p["rhs"], m, sp, "T")
    tendency(p["rhs"], m, sp, "T")
    substitution(p["solve"], m, sp, "V")
    return p


class Ros3Layout:
    """Element offsets (doubles) of a cell's state in shared memory.  The partial-derivative
    products are needed only until the matrix is formed: they lie over the stage vectors,
    then over spare room, then over rates (whose last use the schedule then waits for)."""

    def __init__(self, m, sp, consts: int):
        n, nr = m.nspec, m.nrxns
        self.at = {}
        off = 0
        for v in "YVKLT":                     # Y, V, K1, K2, T
            self.at.update({f"{v}{i}": off + i for i in range(n)})
            setattr(self, v.lower(), off)
            off += n
        self.rki = off
        self.at.update({f"R{r}": off + r for r in range(nr)})
        off += nr
        self.x = off
        self.at.update({f"X{r}": off + r for r in range(nr)})
        off += nr
        self.lu = off
        self.at.update({f"A{st}": off + st - 1 for st in range(1, sp.iarray[0] + 1)})
        off += sp.iarray[0]
        self.g, self.z = off, off + 1
        self.at.update(G=off, Z=off + 1)
        off += 2
        ex = [f"E{r}_{q}" for r in sp.active[0] if m.nreact[r] >= 2 for q in range(m.nreact[r])]
        room = SMEM_MAX - TABLE_SMEM - 8 * consts
        cells = room // (8 * off)
        spare = room // (8 * cells) - off
        slots = list(range(self.k, self.k + 3 * n)) + list(range(off, off + max(0, min(spare, len(ex) - 3 * n))))
        slots += list(range(self.x, self.x + nr))
        self.alias = {e: slots[q] for q, e in enumerate(ex)}
        self.at.update(self.alias)
        self.elems = max(off, max(slots[:len(ex)], default=0) + 1)
        self.cells = room // (8 * self.elems)

    def place(self, ops):
        """The operations with elements named by their places, so that elements that share a
        place depend on one another."""
        def at(e):
            return e if e is None or isinstance(e, tuple) else self.at[e]
        return [(k, at(d), at(a), at(b), neg, init) for k, d, a, b, neg, init in ops]


WIDTH = 32           # lanes of a cell (16, two cells to a warp: 8 % slower, the rows are fewer but wait longer)


def ros3_tables(mech: str, width: int = WIDTH):
    """(layout, constants, {program: encoded rows})."""
    m, sp = mechanism(mech)
    progs = ros3_programs(m, sp)
    consts = sorted({op[3][1] for p in progs.values() for op in p.ops if isinstance(op[3], tuple)})
    lay = Ros3Layout(m, sp, len(consts))
    cof = {c: 8 * q for q, c in enumerate(consts)}
    tables = {}
    for name, p in progs.items():
        ops = lay.place(p.ops)
        tables[name] = encode(ops, schedule(ops, width), lambda e: 8 * e, lambda c: cof[c], 8 * lay.z)
    return lay, consts, tables


def sources(mech: str) -> dict[str, str]:
    """<mech>_coop.cuh (sizes) and <mech>_coop.cu (tables)."""
    lay, consts, tables = ros3_tables(mech)
    banner = [f"// Generated by cmaq_gb300.mechgen.coop from mechs/{mech}/manifest.json.  Do not edit."]
    ns = f"mech_{mech}"
    h = banner + ["// Sizes and tables of the cooperative ROS3 kernel (csrc/coop.cuh).", "#pragma once",
                  "#include <cuda_runtime.h>", f"namespace {ns} {{",
                  f"extern __device__ const double c_coop_const[{len(consts)}];"]
    c = banner + [f'#include "{mech}_coop.cuh"', f"namespace {ns} {{",
                  f"__device__ const double c_coop_const[{len(consts)}] = {{{', '.join(map(c_double, consts))}}};"]
    rows = []                # programs one after the other, each from the start of a chunk
    for table in tables.values():
        rows += table
        rows += [[(0, 0)] * WIDTH] * (-len(rows) % CHUNK)
    h.append(f"extern __device__ const uint2 c_coop_rows[{len(rows) * WIDTH}];")
    c.append(f"__device__ __align__(128) const uint2 c_coop_rows[{len(rows) * WIDTH}] = {{")
    c += ["  " + ", ".join(f"{{0x{a:x}u, 0x{b:x}u}}" for a, b in row) + "," for row in rows]
    c.append("};")
    h += ["struct Coop {",
          f"    static constexpr int ELEMS = {lay.elems}, NCONST = {len(consts)}, MAX_CELLS = {lay.cells};",
          f"    static constexpr int Y = {lay.y}, V = {lay.v}, K1 = {lay.k}, K2 = {lay.l}, T = {lay.t};",
          f"    static constexpr int RKI = {lay.rki}, G = {lay.g}, Z = {lay.z};",
          f"    static constexpr int CHUNK = {CHUNK}, TABLE_SMEM = {TABLE_SMEM};",
          "    static __device__ __forceinline__ const double* constants() { return c_coop_const; }",
          "    static __device__ __forceinline__ const uint2* rows() { return c_coop_rows; }",
          "    static constexpr int " + ", ".join(f"{n.upper()}_ROWS = {len(t)}" for n, t in tables.items()) + ";"]
    h += ["};", f"}}  // namespace {ns}"]
    c.append(f"}}  // namespace {ns}")
    return {f"{mech}_coop.cuh": "\n".join(h) + "\n", f"{mech}_coop.cu": "\n".join(c) + "\n"}


def write(mech: str, out: Path | None = None) -> None:
    out = out or PKG / "csrc" / "gen"
    for name, text in sources(mech).items():
        (out / name).write_text(text)


if __name__ == "__main__":
    for mech_ in ("cb6r5_ae7_aq", "cracmm2"):
        write(mech_)
