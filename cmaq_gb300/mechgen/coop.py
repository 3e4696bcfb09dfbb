"""Lane schedules of the cooperative kernels (a warp's lanes integrate one cell in shared memory).

A routine of the cell's solver (rates, right-hand side, Jacobian, factorisation, triangular
solves) is written down as the sequence of its scalar operations, every one of the form
``acc = +-x[a] * x[b] + c`` or a special one (quotient, square root, maximum, sign), in the
order of the generated sequential code.  `schedule` deals these operations out to W lanes, row by row: a row is one operation
per lane, and an operation is placed as soon as the values that it reads are there, longest
remaining chain first.  No operation is changed and no sum is reordered: each element of the
cell's state goes through the same operations on the same values as in the sequential
routine, so the results have the same bits.

The kernel (csrc/coop.cuh) loads the operands of row t + 2 before it stores the results of
row t, so a value is read at the earliest three rows after the one that computed it, unless
the same lane goes on with it in its accumulator.  The kernel goes through UNROLL rows
without a branch (a test for special rows in each row took 50 of its 165 cycles); a row of
special operations takes the place of such a block.

Tables are made from the mechanism's manifest alone:

    python -m cmaq_gb300.mechgen.coop
"""
from __future__ import annotations

import json
import math
import re
from dataclasses import dataclass, field
from pathlib import Path

from .emit_common import c_double
from .emit_cuda import Layout, _jac_terms
from .fortran_tables import Mechanism
from .sparse import SparseMech, build_sparse

PKG = Path(__file__).resolve().parents[1]
VISIBLE = 3          # rows from the one that computes a value to the first that may load it
CHUNK = 28           # rows of a table that are fetched together (more would cost CRACMM2 a cell)
AHEAD = 3            # rows past a chunk's end whose words the kernel may look at
UNROLL = 4           # rows that the kernel goes through without a branch: a row of special
                     # operations comes only after a multiple of it, in a block of its own
SLACK = 3            # how much shorter a special operation's chain may be than the longest one
SMEM_MAX = 227 * 1024
TABLE_SMEM = 2 * (CHUNK + AHEAD) * 32 * 8 + 64   # two chunks in flight, each with rows of zeros, and their barriers

# where an operation's addend comes from: the element itself, the lane's accumulator, -0.0
# (the exact identity of an addition: a product alone); MULACC: acc * x[b]; LOADACC: acc * x[b] + x[d]
LOAD, KEEP, NEG0, MULACC, LOADACC = range(5)
# special operations: 1 / x[b], x[a] / x[b], sqrt(x[b]), fmax(x[a], x[b]), copysign(1, x[b])
RCP, DIV, SQRT, MAX, SIGN = range(1, 6)
# encoding: word 0 = offset of a | offset of b << 16, word 1 = offset of d, and flags.
# Offsets are bytes (multiples of 8) into the cell's state; b may be a constant's offset.
# Word 1 of a special operation (A_SPECIAL in word 0) holds its kind in place of the addend's.
A_SPECIAL, C_LOAD, C_KEEP, C_MULACC = 1, 1, 2, 4
D_STORE, B_CONST, A_NEG = 1 << 16, 1 << 17, 1 << 31
ADDEND = {LOAD: C_LOAD, KEEP: C_KEEP, NEG0: 0, MULACC: C_MULACC, LOADACC: C_LOAD | C_MULACC}


@dataclass
class Program:
    """Operations in sequential order: ("F", d, a, b, negate a, addend) or ("D", d, a, b, False,
    special kind).  Elements are names; b may be a ("c", value) constant."""
    ops: list = field(default_factory=list)

    def fma(self, d, a, b, neg=False, init=LOAD):
        self.ops.append(("F", d, a, b, neg, init))

    def special(self, kind, d, a, b):
        self.ops.append(("D", d, a, b, False, kind))


def dependencies(ops) -> list[list[tuple[int, str]]]:
    """Per operation its predecessors: "R" reads a value it wrote, "C" goes on with its sum,
    "W" reads what this one overwrites, "O" wrote the same element before."""
    last, readers, preds = {}, {}, []
    for i, (kind, d, a, b, _, init) in enumerate(ops):
        p = []
        scaled = kind == "F" and init == NEG0 and a == d      # d = d * x[b]
        for e in [b] if kind == "F" and init == MULACC or scaled else [a, b]:
            if e is None or isinstance(e, tuple):
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


def schedule(ops, width: int, special_cost: int = 3) -> Schedule:
    """List scheduling, the longest remaining dependence chain first."""
    n = len(ops)
    preds = dependencies(ops)
    succ = [[] for _ in range(n)]
    chain = [None] * n
    factor = [None] * n                  # the operation that forms the factor a of a sum's term
    for i, ps in enumerate(preds):
        for p, k in ps:
            succ[p].append((i, k))
            if k == "C":
                chain[i] = p
            if k == "R" and ops[i][0] == ops[p][0] == "F" and ops[i][5] == LOAD and ops[p][1] == ops[i][2] != ops[i][3]:
                factor[i] = p

    def latency(p, k, i):
        if k in "WO":
            return 0
        if ops[p][0] == "D" or ops[i][0] == "D":
            return 1
        return VISIBLE

    prio = [0] * n
    for i in range(n - 1, -1, -1):
        own = special_cost if ops[i][0] == "D" else 1
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
    kind = [op[5] for op in ops]         # of special operations: not read
    store = [True] * n
    rows, t, done = [], 0, 0

    def earliest(i, skip=None):
        e = 0
        for p, k in preds[i]:
            if (p, k) != skip:
                e = max(e, when[p] + latency(p, k, i))
        return e

    ready_at = {i: 0 for i in waiting}
    while done < n:
        ready = [i for i in waiting if ready_at[i] <= t]
        specials = sorted((i for i in ready if ops[i][0] == "D"), key=lambda i: (-prio[i], i))[:width]
        # operations that a lane can go on with in its accumulator
        goes_on = {i for i in waiting if chain[i] is not None and ops[i][0] == ops[chain[i]][0] == "F"
                   and lane_acc[lane_of[chain[i]]] == chain[i] and earliest(i, (chain[i], "C")) <= t}
        # or whose factor a lane has just formed there
        takes = {i for i in waiting if factor[i] is not None and i not in goes_on and ready_at[i] > t
                 and lane_acc[lane_of[factor[i]]] == factor[i] and earliest(i, (factor[i], "R")) <= t}
        cand = sorted(goes_on.union(takes, (i for i in ready if ops[i][0] == "F" and ops[i][5] != MULACC)),
                      key=lambda i: (-prio[i], i))
        if specials and t % UNROLL == 0 and (not cand or prio[specials[0]] >= prio[cand[0]] - SLACK):
            rows.append(("D", specials + [None] * (width - len(specials))))
            for lane, i in enumerate(specials):
                when[i], lane_of[i] = t - 1, lane
            placed = specials
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
                ln = lane_of[chain[i]] if i in goes_on else lane_of[factor[i]] if i in takes else None
                if ln is not None and lanes[ln] is None and product[ln] is None:
                    lanes[ln] = i
                    room -= 1
                    kind[i] = LOADACC if i in takes else KEEP if kind[i] == LOAD else MULACC
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
            if i is None:
                row.append(idle if what == "F" else (zero | A_SPECIAL | zero << 16, zero))
                continue
            _, d, a, b, neg, special = ops[i]
            const = isinstance(b, tuple)
            if what == "D":
                row.append(((zero if a is None else offset(a)) | A_SPECIAL
                            | (const_offset(b[1]) if const else offset(b)) << 16,
                            offset(d) | special | D_STORE | (B_CONST if const else 0)))
                continue
            k = sch.kind[i]
            w0 = (zero if k in (MULACC, LOADACC) else offset(a)) | (const_offset(b[1]) if const else offset(b)) << 16
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


def partials(P: Program, m, sp, src: str = "Y"):
    """Partial-derivative products of 2- and 3-reactant reactions (rbjacob.F:112-143)."""
    for r in sp.active[0]:
        y = [f"{src}{sp.irm2[r][q]}" for q in range(m.nreact[r])]
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

        di = jpt[(i, i)]
        P.fma(f"A{di}", "G", ("c", -1.0), init=NEG0 if di in empty else LOAD)
        empty.discard(di)
        eliminate(P, sp, i, empty)


def eliminate(P: Program, sp, i: int, empty: set):
    """Row i's elimination by the rows above; `empty`: its entries without terms, not yet formed."""
    jpt = sp.jarraypt[0]
    for st, k in sp.lower[0][i]:
        if st in empty:
            raise ValueError("an entry of L without terms or updates")
        P.fma(f"A{st}", f"A{st}", f"A{jpt[(k, k)]}", init=NEG0)
        for st_kj, j in sp.upper[0][k]:
            o = jpt[(i, j)]
            P.fma(f"A{o}", f"A{st}", f"A{st_kj}", neg=True, init=NEG0 if o in empty else LOAD)
            empty.discard(o)
    if empty:
        raise ValueError("an entry of U without terms or updates")
    P.special(RCP, f"A{jpt[(i, i)]}", None, f"A{jpt[(i, i)]}")


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


def place(ops, where):
    """The operations with elements named by their places, so that elements that share a place
    depend on one another."""
    def at(e):
        return e if e is None or isinstance(e, tuple) else where[e]
    return [(k, at(d), at(a), at(b), neg, init) for k, d, a, b, neg, init in ops]


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
        return place(ops, self.at)


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


# ----------------------------------------------------------------------------- discrete adjoint of ROS3

def transposed_substitution(P: Program, sp, v: str):
    """A^T x = b in place, U^T by ascending rows, then L^T by descending ones (emit_cuda._solve_t_chunks)."""
    n = sp.ischan
    col_u, col_l = [[] for _ in range(n)], [[] for _ in range(n)]
    for k in range(n):
        for st, j in sp.upper[0][k]:
            col_u[j].append((k, st))
        for st, j in sp.lower[0][k]:
            col_l[j].append((k, st))
    for i in range(n):
        for k, st in sorted(col_u[i]):
            P.fma(f"{v}{i}", f"A{st}", f"{v}{k}", neg=True)
        P.fma(f"{v}{i}", f"{v}{i}", f"A{sp.jarraypt[0][(i, i)]}", init=NEG0)
    for i in range(n - 1, -1, -1):
        for k, st in sorted(col_l[i]):
            P.fma(f"{v}{i}", f"A{st}", f"{v}{k}", neg=True)


def stoich_sum(P: Program, m, sp, r: int, vec: str, d: str):
    """d = reaction r's net stoichiometry times vec (emit_cuda._stoich_sum)."""
    for p in range(m.nprdct[r]):
        P.fma(d, f"{vec}{sp.irm2[r][3 + p]}", ("c", m.sc[r][p]), init=NEG0 if p == 0 else LOAD)
    for i in range(m.nreact[r]):
        P.fma(d, f"{vec}{sp.irm2[r][i]}", ("c", 1.0), neg=True, init=NEG0 if not m.nprdct[r] and i == 0 else LOAD)


def jtv(P: Program, m, sp, y: str, out: str, temp):
    """out += J(y)^T P and W_r += w_r R_r(y) (emit_cuda._adj_jtv); w_r and then RKI_r w_r in X_r."""
    for r in sp.active[0]:
        nre = m.nreact[r]
        if nre == 0 and m.nprdct[r] == 0:
            continue
        stoich_sum(P, m, sp, r, "P", f"X{r}")
        P.fma(f"X{r}", f"X{r}", f"R{r}", init=NEG0)
        a = [sp.irm2[r][i] for i in range(nre)]
        if nre == 0:
            P.fma(f"W{r}", f"X{r}", ("c", 1.0))
        elif nre == 1:
            P.fma(f"{out}{a[0]}", f"X{r}", ("c", 1.0))
            P.fma(f"W{r}", f"X{r}", f"{y}{a[0]}")
        elif nre == 2:
            P.fma(f"{out}{a[0]}", f"X{r}", f"{y}{a[1]}")
            P.fma(f"{out}{a[1]}", f"X{r}", f"{y}{a[0]}")
            P.fma(f"X{r}", f"X{r}", f"{y}{a[0]}", init=NEG0)
            P.fma(f"W{r}", f"X{r}", f"{y}{a[1]}")
        else:
            t = temp()
            P.fma(t, f"X{r}", f"{y}{a[1]}", init=NEG0)
            P.fma(f"{out}{a[0]}", t, f"{y}{a[2]}")
            P.fma(f"X{r}", f"X{r}", f"{y}{a[0]}", init=NEG0)
            P.fma(f"{out}{a[1]}", f"X{r}", f"{y}{a[2]}")
            P.fma(f"{out}{a[2]}", f"X{r}", f"{y}{a[1]}")
            P.fma(f"X{r}", f"X{r}", f"{y}{a[1]}", init=NEG0)
            P.fma(f"W{r}", f"X{r}", f"{y}{a[2]}")


def hess3(P: Program, m, sp, temp):
    """The stage solves' second-order terms (emit_cuda._adj_hess3): nu in V, C, D, the stages in K, L, Q."""
    for r in sp.active[0]:
        nre = m.nreact[r]
        if nre == 0:
            continue
        a = [sp.irm2[r][i] for i in range(nre)]
        w = [temp() for _ in range(3)]
        for v, x in zip("VCD", w):
            stoich_sum(P, m, sp, r, v, x)
        wk = []
        for s in a:
            wk.append(temp())
            for v, x, init in zip("KLQ", w, (NEG0, LOAD, LOAD)):
                P.fma(wk[-1], x, f"{v}{s}", init=init)
        y = [f"Y{s}" for s in a]

        def pair(u, i, v, j):        # u * wk_i + v * wk_j
            t = temp()
            P.fma(t, v, wk[j], init=NEG0)
            P.fma(t, u, wk[i])
            return t
        if nre == 1:
            P.fma(f"W{r}", f"R{r}", wk[0], neg=True)
        elif nre == 2:
            P.fma(f"W{r}", f"R{r}", pair(y[1], 0, y[0], 1), neg=True)
            P.fma(f"M{a[0]}", f"R{r}", wk[1], neg=True)
            P.fma(f"M{a[1]}", f"R{r}", wk[0], neg=True)
        else:
            t = temp()
            P.fma(t, y[0], y[1], init=NEG0)
            P.fma(t, t, wk[2], init=NEG0)
            for u, v, k in ((0, 2, 1), (1, 2, 0)):
                q = temp()
                P.fma(q, y[u], y[v], init=NEG0)
                P.fma(t, q, wk[k])
            P.fma(f"W{r}", f"R{r}", t, neg=True)
            P.fma(f"M{a[0]}", f"R{r}", pair(y[2], 1, y[1], 2), neg=True)
            P.fma(f"M{a[1]}", f"R{r}", pair(y[2], 0, y[0], 2), neg=True)
            P.fma(f"M{a[2]}", f"R{r}", pair(y[1], 0, y[0], 1), neg=True)


def adjoint_programs(m, sp) -> tuple[dict[str, Program], list, list]:
    """Of the step and its adjoint (csrc/adj_coop.cuh): stage1, rhs and solve as ros3_programs' with the
    emission tendency N added to f, tsolve (V), jtv (V += J(T)^T P) and gradient (M += J(Y)^T P, then
    the second-order terms).  Returns also the temporaries of jtv and of gradient."""
    p = {k: Program() for k in ("stage1", "rhs", "solve", "tsolve", "jtv", "gradient")}
    for name, src, dst in (("stage1", "Y", "V"), ("rhs", "T", "T")):
        rates(p[name], m, sp, src)
        tendency(p[name], m, sp, dst)
        for i in range(sp.ischan):
            p[name].fma(f"{dst}{i}", f"N{i}", ("c", 1.0))
    partials(p["stage1"], m, sp)
    iteration_matrix(p["stage1"], m, sp)
    substitution(p["stage1"], m, sp, "V")
    substitution(p["solve"], m, sp, "V")
    transposed_substitution(p["tsolve"], sp, "V")
    temps = {"j": [], "h": []}

    def temp(kind):
        temps[kind].append(f"{kind}{len(temps[kind])}")
        return temps[kind][-1]
    jtv(p["jtv"], m, sp, "T", "V", lambda: temp("j"))
    jtv(p["gradient"], m, sp, "Y", "M", lambda: temp("h"))
    hess3(p["gradient"], m, sp, lambda: temp("h"))
    return p, temps["j"], temps["h"]


class AdjointLayout:
    """Element offsets (doubles) of a cell's state.  The partial-derivative products lie over vectors that
    are formed after the factors; the gradient's temporaries over the factors, in turn."""

    VECTORS = dict(y="Y", v="V", k1="K", k2="L", t="T", k3="Q", nu2="C", nu3="D", phi="P", lam="M", emis="N")

    def __init__(self, m, sp, jtemps, htemps):
        n, nr = m.nspec, m.nrxns
        self.at, off = {}, 0
        for name, v in self.VECTORS.items():
            self.at.update({f"{v}{i}": off + i for i in range(n)})
            setattr(self, name, off)
            off += n
        for name, v in (("rki", "R"), ("x", "X"), ("gk", "W")):
            self.at.update({f"{v}{r}": off + r for r in range(nr)})
            setattr(self, name, off)
            off += nr
        self.lu = off
        self.at.update({f"A{st}": off + st - 1 for st in range(1, sp.iarray[0] + 1)})
        off += sp.iarray[0]
        self.g, self.z = off, off + 1
        self.at.update(G=off, Z=off + 1)
        off += 2
        self.at.update({e: off + q for q, e in enumerate(jtemps)})
        self.elems = off + len(jtemps)
        ex = [f"E{r}_{q}" for r in sp.active[0] if m.nreact[r] >= 2 for q in range(m.nreact[r])]
        if len(ex) > 7 * n:
            raise ValueError("no room for the partial-derivative products")
        self.at.update({e: self.k1 + q for q, e in enumerate(ex)})          # K1 ... PHI
        self.at.update({e: self.lu + q % sp.iarray[0] for q, e in enumerate(htemps)})
        if 8 * self.elems > 1 << 16:
            raise ValueError("an operation's offsets have 16 bits")


def adjoint_tables(mech: str, width: int = WIDTH):
    """(layout, constants, {program: encoded rows})."""
    m, sp = mechanism(mech)
    progs, jtemps, htemps = adjoint_programs(m, sp)
    lay = AdjointLayout(m, sp, jtemps, htemps)
    consts = sorted({op[3][1] for p in progs.values() for op in p.ops if isinstance(op[3], tuple)})
    cof = {c: 8 * q for q, c in enumerate(consts)}
    tables = {}
    for name, p in progs.items():
        ops = place(p.ops, lay.at)
        tables[name] = encode(ops, schedule(ops, width), lambda e: 8 * e, lambda c: cof[c], 8 * lay.z)
    return lay, consts, tables


class GearLayout:
    """Places of SMVGEAR's programs in the one-cell workspace of the Gear kernels (emit_cuda.Layout):
    a pivot's reciprocal takes the pivot's place, the concentrations with CEFF's zeros the place of
    VDIAG, and the coefficients times R1DELT that of the rates, which are formed after the
    matrix, and of the scratch array.  R1DELT, 0 and 1 lie before the workspace."""

    WORKSPACE = 4

    def __init__(self, m, sp, coefs):
        lay = Layout(m, sp)
        n, nr, w = m.nspec, m.nrxns, self.WORKSPACE
        self.q = w + lay.vdiag
        self.at = dict(H=0, Z=1, O=2)
        for v, off in (("Y", lay.y), ("U", lay.ydot), ("Q", lay.vdiag)):
            self.at.update({f"{v}{i}": w + off + i for i in range(n)})
        for v, off in (("R", lay.rki), ("X", lay.rxrat)):
            self.at.update({f"{v}{r}": w + off + r for r in range(nr)})
        self.at.update({f"E{r}_{q}": w + off for (r, q), off in lay.ex.items()})
        self.at.update({f"A{st}": w + lay.lu + st for st in range(1, sp.iarray[0] + 1)})
        slots = list(range(lay.rxrat, lay.rxrat + nr)) + list(range(lay.yp, lay.yp + n))
        if len(coefs) > len(slots):
            raise ValueError("no room for the scaled coefficients")
        self.at.update({f"S{q}": w + slots[q] for q in range(len(coefs))})
        self.elems = w + lay.gear_total
        if 8 * max(self.at.values()) >= 1 << 16:
            raise ValueError("an operation's offsets have 16 bits")


def gear_programs(m, sp) -> tuple[dict[str, Program], list]:
    """Of one SMVGEAR evaluation: predictor (P = I - ASN1*DELT*J at the concentrations Q, with R1DELT =
    -ASN1*DELT in H, and its factors: grpderiv.F:131-226, grdecomp.F), rhs (U = f(Y), grsubfun.F) and
    solve (U, grbacksub.F).  Returns the programs and the coefficients that are scaled by R1DELT."""
    terms = _jac_terms(m, sp, 0)
    coefs = sorted({c for tl in terms.values() for _, _, c, sign in tl if sign > 0 and c is not None})
    slot = {c: f"S{q}" for q, c in enumerate(coefs)}
    p = {"predictor": Program(), "rhs": Program(), "solve": Program()}
    P = p["predictor"]
    for c in coefs:
        P.fma(slot[c], "H", ("c", c), init=NEG0)
    partials(P, m, sp, "Q")
    jpt = sp.jarraypt[0]
    for i in range(sp.ischan):
        di = jpt[(i, i)]
        empty = set()
        for st in [st for st, _ in sp.lower[0][i]] + [di] + [st for st, _ in sp.upper[0][i]]:
            if st == di:
                P.fma(f"A{st}", "O", ("c", 1.0), init=NEG0)
            elif not terms.get(st):
                empty.add(st)
            for q, (r, ial, coef, sign) in enumerate(terms.get(st, [])):
                a = f"R{r}" if m.nreact[r] == 1 else f"E{r}_{ial}"
                P.fma(f"A{st}", a, "H" if sign < 0 or coef is None else slot[coef], neg=sign < 0,
                      init=NEG0 if q == 0 and st != di else LOAD)
        eliminate(P, sp, i, empty)
    rates(p["rhs"], m, sp, "Y")
    tendency(p["rhs"], m, sp, "U")
    substitution(p["solve"], m, sp, "U")
    return p, coefs


def gear_tables(mech: str, width: int = WIDTH):
    """(layout, constants, {program: encoded rows})."""
    m, sp = mechanism(mech)
    progs, coefs = gear_programs(m, sp)
    lay = GearLayout(m, sp, coefs)
    consts = sorted({op[3][1] for p in progs.values() for op in p.ops if isinstance(op[3], tuple)})
    cof = {c: 8 * q for q, c in enumerate(consts)}
    tables = {}
    for name, p in progs.items():
        ops = place(p.ops, lay.at)
        tables[name] = encode(ops, schedule(ops, width), lambda e: 8 * e, lambda c: cof[c], 8 * lay.at["Z"])
    return lay, consts, tables


# ----------------------------------------------------------------------------- EBI
# HRRATES, HRG1-HRG4 and HRPRODLOSS as straight-line C (gen/<mech>_ebi.cu), turned into operations.
# Their products and sums are rounded one by one (no fused multiply-add in the EBI code), so a term
# takes a product and an addition, x * 1.0 + acc, unless its factor is a power of two: such a
# product is exact, and the fused operation gives the same sum.

_TOKEN = re.compile(r"\s*(?:(0x[0-9a-f.]+p[-+]?\d+|\d+\.?\d*(?:e[-+]?\d+)?)|(EBI_\w+)\((\d+)\)"
                    r"|(\w+)\[(\d+) \* KQ_S\]|(\w+)|(.))")
_EBI_ARRAYS = {"EBI_YC": "C", "EBI_YC0": "B", "EBI_YCP": "P", "EBI_RKI": "R", "EBI_RXRAT": "X", "EBI_PROD": "M",
               "EBI_LOSS": "L", "EBI_PNEG": "N"}


def _parse(text: str, arrays=None):
    """An expression of numbers, elements, + - * /, fmax, sqrt, fabs and copysign as nested tuples;
    `arrays`: the elements' prefix per array of the KPP code."""
    toks = []
    for num, arr, idx, karr, kidx, name, ch in _TOKEN.findall(text):
        toks.append(("num", float.fromhex(num) if "x" in num else float(num)) if num else
                    ("el", _EBI_ARRAYS[arr] + idx) if arr else ("el", arrays[karr] + kidx) if karr else
                    ("name", name) if name else (ch, None))
    pos = 0

    def peek():
        return toks[pos][0] if pos < len(toks) else None

    def take(kind=None):
        nonlocal pos
        t = toks[pos]
        if kind is not None and t[0] != kind:
            raise ValueError(f"expected {kind} in {text}")
        pos += 1
        return t

    def atom():
        t = take()
        if t[0] in ("num", "el"):
            return t
        if t[0] == "-":
            e = atom()
            return ("num", -e[1]) if e[0] == "num" else ("neg", e)
        if t[0] == "(":
            e = add()
            take(")")
            return e
        if t[0] == "name" and peek() == "(":
            take("(")
            args = [add()]
            while peek() == ",":
                take(",")
                args.append(add())
            take(")")
            return (t[1], *args)
        if t[0] == "name":
            return ("el", t[1])
        raise ValueError(f"unexpected {t} in {text}")

    def mul():
        e = atom()
        while peek() in ("*", "/"):
            op = take()[0]
            e = (op, e, atom())
        return e

    def add():
        e = mul()
        while peek() in ("+", "-"):
            op = take()[0]
            e = (op, e, mul())
        return e

    e = add()
    if pos != len(toks):
        raise ValueError(f"trailing text in {text}")
    return e


class _Emit:
    """Expressions to operations; temporaries come from a ring of places."""

    def __init__(self, P: Program, temps: int, memo: bool = False):
        self.P, self.temps, self.next = P, temps, 0
        self.memo = {} if memo else None     # products that keep their place (their factors do not change)

    def temp(self):
        self.next += 1
        return f"t{(self.next - 1) % self.temps}"

    @staticmethod
    def exact(v: float) -> bool:
        return v != 0.0 and abs(math.frexp(v)[0]) == 0.5

    @classmethod
    def reads(cls, e, element) -> bool:
        return e == ("el", element) or any(cls.reads(x, element) for x in e[1:] if isinstance(x, tuple))

    def product(self, e, d):
        """A product of elements, factor by factor in d."""
        if e[1][0] == "*":
            self.product(e[1], d)
            self.P.fma(d, None, ("c", e[2][1]) if e[2][0] == "num" else self.operand(e[2]), init=MULACC)
        elif e[1][0] == "num":
            self.P.fma(d, self.operand(e[2]), ("c", e[1][1]), init=NEG0)
        else:
            self.P.fma(d, self.operand(e[1]), ("c", e[2][1]) if e[2][0] == "num" else self.operand(e[2]), init=NEG0)

    def operand(self, e):
        """An element that holds the value of e (constants have no element: see `b`)."""
        return e[1] if e[0] == "el" else self.value(e)

    def value(self, e, dst=None):
        """e's value in dst or a new temporary; returns the element."""
        P, kind = self.P, e[0]
        if kind == "el":
            if dst is None:
                return e[1]
            P.fma(dst, e[1], ("c", 1.0), init=NEG0)
            return dst
        if kind == "num":
            dst = dst or self.temp()
            P.fma(dst, "O", ("c", e[1]), init=NEG0)
            return dst
        if kind == "neg":
            a = self.operand(e[1])
            dst = dst or self.temp()
            P.fma(dst, a, ("c", 1.0), neg=True, init=NEG0)
            return dst
        if kind == "*":
            if self.memo is not None and dst is None:
                if e not in self.memo:
                    self.memo[e] = f"p{len(self.memo)}"
                    self.product(e, self.memo[e])
                return self.memo[e]
            x, y = e[1], e[2]
            if x[0] == "num":
                x, y = y, x
            if x[0] == "num":
                raise ValueError("a product of constants")
            a = self.operand(x)
            b = ("c", y[1]) if y[0] == "num" else self.operand(y)
            dst = dst or self.temp()
            P.fma(dst, a, b, init=NEG0)
            return dst
        if kind in "+-":
            terms = []                       # a left-associated sum: its terms in order
            while e[0] in ("+", "-"):
                terms.append((e[0], e[2]))
                e = e[1]
            terms.reverse()
            # in dst itself, unless a later term reads it
            inplace = dst is not None and not any(self.reads(t, dst) for _, t in terms)
            acc = dst if inplace else self.temp()
            init = LOAD
            if e == ("num", 0.0):
                init = NEG0                  # 0.0 +- x: only the sign of a zero could differ
            elif e[0] == "num" and e[1] == 1.0:
                P.fma(acc, "O", ("c", 1.0), init=NEG0)
            elif e != ("el", acc):
                self.value(e, acc)
            for sign, t in terms:
                neg = sign == "-"
                if t[0] == "*" and t[1][0] == "num" and self.exact(t[1][1]):
                    P.fma(acc, self.operand(t[2]), ("c", t[1][1]), neg=neg, init=init)
                elif t[0] == "num":
                    P.fma(acc, "O", ("c", t[1]), neg=neg, init=init)
                else:
                    P.fma(acc, self.operand(t), ("c", 1.0), neg=neg, init=init)
                init = LOAD
            if inplace:
                return dst
            if dst is None:
                return acc
            P.fma(dst, acc, ("c", 1.0), init=NEG0)
            return dst
        if kind == "/":
            b = self.operand(e[2])
            if e[1] == ("num", 1.0):
                dst = dst or self.temp()
                P.special(RCP, dst, None, b)
                return dst
            a = self.operand(e[1])
            dst = dst or self.temp()
            P.special(DIV, dst, a, b)
            return dst
        if kind == "fmax":
            a = "Z" if e[1] == ("num", 0.0) else self.operand(e[1])
            b = self.operand(e[2])
            dst = dst or self.temp()
            P.special(MAX, dst, a, b)
            return dst
        if kind == "sqrt":
            b = self.operand(e[1])
            dst = dst or self.temp()
            P.special(SQRT, dst, None, b)
            return dst
        if kind == "copysign" and e[1] == ("fabs", ("num", 1.0)):
            b = self.operand(e[2])
            dst = dst or self.temp()
            P.special(SIGN, dst, None, b)
            return dst
        raise ValueError(f"unknown expression {kind}")


def ebi_program(mech: str, temps: int = 768) -> Program:
    """One iteration's HRRATES, HRG1-HRG4 and HRPRODLOSS."""
    text = (PKG / "csrc" / "gen" / f"{mech}_ebi.cu").read_text()
    P = Program()
    em = _Emit(P, temps)
    for name in ("hrrates", "hrg1", "hrg2", "hrg3", "hrg4", "hrprodloss"):
        body = re.search(rf"void ebi_{name}\([^)]*\)\n\{{\n(.*?)\n\}}", text, re.S).group(1)
        own = {}
        for line in body.splitlines():
            line = line.strip()
            if line.startswith(("double ", "(void)")):
                continue
            lhs, rhs = line.rstrip(";").split(" = ", 1)
            e = _parse(rhs)
            d = _parse(lhs)[1]

            def local(x):          # a routine's own variables: each assignment is a new element
                if x[0] == "el":
                    return ("el", own.get(x[1], x[1]))
                return tuple(local(y) if isinstance(y, tuple) else y for y in x)
            e = local(e)
            if d.startswith("l_") or d == "dtc":
                own[d] = e[1] if e[0] == "el" else em_keep(em, e)
            elif e[0] == "num":
                P.fma(d, "Z" if e[1] == 0.0 else "O", ("c", 1.0 if e[1] == 0.0 else e[1]), init=NEG0)
            elif name == "hrrates":
                rate_chain(P, em, d, e)
            else:
                em.value(e, d)
    return P


def em_keep(em, e):
    """e's value in an element of its own (a routine's variable lives longer than a temporary)."""
    em.kept = getattr(em, "kept", 0) + 1
    return em.value(e, f"v{em.kept - 1}")


def rate_chain(P, em, d, e):
    """RKI * YC * YC ...: the products in place."""
    if e[0] == "el":
        P.fma(d, e[1], ("c", 1.0), init=NEG0)
        return
    if e[0] != "*":
        raise ValueError("a rate is a product")
    if e[1][0] == "el":
        P.fma(d, e[1][1], e[2][1], init=NEG0)
        return
    rate_chain(P, em, d, e[1])
    P.fma(d, None, e[2][1], init=MULACC)


class EbiLayout:
    """Element offsets (doubles) of a cell's EBI state in shared memory."""

    def __init__(self, m, P: Program):
        n, nr = m.nspec, m.nrxns
        self.at, off = {}, 0
        for v in "CBPMLN":                    # YC, YC0, YCP, PROD, LOSS, PNEG
            self.at.update({f"{v}{i}": off + i for i in range(n)})
            setattr(self, "yc yc0 ycp prod loss pneg".split()["CBPMLN".index(v)], off)
            off += n
        for v, name in (("R", "rki"), ("X", "rxrat")):
            self.at.update({f"{v}{r}": off + r for r in range(nr)})
            setattr(self, name, off)
            off += nr
        self.dtc, self.z, self.one = off, off + 1, off + 2
        self.at.update(dtc=off, Z=off + 1, O=off + 2)
        off += 3
        used = {x for op in P.ops for x in (op[1], op[2], op[3]) if isinstance(x, str)}
        for e in sorted(used - set(self.at), key=lambda x: (x[0], int(x[1:]))):
            self.at[e] = off
            off += 1
        self.elems = off


def ebi_tables(mech: str, width: int = WIDTH):
    """(layout, constants, encoded rows)."""
    m, _ = mechanism(mech)
    P = ebi_program(mech)
    lay = EbiLayout(m, P)
    consts = sorted({op[3][1] for op in P.ops if isinstance(op[3], tuple)})
    cof = {c: 8 * q for q, c in enumerate(consts)}
    ops = place(P.ops, lay.at)
    return lay, consts, encode(ops, schedule(ops, width), lambda e: 8 * e, lambda c: cof[c], 8 * lay.z)


def _rows_text(sym, tables, chunk):
    """Programs one after the other, each from the start of a chunk: (declaration, definition)."""
    rows = []
    for table in tables:
        rows += table
        rows += [[(0, 0)] * WIDTH] * (-len(rows) % chunk)
    size = len(rows) * WIDTH
    return (f"extern __device__ const uint2 {sym}[{size}];",
            [f"__device__ __align__(128) const uint2 {sym}[{size}] = {{"]
            + ["  " + ", ".join(f"{{0x{a:x}u, 0x{b:x}u}}" for a, b in row) + "," for row in rows] + ["};"])


def _consts_text(sym, consts):
    return (f"extern __device__ const double {sym}[{len(consts)}];",
            f"__device__ const double {sym}[{len(consts)}] = {{{', '.join(map(c_double, consts))}}};")


def reverse_chunk(n: dict) -> str:
    """Where chunk k of the reverse step's pass lies: its second solve and second and third tsolve
    are the first ones' chunks again."""
    s = n["stage1"] + n["rhs"] + n["solve"]            # end of the first solve
    t = s + n["solve"] + n["tsolve"]                   # of the first tsolve
    j = t + n["tsolve"] + n["jtv"]                     # of jtv
    again = n["solve"] + n["tsolve"]
    return (f"k < {s} ? k : k < {t} ? k - {n['solve']} : k < {j} ? k - {again} : "
            f"k < {j + n['tsolve']} ? k - {again + n['tsolve'] + n['jtv']} : k - {again + n['tsolve']}")


def sources(mech: str) -> dict[str, str]:
    """<mech>_coop.cuh (sizes) and <mech>_coop.cu (tables)."""
    banner = [f"// Generated by cmaq_gb300.mechgen.coop from mechs/{mech}/manifest.json and gen/{mech}_ebi.cu.  Do not edit."]
    ns = f"mech_{mech}"
    h = banner + ["// Sizes and tables of the cooperative kernels (csrc/coop.cuh, csrc/ebi_coop.cuh).", "#pragma once",
                  "#include <cuda_runtime.h>", f"namespace {ns} {{"]
    c = banner + [f'#include "{mech}_coop.cuh"', f"namespace {ns} {{"]

    def traits(name, lay, consts, progs, fields, seq, at, chunk=CHUNK):
        low = name.lower()
        for d, t in (_consts_text(f"c_{low}_const", consts), _rows_text(f"c_{low}_rows", progs.values(), chunk)):
            h.append(d)
            c.extend(t if isinstance(t, list) else [t])
        n = {k: -(-len(t) // chunk) for k, t in progs.items()}
        table = 2 * (chunk + AHEAD) * WIDTH * 8 + 64
        cells = (SMEM_MAX - table - 8 * len(consts)) // (8 * lay.elems)
        return [f"struct {name} {{",
                f"    static constexpr int ELEMS = {lay.elems}, NCONST = {len(consts)}, MAX_CELLS = {cells};",
                "    static constexpr int " + ", ".join(f"{k} = {v}" for k, v in fields.items()) + ";",
                f"    static constexpr int CHUNK = {chunk}, TABLE_SMEM = {table};",
                "    static constexpr int " + ", ".join(f"{k.upper()}_ROWS = {len(t)}" for k, t in progs.items()) + ";",
                f"    // chunks of one pass through the programs ({', '.join(seq)}), and where each lies",
                f"    static constexpr int PASS = {sum(n[k] for k in seq)};",
                f"    static __device__ __forceinline__ int chunk(int k) {{ return {at(n)}; }}",
                f"    static __device__ __forceinline__ const double* constants() {{ return c_{low}_const; }}",
                f"    static __device__ __forceinline__ const uint2* rows() {{ return c_{low}_rows; }}", "};"]
    lay, consts, tables = ros3_tables(mech)
    tail = traits("Coop", lay, consts, tables,
                  dict(Y=lay.y, V=lay.v, K1=lay.k, K2=lay.l, T=lay.t, RKI=lay.rki, G=lay.g, Z=lay.z),
                  ["stage1", "rhs", "solve", "solve"],
                  lambda n: f"k < {sum(n.values())} ? k : k - {n['solve']}")
    alay, aconsts, atabs = adjoint_tables(mech)
    tail += traits("CoopAdj", alay, aconsts, atabs,
                   dict(Y=alay.y, V=alay.v, K1=alay.k1, K2=alay.k2, T=alay.t, K3=alay.k3, NU2=alay.nu2, NU3=alay.nu3,
                        PHI=alay.phi, LAM=alay.lam, EMIS=alay.emis, RKI=alay.rki, GK=alay.gk, G=alay.g, Z=alay.z),
                   ["stage1", "rhs", "solve", "solve", "tsolve", "tsolve", "jtv", "tsolve", "gradient"], reverse_chunk)
    step = [-(-len(atabs[k]) // CHUNK) for k in ("stage1", "rhs", "solve")]
    tail += ["// the forward pass's programs of the same tables: stage1, rhs, solve, solve",
             "struct CoopAdjForward : CoopAdj {",
             f"    static constexpr int PASS = {sum(step) + step[2]};",
             f"    static __device__ __forceinline__ int chunk(int k) {{ return k < {sum(step)} ? k : k - {step[2]}; }}", "};"]
    elay, econsts, rows = ebi_tables(mech)
    tail += traits("CoopEbi", elay, econsts, {"iteration": rows},
                   dict(YC=elay.yc, YC0=elay.yc0, YCP=elay.ycp, PROD=elay.prod, LOSS=elay.loss, PNEG=elay.pneg,
                        RKI=elay.rki, DTC=elay.dtc, Z=elay.z, ONE=elay.one), ["iteration"], lambda n: "k")
    glay, gconsts, gtabs = gear_tables(mech)
    # one-warp blocks with a stream each: chunks as large as leave room for 4 (CB6r5) and 3 (CRACMM2) on an SM
    tail += traits("CoopGear", glay, gconsts, gtabs, dict(Q=glay.q, R1=0, Z=1, ONE=2, WORKSPACE=glay.WORKSPACE),
                   ["predictor", "rhs", "solve"], lambda n: "k", 16 if glay.elems < 6000 else 8)
    h += tail + [f"}}  // namespace {ns}"]
    c.append(f"}}  // namespace {ns}")
    return {f"{mech}_coop.cuh": "\n".join(h) + "\n", f"{mech}_coop.cu": "\n".join(c) + "\n"}


# ----------------------------------------------------------------------------- KMT2
# Fun, Jac_SP, KppDecomp and KppSolve of the aqueous mechanism (gen/kmt2_aq.cuh), products and
# sums rounded one by one as in the EBI code; a product that several sums use is formed once.

def _kmt2_body(name: str) -> list[str]:
    """The statements of a routine's parts in order."""
    text = (PKG / "csrc" / "gen" / "kmt2_aq.cuh").read_text()
    out = []
    for m in re.finditer(rf"KQ_HD KQ_NOINLINE (?:void|int) {name}\d+\([^)]*\)\n\{{\n(.*?)\n\}}", text, re.S):
        out += [x.strip() for x in m.group(1).splitlines()]
    return out


def kmt2_programs() -> dict[str, Program]:
    """Of one Rodas3 step: fjac (F = Fun(Y), J = Jac(Y)), decomp (G in place), solve (V in place),
    fun (V = Fun(YNEW = W))."""
    p = {k: Program() for k in ("fjac", "decomp", "solve", "fun")}
    for name, v, dst, jac in (("fjac", "Y", "F", True), ("fun", "W", "V", False)):
        em = _Emit(p[name], 0, memo=True)
        arrays = {"v": v, "f": "H", "r": "R", "vdot": dst, "jvs": "J"}
        for line in _kmt2_body("kqu_fun_") + (_kmt2_body("kqu_jac_") if jac else []):
            lhs, rhs = line.rstrip(";").split(" = ", 1)
            d, e = _parse(lhs, arrays)[1], _parse(rhs, arrays)
            if e == ("num", 0.0):
                p[name].fma(d, "Z", ("c", 1.0), init=NEG0)
            else:
                em.value(e, d)
    em = _Emit(p["decomp"], KMT2_RING)
    arrays = {"jvs": "G", "x": "V"}
    for line in _kmt2_body("kqu_decomp_"):
        if line.startswith(("if (fabs(", "return 0")) or line == "}":
            continue                       # pivots are tested before the program (as they come in)
        m = re.match(r"\{ const double a = -jvs\[(\d+) \* KQ_S\] / jvs\[(\d+) \* KQ_S\]; jvs\[(\d+) \* KQ_S\] = -a;$", line)
        if m:
            low = f"G{m.group(1)}"
            if m.group(3) != m.group(1):
                raise ValueError(line)
            p["decomp"].special(DIV, low, low, f"G{m.group(2)}")
            continue
        lhs, rhs = line.rstrip(";").split(" = ", 1)
        m = re.fullmatch(r"jvs\[(\d+) \* KQ_S\] \+ a \* jvs\[(\d+) \* KQ_S\]", rhs)
        if not m or lhs != f"jvs[{m.group(1)} * KQ_S]":
            raise ValueError(line)
        t = em.temp()                      # x + a b with a = -L: x - L b
        p["decomp"].fma(t, low, f"G{m.group(2)}", init=NEG0)
        p["decomp"].fma(f"G{m.group(1)}", t, ("c", 1.0), neg=True)
    em = _Emit(p["solve"], KMT2_TEMPS)
    for line in _kmt2_body("kqu_solve_f") + _kmt2_body("kqu_solve_b"):
        lhs, rhs = line.rstrip(";").split(" = ", 1)
        d, e = _parse(lhs, arrays)[1], _parse(rhs, arrays)
        if e[0] == "/":
            if e[1] != ("el", d):
                em.value(e[1], d)
            p["solve"].special(DIV, d, d, em.operand(e[2]))
        else:
            em.value(e, d)
    return p


KMT2_TEMPS, KMT2_RING = 288, 640


class Kmt2Layout:
    """Offsets of the one-cell workspace: kmt2.cuh's with stride 1 (Y, YNEW, FCN0, K1-K4, JAC0, GHIMJ, R,
    FIX), then the temperature factors, the cell's scalars and temporaries.  K4 is the vector
    that is solved for; products of fjac and decomp lie over YNEW and the stage vectors."""

    def __init__(self, nvar, nlu, nreact, nfix, nfactor, ncell):
        self.at = {}
        y, w, f, k = 0, nvar, 2 * nvar, 3 * nvar
        jac = 7 * nvar
        g, r, h = jac + nlu, jac + 2 * nlu, jac + 2 * nlu + nreact
        for v, off, n in (("Y", y, nvar), ("W", w, nvar), ("F", f, nvar), ("V", k + 3 * nvar, nvar), ("J", jac, nlu),
                          ("G", g, nlu), ("R", r, nreact), ("H", h, nfix)):
            self.at.update({f"{v}{i}": off + i for i in range(n)})
        off = h + nfix
        self.ws_elems = off
        self.factor, off = off, off + nfactor
        self.cell, off = off, off + ncell
        self.temps, off = off, off + KMT2_TEMPS
        self.at.update(Z=off, O=off + 1)
        self.elems = off + 2
        own = list(range(self.temps, self.temps + KMT2_TEMPS))
        over = list(range(w, w + nvar)) + list(range(k, k + 4 * nvar))
        self.place = {"fjac": over + own, "decomp": over, "solve": own, "fun": own}


def kmt2_rates() -> list[tuple]:
    """Update_RCONST's rates: (kind, r, integer arguments, real arguments), like kinds together."""
    text = (PKG / "csrc" / "gen" / "kmt2_aq.cuh").read_text()
    body = re.search(r"void kq_rates_update\([^)]*\)\n\{\n(.*?)\n\}", text, re.S).group(1)
    kinds = ("disf", "disb", "krxn", "kiepox")
    out = []
    for line in body.splitlines():
        m = re.fullmatch(r"\s*r\[(\d+) \* KQ_S\] = kq_(\w+)\(c, (?:v, )?(?:f, )?(.*)\);", line)
        args = [float.fromhex(a) if "x" in a else int(a) for a in m.group(3).split(", ")]
        ints = [a for a in args if isinstance(a, int)]
        out.append((kinds.index(m.group(2)), int(m.group(1)), (ints + [0, 0, 0])[:3],
                    ([a for a in args if isinstance(a, float)] + [0.0, 0.0, 0.0])[:3]))
    # rates that the aqueous diffusion limits last, those with a power before them: whole rounds of lanes
    return sorted(out, key=lambda q: (q[0] == 3 or (q[0] == 2 and q[2][1] > 0), q[0] == 2 and q[2][2] > 0, q[0], q[1]))


def kmt2_tables(width: int = WIDTH):
    """(layout, constants, {program: encoded rows})."""
    consts_text = (PKG / "csrc" / "gen" / "kmt2_aq_consts.cuh").read_text()
    num = lambda n: int(re.search(rf"constexpr int {n} = (\d+);", consts_text).group(1))
    progs = kmt2_programs()
    lay = Kmt2Layout(num("NVAR"), num("LU_NONZERO"), num("NREACT"), num("NFIX"), len(kmt2_rates()), 64)
    consts = sorted({op[3][1] for p in progs.values() for op in p.ops if isinstance(op[3], tuple)})
    cof = {c: 8 * q for q, c in enumerate(consts)}
    tables = {}
    for name, p in progs.items():
        ops = place(p.ops, kmt2_places(lay, name, p))
        tables[name] = encode(ops, schedule(ops, width), lambda e: 8 * e, lambda c: cof[c], 8 * lay.at["Z"])
    return lay, consts, tables


def kmt2_places(lay, name, P):
    """The layout with a program's products and temporaries."""
    at = dict(lay.at)
    free = lay.place[name]
    for op in P.ops:
        for x in op[1:4]:
            if isinstance(x, str) and x[0] in "pt":
                if int(x[1:]) >= len(free):
                    raise ValueError(f"{name}: too many temporaries")
                at[x] = free[int(x[1:])]
    return at


def kmt2_sources() -> dict[str, str]:
    lay, consts, tables = kmt2_tables()
    text = (PKG / "csrc" / "gen" / "kmt2_aq.cuh").read_text()
    body = re.search(r"void kq_add_diagonal\([^)]*\)\n\{\n(.*?)\n\}", text, re.S).group(1)
    diag = [int(x) for x in re.findall(r"^\s*g\[(\d+) \* KQ_S\] =", body, re.M)]
    rates = kmt2_rates()
    banner = "// Generated by cmaq_gb300.mechgen.coop from gen/kmt2_aq.cuh.  Do not edit."
    n = {k: -(-len(t) // CHUNK) for k, t in tables.items()}
    first, pos = {}, 0
    for k, v in n.items():
        first[k], pos = pos, pos + v
    order = ["fjac", "decomp", "solve", "solve", "fun", "solve", "fun", "solve"]
    where, pos = "", 0                       # nested choice of the segment that chunk k of a pass lies in
    for q, k in enumerate(order):
        shift = first[k] - pos
        pos += n[k]
        where += (f"k < {pos} ? " if q < len(order) - 1 else "") + f"k + {shift}" + (" : " if q < len(order) - 1 else "")
    dc, tc = _consts_text("c_kmt2_const", consts)
    dr, tr = _rows_text("c_kmt2_rows", tables.values(), CHUNK)
    cells = (SMEM_MAX - TABLE_SMEM - 8 * len(consts)) // (8 * lay.elems)
    h = [banner, "// Sizes and tables of the cooperative KMT2 kernels (csrc/kmt2_coop.cuh).", "#pragma once",
         "#include <cuda_runtime.h>", "namespace kmt2_coop {", dc, dr,
         f"extern __device__ const short c_kmt2_diag[{len(diag)}];",
         "struct Rate { int kind, r, i0, i1, i2; double p0, p1, p2; };   // 0 DISF, 1 DISB, 2 KRXN, 3 KIEPOX",
         f"extern __device__ const Rate c_kmt2_rate[{len(rates)}];", "struct Coop {",
         f"    static constexpr int ELEMS = {lay.elems}, NCONST = {len(consts)}, MAX_CELLS = {cells};",
         f"    static constexpr int WS_ELEMS = {lay.ws_elems}, FACTOR = {lay.factor}, CELL = {lay.cell}, CELL_DOUBLES = 64, "
         f"Z = {lay.at['Z']}, ONE = {lay.at['O']}, NRATE = {len(rates)};",
         f"    static constexpr int CHUNK = {CHUNK}, TABLE_SMEM = {TABLE_SMEM};",
         "    static constexpr int " + ", ".join(f"{k.upper()}_ROWS = {len(t)}" for k, t in tables.items()) + ";",
         f"    // chunks of one pass ({', '.join(order)}), and where each lies",
         f"    static constexpr int PASS = {pos};",
         f"    static __device__ __forceinline__ int chunk(int k) {{ return {where}; }}",
         "    static __device__ __forceinline__ const double* constants() { return c_kmt2_const; }",
         "    static __device__ __forceinline__ const uint2* rows() { return c_kmt2_rows; }", "};",
         "}  // namespace kmt2_coop"]
    c = [banner, '#include "kmt2_coop_tables.cuh"', "namespace kmt2_coop {", tc, *tr,
         f"__device__ const short c_kmt2_diag[{len(diag)}] = {{{', '.join(map(str, diag))}}};",
         f"__device__ const Rate c_kmt2_rate[{len(rates)}] = {{",
         *[f"  {{{k}, {r}, {', '.join(map(str, i))}, {', '.join(map(c_double, x))}}}," for k, r, i, x in rates], "};",
         "}  // namespace kmt2_coop"]
    return {"kmt2_coop_tables.cuh": "\n".join(h) + "\n", "kmt2_coop_tables.cu": "\n".join(c) + "\n"}


def write(mech: str, out: Path | None = None) -> None:
    out = out or PKG / "csrc" / "gen"
    for name, text in sources(mech).items():
        (out / name).write_text(text)


def write_kmt2(out: Path | None = None) -> None:
    for name, text in kmt2_sources().items():
        ((out or PKG / "csrc" / "gen") / name).write_text(text)


if __name__ == "__main__":
    write_kmt2()
    for mech_ in ("cb6r5_ae7_aq", "cracmm2"):
        write(mech_)
