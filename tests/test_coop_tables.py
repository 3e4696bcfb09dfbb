"""The lane schedules of the cooperative kernels (mechgen/coop.py) against the sequential
operations, on the CPU: both are carried out on expressions instead of numbers, the
schedule from its encoded rows with the kernel's visibility of stores, and every element must
end as the same expression (the same operations on the same values in the same order).
"""
import pytest

from cmaq_gb300.mechgen import coop as C


class Terms:
    """Expressions by number: equal operations on equal operands have equal numbers."""

    def __init__(self):
        self.ids = {}

    def __call__(self, *key):
        return self.ids.setdefault(key, len(self.ids))


def sequential(ops, start, term):
    x = dict(start)
    for kind, d, a, b, neg, init in ops:
        vb = term("const", b[1]) if isinstance(b, tuple) else x[b]
        if kind == "D":
            x[d] = term("special", init, x[a] if init in (C.DIV, C.MAX) else None, vb)
            continue
        va = x[d] if init == C.MULACC else x[a]
        x[d] = term("fma", neg, va, vb, x[d] if init == C.LOAD else "-0")
    return x


def rows_run(rows, start, consts, term):
    """The kernel's loop: operands of row t + 2 loaded before the results of row t are stored."""
    x = dict(start)
    width = len(rows[0])
    acc = [term("idle", ln) for ln in range(width)]

    def load(row):
        got = []
        for w0, w1 in row:
            a, b, d = (w0 & 0xfff8) // 8, (w0 >> 19) & 0x1fff, (w1 & 0xfff8) // 8
            got.append((x[a], term("const", consts[b]) if w1 & C.B_CONST else x[b], x[d]))
        return got

    idle = [(0, 0)] * width
    at = lambda t: load(rows[t] if t < len(rows) else idle)
    ops, pending, special = [at(0), at(1)], {}, False
    for t, row in enumerate(rows):
        if t % C.UNROLL == 0:
            special = bool(row[0][0] & C.A_SPECIAL)
            if special:                                      # a block of its own: the rest of it is not read
                x.update(pending)
                pending = {}
                assert all(w0 & C.A_SPECIAL for w0, _ in row)
                got = [(w1, v) for (_, w1), v in zip(row, load(row)) if w1 & C.D_STORE]
                for w1, (a, b, _) in got:
                    kind = w1 & 7
                    x[(w1 & 0xfff8) // 8] = term("special", kind, a if kind in (C.DIV, C.MAX) else None, b)
                ops = [at(t + C.UNROLL), at(t + C.UNROLL + 1)]
        if special:
            continue
        assert not any(w0 & C.A_SPECIAL for w0, _ in row)
        cur, results = ops.pop(0), {}
        for ln, (w0, w1) in enumerate(row):
            a, b, c = cur[ln]
            if w1 & C.C_KEEP and w1 & C.A_NEG and (w0 & 0xffff) == (w0 >> 16) == (w1 & 0xfff8):
                continue                                   # idle lane: acc = -0 * 0 + acc
            if not w1 & C.C_LOAD:
                c = acc[ln] if w1 & C.C_KEEP else "-0"
            if w1 & C.C_MULACC:
                a = acc[ln]
            acc[ln] = term("fma", bool(w1 & C.A_NEG), a, b, c)
            if w1 & C.D_STORE:
                d = (w1 & 0xfff8) // 8
                assert d not in results
                results[d] = acc[ln]
        x.update(pending)                                  # row t - 1's results, then row t + 2's operands
        pending = results
        ops.append(at(t + 2))
    x.update(pending)
    return x


@pytest.mark.parametrize("mech", ["cb6r5_ae7_aq", "cracmm2"])
@pytest.mark.parametrize("width", [C.WIDTH, 8])
def test_rows_carry_out_the_sequential_operations(mech, width):
    m, sp = C.mechanism(mech)
    lay, consts, tables = C.ros3_tables(mech, width)
    for name, prog in C.ros3_programs(m, sp).items():
        ops = lay.place(prog.ops)
        term = Terms()
        start = {e: term("in", e) for e in range(lay.elems)}
        want = sequential(ops, start, term)
        got = rows_run(tables[name], start, consts, term)
        # partial-derivative products are scratch: elements that nothing reads any more
        scratch = set(lay.alias.values()) if name == "stage1" else set()
        assert all(got[e] == want[e] for e in range(lay.elems) if e not in scratch), name


@pytest.mark.parametrize("mech", ["cb6r5_ae7_aq", "cracmm2"])
@pytest.mark.parametrize("width", [C.WIDTH, 8])
def test_ebi_rows_carry_out_the_sequential_operations(mech, width):
    lay, consts, rows = C.ebi_tables(mech, width)
    ops = C.place(C.ebi_program(mech).ops, lay.at)
    term = Terms()
    start = {e: term("in", e) for e in range(lay.elems)}
    want, got = sequential(ops, start, term), rows_run(rows, start, consts, term)
    assert all(got[i] == want[i] for i in range(lay.elems)
               if i in {lay.at[e] for e in lay.at if e[0] in "CBPMLNRX"})


@pytest.mark.parametrize("mech", ["cb6r5_ae7_aq", "cracmm2"])
def test_gear_rows_carry_out_the_sequential_operations(mech):
    m, sp = C.mechanism(mech)
    lay, consts, tables = C.gear_tables(mech)
    progs, coefs = C.gear_programs(m, sp)
    for name, prog in progs.items():
        ops = C.place(prog.ops, lay.at)
        term = Terms()
        start = {e: term("in", e) for e in range(lay.elems)}
        want, got = sequential(ops, start, term), rows_run(tables[name], start, consts, term)
        scratch = {lay.at[f"S{q}"] for q in range(len(coefs))} if name == "predictor" else set()
        assert all(got[e] == want[e] for e in range(lay.elems) if e not in scratch), name


@pytest.mark.parametrize("mech", ["cb6r5_ae7_aq", "cracmm2"])
def test_adjoint_rows_carry_out_the_sequential_operations(mech):
    m, sp = C.mechanism(mech)
    lay, consts, tables = C.adjoint_tables(mech)
    for name, prog in C.adjoint_programs(m, sp)[0].items():
        ops = C.place(prog.ops, lay.at)
        term = Terms()
        start = {e: term("in", e) for e in range(lay.elems)}
        want, got = sequential(ops, start, term), rows_run(tables[name], start, consts, term)
        # products of the matrix (E) and the gradient's temporaries (h) are scratch
        scratch = {i for e, i in lay.at.items() if e[0] in {"stage1": "E", "gradient": "h"}.get(name, "")}
        assert all(got[e] == want[e] for e in range(lay.elems) if e not in scratch), name
    n = {k: -(-len(t) // C.CHUNK) for k, t in tables.items()}
    first = dict(zip(n, [sum(list(n.values())[:i]) for i in range(len(n))]))
    order = ["stage1", "rhs", "solve", "solve", "tsolve", "tsolve", "jtv", "tsolve", "gradient"]
    chunk = C.reverse_chunk(n).replace("?", "and").replace(":", "or")
    for k, want in enumerate(first[p] + i for p in order for i in range(n[p])):
        # Python's `c and a or b` is C's `c ? a : b` but for a == 0, which is chunk 0's
        assert eval(chunk, {"k": k}) == want or k == want == 0


def test_kmt2_rows_carry_out_the_sequential_operations():
    lay, consts, tables = C.kmt2_tables()
    for name, prog in C.kmt2_programs().items():
        at = C.kmt2_places(lay, name, prog)
        ops = C.place(prog.ops, at)
        term = Terms()
        start = {e: term("in", e) for e in range(lay.elems)}
        want, got = sequential(ops, start, term), rows_run(tables[name], start, consts, term)
        scratch = {i for e, i in at.items() if e[0] in "pt"}
        assert all(got[e] == want[e] for e in range(lay.elems) if e not in scratch), name


@pytest.mark.parametrize("mech", ["cb6r5_ae7_aq", "cracmm2", "kmt2"])
def test_tables_are_the_generated_ones(mech):
    for name, text in (C.kmt2_sources() if mech == "kmt2" else C.sources(mech)).items():
        assert (C.PKG / "csrc" / "gen" / name).read_text() == text
