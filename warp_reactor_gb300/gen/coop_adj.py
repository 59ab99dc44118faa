"""Vector programs of the differentiation form, for the cooperative (lanes-per-cell)
forward and adjoint kernels (csrc/wr_diff_coop.cu).

The step format, scheduling and slot map are ``coop.py``'s.  The programs, for ``G`` = 32
lanes per cell:

* ``jrhsp``: the Jacobian of the unscaled network and the RHS with one multiplier per
  rate coefficient (``adjoint.multiplied_rhs``) at y.  The values are the same operations
  as the straight-line code's, so the forward map keeps its bits;
* ``rhsp``: that RHS alone;
* ``rhsvjp``: the RHS vector-Jacobian product: given fbar (15), the adjoints of y (14
  number densities and the energy, through the floor and the equation of state) and
  of the multipliers;
* ``jacvjp``: the Jacobian's: given Jbar (15 x 15, in the matrix slots), the adjoint of y;

each for any state and once more for every temperature regime (``coop.REGIMES``).

Reverse mode (``reverse``) performs the operations of the straight-line derivative code
that ``adjoint.py`` emits, one by one: each adjoint is the sum of its contributions in
the order in which that code adds them (reverse schedule order, a Jacobian root's seed
at its chunk), products are guarded -- 0 where the adjoint is 0, because the branch that
a select did not take may hold infinities, and 0 * inf must not reach the inputs
(classes ``C_GMUL``, ``C_GDIV``) -- and products and sums round separately.  A stiff step's
adjoint cancels ten digits and more, so another order of the same sums would give
gradients that agree with the straight-line code's to six digits only, no better and no
worse; this one gives the same bits (a zero may have the other sign).  (The price is the
serial sum of the contributions to T and log T, several hundred for the Jacobian: it is
the program's critical path.)

Slots: the multipliers and fbar have reserved slots above the constants; no program
writes them, nor the matrix slots but for ``jrhsp``.
"""
from __future__ import annotations

import collections
import math
import os

from . import adjoint, coop, ir_io
from .emit import schedule as schedule_dag
from .coop import (FLOOR, K_GAS, K_MP, MASS, PREFETCH_PAD, REGIMES, RES_BASE, Program, dbits, device_words,
                   encode, inv_gm1, lower, resolve, schedule)

G = 32
# (latency weight, hold, seed, amplitude, fill), live-set limit: chosen offline by a seeded
# random search for the cheapest schedules (FP64 issue slots, steps), as coop.SCHED_TUNE
TUNE = {
    ("jrhsp", 0): ((3.5, 2.0, 631732, 0.1, 23), 900),
    ("rhsp", 0): ((3.0, {coop.C_EXP: 10.0, coop.C_LOG: 30.0, coop.C_SQRT: 0.0}, 655940, 1.0, 24), 1400),
    ("rhsvjp", 0): ((8.0, 8.0, 634511, 0.5, 32), 1400),
    ("jacvjp", 0): ((3.5, 8.0, 742423, 1.0, 30), 1300),
    ("jrhsp", 1): ((6.0, 0.0, 964175, 1.0, 22), 550),
    ("rhsp", 1): ((3.0, {coop.C_EXP: 10.0, coop.C_LOG: 0.0, coop.C_SQRT: 5.0}, 428434, 0.5, 16), 1000),
    ("rhsvjp", 1): ((7.0, 5.0, 234041, 0.1, 28), 500),
    ("jacvjp", 1): ((8.0, 2.0, 618195, 1.0, 23), 1750),
    ("jrhsp", 2): ((6.0, None, 594332, 0.1, 30), 550),
    ("rhsp", 2): ((3.5, {coop.C_EXP: 20.0, coop.C_LOG: 30.0, coop.C_SQRT: 5.0}, 999955, 2.0, 17), 1400),
    ("rhsvjp", 2): ((3.0, 2.0, 448081, 0.01, 32), 1400),
    ("jacvjp", 2): ((6.5, 2.0, 979543, 0.001, 28), None),
    ("jrhsp", 3): ((4.0, 0.0, 236978, 0.1, 31), 550),
    ("rhsp", 3): ((2.0, {coop.C_EXP: 20.0, coop.C_LOG: 10.0, coop.C_SQRT: 0.0}, 442818, 1.0, 22), 600),
    ("rhsvjp", 3): ((1.5, {coop.C_EXP: 2.0, coop.C_LOG: 10.0, coop.C_SQRT: 5.0}, 881195, 0.5, 27), 1800),
    ("jacvjp", 3): ((10.0, 0.0, 473535, 0.1, 22), 1400),
    ("jrhsp", 4): ((8.0, 0.0, 208630, 0.1, 29), 600),
    ("rhsp", 4): ((5.0, {coop.C_EXP: 20.0, coop.C_LOG: 30.0, coop.C_SQRT: 5.0}, 655449, 0.01, 11), None),
    ("rhsvjp", 4): ((11.0, {coop.C_EXP: 2.0, coop.C_LOG: 30.0, coop.C_SQRT: 0.0}, 634517, 0.5, 31), 1000),
    ("jacvjp", 4): ((6.0, 2.0, 648360, 1.0, 21), 500),
    ("jrhsp", 5): ((3.0, 2.0, 799792, 1.0, 22), 550),
    ("rhsp", 5): ((5.0, {coop.C_EXP: 20.0, coop.C_LOG: 30.0, coop.C_SQRT: 20.0}, 253558, 0.5, 10), 550),
    ("rhsvjp", 5): ((3.5, 0.0, 531697, 0.1, 23), 1800),
    ("jacvjp", 5): ((8.0, {coop.C_EXP: 10.0, coop.C_LOG: 0.0, coop.C_SQRT: 0.0}, 141019, 0.001, 20), 600),
    ("jrhsp", 6): ((1.5, 0.0, 979613, 0.01, 20), 600),
    ("rhsp", 6): ((4.5, {coop.C_EXP: 10.0, coop.C_LOG: 30.0, coop.C_SQRT: 5.0}, 619996, 2.0, 16), 1400),
    ("rhsvjp", 6): ((1.5, 5.0, 66987, 0.1, 30), 1800),
    ("jacvjp", 6): ((6.0, None, 701470, 0.01, 30), 1500),
}


def prologue(P: Program):
    """burn_state_from_y (reproducer.cpp:7029-7038) as coop.build has it: y, the floor
    conditions, X, the mass sum and T."""
    Y = [P.add("in", k) for k in range(15)]
    floor = P.const(FLOOR)
    low = [P.add("lt", Y[k], floor) for k in range(14)]
    X = [P.add("sel", low[k], floor, Y[k]) for k in range(14)]
    rhotot = P.add("mul", X[0], P.const(MASS[0]))
    for n in range(1, 14):
        rhotot = P.add("add", rhotot, P.add("mul", X[n], P.const(MASS[n])))
    sa = X[0]
    for n in range(1, 14):
        sa = P.add("add", sa, X[n])
    sg = None
    for n in range(14):
        term = P.add("mul", P.add("div", P.add("mul", X[n], P.const(K_MP)), rhotot), P.const(inv_gm1(n)))
        sg = term if sg is None else P.add("add", sg, term)
    sa = P.add("mul", sa, P.add("div", P.const(K_MP), rhotot))
    sg = P.add("div", sg, sa)
    T = P.add("div", Y[14], P.add("mul", P.add("mul", sg, P.const(K_GAS)), sa))
    return Y, low, X, rhotot, T


def load_dag(P: Program, dag, roots, X, T):
    """The DAG's nodes below the roots as program nodes: the map, and the multipliers'
    nodes by index."""
    m, par = {}, {}
    for x in dag.live_from(roots):
        n = dag.nodes[x]
        if n.op == "in":
            a = n.args[0]
            if a.startswith("M"):
                m[x] = par[int(a[1:])] = P.add("fix", "mult", int(a[1:]))
            else:
                m[x] = T if a == "T" else X[int(a[1:])]
        elif n.op == "const":
            m[x] = P.const(float.fromhex(n.args[0]))
        elif n.op == "bconst":
            m[x] = P.const_bits(1 if n.args[0] else 0)
        else:
            m[x] = P.add(n.op, *[m[a] for a in n.args])
    return m, par


def reverse(P: Program, dag, m, roots, seeds, chunks=None) -> dict:
    """Adjoint nodes of the DAG's input nodes: ``adjoint._vjp_body`` (``chunks`` None) or
    ``adjoint._vjp_chunked`` on program nodes.  ``m``: the DAG's nodes in the program;
    ``seeds``: the roots' adjoints."""
    order = schedule_dag(dag, roots)
    active = adjoint._active(dag, order)
    zero, half = P.const(0.0), P.const(0.5)
    bar = {}

    def give(x, g, neg=False):
        if x not in active:
            return
        if x not in bar:
            bar[x] = P.add("neg", g) if neg else g
        else:
            bar[x] = P.add("sub" if neg else "add", bar[x], g)

    def node(x):
        g = bar[x]
        op, a = dag.nodes[x].op, dag.nodes[x].args
        if op in ("add", "sub"):
            give(a[0], g)
            give(a[1], g, op == "sub")
        elif op == "mul":
            give(a[0], P.add("gmul", g, m[a[1]]))
            give(a[1], P.add("gmul", g, m[a[0]]))
        elif op == "div":
            give(a[0], P.add("gdiv", g, m[a[1]]))
            give(a[1], P.add("gdiv", P.add("gmul", g, m[x]), m[a[1]]), True)
        elif op == "neg":
            give(a[0], g, True)
        elif op == "abs":
            give(a[0], P.add("sel", P.add("lt", m[a[0]], zero), P.add("neg", g), g))
        elif op == "exp":
            give(a[0], P.add("gmul", g, m[x]))
        elif op == "log":
            give(a[0], P.add("gdiv", g, m[a[0]]))
        elif op == "sqrt":
            give(a[0], P.add("gdiv", P.add("mul", g, half), m[x]))
        elif op == "sel":
            give(a[1], P.add("sel", m[a[0]], g, zero))
            give(a[2], P.add("sel", m[a[0]], zero, g))
        elif op != "in":
            raise ValueError(f"no derivative rule for {op}")

    if chunks is None:
        for r, s in zip(roots, seeds):
            give(r, s)
        for x in reversed(order):
            if x in active and x in bar and dag.nodes[x].op != "in":
                node(x)
        return bar
    body = [x for x in order if dag.nodes[x].op not in ("const", "in", "bconst")]
    size = (len(body) + chunks - 1) // chunks
    at = collections.defaultdict(list)
    for r, s in zip(roots, seeds):
        at[r].append(s)
    for k in range((len(body) + size - 1) // size - 1, -1, -1):
        mine = body[k * size:(k + 1) * size]
        for x in mine:
            for s in at.get(x, []):
                give(x, s)
        for x in reversed(mine):
            if x in active and x in bar:
                node(x)
    for r, s in zip(roots, seeds):
        if dag.nodes[r].op == "in":
            give(r, s)
    return bar


def build(kind: str, dag, mdag, regime=None) -> tuple:
    """A program and its outputs: ``rhs`` (a list of nodes), ``T`` and for ``jac`` the
    Jacobian's entries."""
    P = Program()
    Y, low, X, rhotot, T = prologue(P)
    d = dag if kind == "jacvjp" else mdag
    roots = dag.jac_roots() if d is dag else mdag.rhs_roots()
    m, par = load_dag(P, d, roots, X, T)
    if kind in ("jrhsp", "rhsp"):
        out = {"rhs": [m[x] for x in roots], "T": T}
        if kind == "jrhsp":
            mj, _ = load_dag(P, dag, dag.jac_roots(), X, T)
            keys = [(r, c) for r in range(15) for c in range(15)]
            out["jac"] = dict(zip(keys, [mj[x] for x in dag.jac_roots()]))
    else:
        if kind == "rhsvjp":
            bar = reverse(P, d, m, roots, [P.add("fix", "fbar", i) for i in range(15)])
        else:
            bar = reverse(P, d, m, roots, [P.add("fix", "jbar", i) for i in range(225)], adjoint.JAC_VJP_CHUNKS)
        inputs = {d.nodes[x].args[0]: g for x, g in bar.items() if d.nodes[x].op == "in"}
        zero = P.const(0.0)
        # the adjoint of state_from_y: T = e A / (R mp B), A = sum m x, B = sum x / (gamma - 1)
        B = P.add("mul", X[0], P.const(inv_gm1(0)))
        for n in range(1, 14):
            B = P.add("add", B, P.add("mul", X[n], P.const(inv_gm1(n))))
        c = P.add("mul", B, P.const(K_GAS * K_MP))
        t = P.add("mul", inputs["T"], P.add("div", P.add("mul", Y[14], rhotot), c))
        over = {w: P.add("div", P.const(w), B) for w in {inv_gm1(n) for n in range(14)}}
        ybar = []
        for n in range(14):
            g = P.add("mul", t, P.add("sub", P.add("div", P.const(MASS[n]), rhotot), over[inv_gm1(n)]))
            if f"X{n}" in inputs:
                g = P.add("add", inputs[f"X{n}"], g)
            ybar.append(P.add("sel", low[n], zero, g))
        ybar.append(P.add("div", P.add("mul", inputs["T"], rhotot), c))
        mbar = [inputs[f"M{r}"] for r in range(len(par))] if kind == "rhsvjp" else []
        out = {"rhs": ybar + mbar, "T": T}
    # (the general program too: equal nodes of the two DAGs become one)
    P, out = coop.specialize(P, out, *(regime or (-math.inf, math.inf)))
    coop.rebalance_boolean_chains(P)
    lower(P)
    return P, out


def generate(regimes=REGIMES, tune=TUNE) -> dict:
    """All programs on one slot map: ``progs`` [(kind, regime index, program)] with the
    ``jrhsp`` and ``rhsp`` of regime 0, 1, ..., then their ``rhsvjp`` and ``jacvjp``."""
    dag = ir_io.load()
    mdag, rates = adjoint.multiplied_rhs(dag)
    wanted = [(kind, r) for pair in (("jrhsp", "rhsp"), ("rhsvjp", "jacvjp")) for r in range(1 + len(regimes))
              for kind in pair]
    built = {(kind, r): build(kind, dag, mdag, regimes[r - 1] if r else None) for kind, r in wanted}
    fixed = [0, 1, dbits(1.0), dbits(-1.0), dbits(-0.0)]
    pool, funs = set(fixed), set()
    for P, out in built.values():
        pool |= coop.reserved_constants(P, out)
        funs |= coop.device_constants(P, out)
    rconst = fixed + sorted(pool - set(fixed))
    rfun = sorted(funs)
    keys = rconst + rfun + [("mult", r) for r in range(len(rates))] + [("fbar", i) for i in range(15)]
    res = {k: RES_BASE + i for i, k in enumerate(keys)}
    res.update({("jbar", i): i for i in range(225)})
    first = RES_BASE + len(keys)
    scheds = {}
    for (kind, r), (P, out) in built.items():
        t, lim = tune[kind, r]
        scheds[kind, r] = schedule(P, out, G, jac=kind == "jrhsp", limit=lim, first_scratch=first, tune=t)[0]
    # two sizes of the slot array: the forward kernel holds the first alone
    fwd = max(s.nv for (kind, _), s in scheds.items() if kind in ("jrhsp", "rhsp"))
    nva = max(max(s.nv for s in scheds.values()), fwd) + 6 * 16  # the adjoint kernel's scratch vectors
    if nva > coop.MAX_SLOTS:
        raise ValueError(f"{nva} slots do not fit the output operands")
    progs = []
    for kind, r in wanted:
        P, out = built[kind, r]
        sch = scheds[kind, r]
        st = coop.stats(sch)
        sch.nv = nv = fwd if kind in ("jrhsp", "rhsp") else nva
        words = encode(P, sch, res)

        def outop(o, negate=False):
            b, neg, ab = o
            op, a = P.nodes[b]
            v = res[a[0]] if op == "const" else res[a] if op in ("dconst", "fix") else sch.slot[b]
            return v | (coop.OPF_NEG if neg != negate else 0) | (coop.OPF_ABS if ab else 0)

        pr = {"words": words, "out": [outop(o) for o in sch.outputs["rhs"]], "T_out": outop(sch.outputs["T"]),
              "nsteps": len(words) - PREFETCH_PAD, "stats": st, "nv": nv}
        if kind == "jrhsp":
            pr["jac_out"] = [outop(o, negate=True) for o in sch.outputs["jac"]]
        progs.append((kind, r, pr))
    return {"nv": fwd, "nva": nva, "rconst": rconst, "rfun": rfun, "mult": res["mult", 0], "fbar": res["fbar", 0],
            "progs": progs, "nmult": len(rates), "regimes": regimes}


def emit_header(gen: dict, digest: str) -> str:
    progs = gen["progs"]
    nreg = 1 + len(gen["regimes"])
    dev = [device_words(pr, pr["nv"]) for _, _, pr in progs]
    lines = [
        "// Generated by warp_reactor_gb300/gen/coop_adj.py from network.ir",
        f"// network.ir sha256 {digest}",
        "// Vector programs of the differentiation form, 32 lanes per cell.",
        "#pragma once",
        "#include <stdint.h>",
        "",
        "namespace wr { namespace coop_diff {",
        f"constexpr int kG = {G};",
        f"constexpr int kNV = {gen['nv']};    // slots of the forward programs",
        f"constexpr int kNVA = {gen['nva']};  // slots of all programs and the adjoint's scratch vectors",
        f"constexpr int kNR = {len(gen['rconst'])};  // reserved constant slots from {RES_BASE}",
        f"constexpr int kNF = {len(gen['rfun'])};  // then the transcendentals of constants",
        f"constexpr int kMult = {gen['mult']};  // then the multipliers",
        f"constexpr int kNumMult = {gen['nmult']};",
        f"constexpr int kFbar = {gen['fbar']};  // then the RHS adjoint of the RHS vector-Jacobian product",
        f"constexpr int kRegimes = {nreg};  // 0: any state, the others by temperature",
        "// first step and steps of each program: Jacobian + RHS and RHS of regime 0, 1, ..., then the RHS and",
        "// the Jacobian vector-Jacobian products of regime 0, 1, ...",
        f"static __constant__ const int kProgStep[{len(progs)}][2] = {{",
    ]
    total = 0
    for (kind, r, pr), (words, _) in zip(progs, dev):
        lines.append(f"    {{{total}, {len(words) - PREFETCH_PAD}}},  // {kind}, regime {r}: {pr['stats']['by_class']}, "
                     f"{pr['stats']['slots']} slots")
        total += len(words)
    lines.append("};")
    lines.append(f"static __constant__ const uint64_t kRegimeT[{nreg}][2] = {{{{0ULL, 0x7ff0000000000000ULL}},")
    for lo, hi in gen["regimes"]:
        lines.append(f"    {{0x{dbits(lo):016x}ULL, 0x{dbits(hi):016x}ULL}},")
    lines.append("};")
    ctl = [sum(c[s + k] << (8 * k) for k in range(4)) for _, c in dev for s in range(0, len(c), 4)]

    def table(head, items, per):
        lines.append(head + " = {")
        for i in range(0, len(items), per):
            lines.append("    " + ", ".join(items[i:i + per]) + ",")
        lines.append("};")

    table(f"static __device__ const uint64_t kVConst[kNR]", [f"0x{b:016x}ULL" for b in gen["rconst"]], 4)
    table(f"static __device__ const ulonglong2 kVFun[{max(1, len(gen['rfun']))}]",
          [f"{{{c}ULL, 0x{b:016x}ULL}}" for c, b in gen["rfun"] or [(0, 0)]], 2)
    table(f"static __constant__ const uint32_t kCtl[{len(ctl)}]", [f"0x{w:x}U" for w in ctl], 8)
    table(f"static __device__ const ulonglong2 kProg[{total} * kG]",
          [f"{{0x{m:x}ULL, 0x{i:x}ULL}}" for words, _ in dev for lanes in words for m, i, _ in lanes], 8)
    table(f"static __device__ const uint64_t kLit[{total} * kG]",
          [f"0x{v:x}ULL" for words, _ in dev for lanes in words for _, _, v in lanes], 8)
    outs = []
    for kind, r, pr in progs[:2 * nreg]:
        outs.append("{" + ", ".join(str(v) for v in pr["out"] + [pr["T_out"]]) + "}")
    table(f"static __device__ const uint16_t kOut[{2 * nreg}][16]", outs, 1)
    table(f"static __device__ const uint16_t kJac[{nreg}][225]",
          ["{" + ", ".join(str(v) for v in pr["jac_out"]) + "}" for kind, _, pr in progs if kind == "jrhsp"], 1)
    # outputs, then T
    for name, kind, n in (("kRhsVjpOut", "rhsvjp", 15 + gen["nmult"]), ("kJacVjpOut", "jacvjp", 15)):
        table(f"static __device__ const uint16_t {name}[{nreg}][{n + 1}]",
              ["{" + ", ".join(str(v) for v in pr["out"] + [pr["T_out"]]) + "}" for k, _, pr in progs if k == kind], 1)
    lines.append("} }  // namespace wr::coop_diff")
    return "\n".join(lines) + "\n"


def emit(out_dir: str, ir_path: str = ir_io.DEFAULT_PATH) -> str:
    from .build_network import _write_if_changed
    path = os.path.join(out_dir, "coop_diff.h")
    _write_if_changed(path, f"// generator {coop.generator_digest(ir_path)}\n" +
                      emit_header(generate(), ir_io.digest(ir_path)))
    return path


if __name__ == "__main__":
    g = generate()
    print(g["nv"], g["nva"], len(g["rconst"]), g["mult"], g["fbar"])
    for kind, r, pr in g["progs"]:
        print(kind, r, pr["stats"], len(device_words(pr, pr["nv"])[0]))
