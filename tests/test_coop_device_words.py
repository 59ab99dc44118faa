"""The words the device executes (``coop.device_words``), run on the CPU the way the
interpreter of ``csrc/wr_coop.cuh`` overlaps its steps: a step computes on operands
loaded during the step before, then the previous step's main results and its own
integer results are stored, then the next step's operands are loaded.  The result
must equal the step-by-step execution of the encoded program in every slot the
program keeps."""
import math

import pytest

from test_coop_programs import (ABS, C_DIV, C_EXP, C_FMA, C_LOG, C_NONE, C_SQRT, I_LE, I_LT, I_SGN, SIGN, d, fetch,
                                fma, run, same, states, u)
from warp_reactor_gb300.gen import coop, ir_io


def slow(cls, x, y, fl, oracle):
    if cls in (C_DIV, coop.C_GDIV):
        x = (x & ABS) if fl & coop.DV_ABS else x
        x = (x ^ SIGN) if fl & coop.DV_NEG else x
        num, den = (d(y), d(x)) if fl & coop.DV_SWAP else (d(x), d(y))
        if den != 0:
            return num / den
        return math.copysign(math.inf, num) * math.copysign(1, den) if num != 0 and num == num else float("nan")
    y = (y & ABS) if fl & coop.DV_ABS else y
    y = (y ^ SIGN) if fl & coop.DV_NEG else y
    if cls == C_EXP:
        return oracle.exp(d(y))
    if cls == C_LOG:
        return oracle.log(d(y))
    assert cls == C_SQRT
    return math.sqrt(d(y)) if d(y) >= 0 else float("nan")


def integer(i, ctl, A, B, C):
    d2 = (i >> 48) & 0xffff
    r, iop = (B if A != 0 else C), d2 & 3
    if ctl & coop.CTL_SPECIAL:
        if iop == I_LE:
            r = int(d(A) <= d(B))
        elif iop == I_LT:
            r = int(d(A) < d(B))
        elif iop == I_SGN:
            r = (A & ABS) if d2 & coop.FL_SABS else (A ^ SIGN)
    return d2 >> 3, r


def overlapped(words, ctl, V, oracle):
    def load(s):
        out = []
        for m, _, lit in words[s]:
            f = [(m >> (16 * k)) & 0xffff for k in range(3)]
            assert all(v % 8 == 0 for v in f), "flags on a loaded field"
            x, y, z = (V[a >> 3] for a in f)
            out.append((x, y ^ lit, z))
        return out

    ops, pending = load(0), []
    for s in range(len(words) - coop.PREFETCH_PAD):
        cls, results, ints = ctl[s] & 7, [], []
        for (m, i, _), (x, y, z) in zip(words[s], ops):
            dst = (m >> 48) & 0xffff
            if cls == C_FMA:
                results.append((dst >> 3, u(fma(d(x), d(y), d(z)))))
            elif cls == coop.C_GMUL:
                results.append((dst >> 3, 0 if x & ABS == 0 else u(d(x) * d(y))))
            elif cls == coop.C_GDIV and x & ABS == 0:
                results.append((dst >> 3, 0))
            elif cls != C_NONE:
                results.append((dst >> 3, u(slow(cls, x, y, dst & 7, oracle))))
            else:
                results.append((dst >> 3, 0))
            if ctl[s] & coop.CTL_INT:
                f = [(i >> (16 * k)) & 0xffff for k in range(3)]
                assert all(v % 8 == 0 for v in f), "flags on a loaded field"
                ints.append(integer(i, ctl[s], *(V[a >> 3] for a in f)))
        for a, r in ints + (results if ctl[s] & coop.CTL_FLUSH else []) + pending:
            V[a] = r
        ops, pending = load(s + 1), results
    for a, r in pending:
        V[a] = r


def start(gen, y, oracle):
    V = [0x7ff4000000000000] * gen["nv"]
    V[:coop.E_SLOTS] = [u(1.0 + k) for k in range(coop.E_SLOTS)]
    for i, b in enumerate(gen["rconst"]):
        V[coop.RES_BASE + i] = b
    fn = {C_EXP: oracle.exp, C_LOG: oracle.log, C_SQRT: math.sqrt}
    for j, (cls, b) in enumerate(gen["rfun"]):
        V[coop.RES_BASE + len(gen["rconst"]) + j] = u(fn[cls](d(b)))
    for k in range(15):
        V[coop.Y_BASE + k] = u(y[k])
    return V


@pytest.mark.parametrize("G", [8, 16, 32])
def test_overlapped_steps_equal_sequential_steps(oracle_port, G):
    gen = coop.generate(G, ir_io.load())
    nres = len(gen["rconst"]) + len(gen["rfun"])
    for y in states(3, 100 + G):
        for pr in gen["progs"].values():
            V = start(gen, y, oracle_port)
            W = list(V)
            run(pr["words"], V, nres, oracle_port)
            words, ctl = coop.device_words(pr, gen["nv"])
            assert len(words) == len(ctl) and (len(words) - coop.PREFETCH_PAD) % coop.DEVICE_ALIGN == 0
            overlapped(words, ctl, W, oracle_port)
            outs = pr["rhs_out"] + [pr["T_out"]] + pr.get("jac_out", [])
            assert same([d(fetch(V, o)) for o in outs], [d(fetch(W, o)) for o in outs])
            if "jac_out" not in pr:  # the LU factors are left alone
                assert W[:coop.E_SLOTS] == [u(1.0 + k) for k in range(coop.E_SLOTS)]


@pytest.mark.parametrize("G", coop.REGIME_LANES)
def test_regime_programs_equal_oracle(oracle_port, G):
    """The program of a temperature regime gives the oracle's Jacobian and RHS at
    temperatures inside it and next to its ends."""
    gen = coop.generate(G, ir_io.load(), regimes=coop.REGIMES)
    assert gen["warps"] == coop.MAX_WARPS
    for n, reg in enumerate(gen["regimes"]):
        lo, hi = reg["lo"], reg["hi"]
        for k, want in enumerate((lo * (1 + 1e-9), (lo * hi) ** 0.5, hi * (1 - 1e-9))):
            y = states(1, 1000 * G + 10 * n + k)[0]
            for _ in range(2):  # T is proportional to the energy
                V = start(gen, y, oracle_port)
                words, ctl = coop.device_words(reg["progs"]["rhs"], gen["nv"])
                overlapped(words, ctl, V, oracle_port)
                T = d(fetch(V, reg["progs"]["rhs"]["T_out"]))
                if lo < T <= hi:
                    break
                y[14] *= want / T
            assert lo < T <= hi
            assert same([d(fetch(V, o)) for o in reg["progs"]["rhs"]["rhs_out"]], oracle_port.rhs(y))
            pr = reg["progs"]["jrhs"]
            V = start(gen, y, oracle_port)
            words, ctl = coop.device_words(pr, gen["nv"])
            overlapped(words, ctl, V, oracle_port)
            assert same([d(fetch(V, o)) for o in pr["rhs_out"]], oracle_port.rhs(y))
            assert same([-d(fetch(V, o)) for o in pr["jac_out"]], oracle_port.jac(y))
