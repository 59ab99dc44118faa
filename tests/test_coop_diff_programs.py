"""The differentiation form's vector programs (``gen/coop_adj.py``), run on the CPU as the
device runs them: the forward programs give the oracle's Jacobian and RHS with
multipliers bit for bit; the vector-Jacobian products agree with the oracle's
tangents in inner products, <fbar, df> = <ybar, dy> + <mbar, dm> and <Jbar, dJ> = <ybar, dy>.
Tolerance: a product sums some 1e4 rounded terms, 1e-16 each, so 1e-10 of the terms'
magnitudes leaves two digits for cancellation."""
import numpy as np
import pytest

from test_coop_device_words import overlapped, start
from test_coop_programs import d, fetch, same, u
from warp_reactor_gb300.gen import coop, coop_adj

MASS = np.array(coop.MASS)
INV = np.array([coop.inv_gm1(n) for n in range(14)])


@pytest.fixture(scope="module")
def diff_oracle(built):
    from oracle import oracle as O
    return O.load_diff()


@pytest.fixture(scope="module")
def programs():
    return coop_adj.generate()


def state(seed, T):
    """A state with the abundances of a collapsing cell, spread, at temperature T."""
    rng = np.random.default_rng(seed)
    X = np.array([3e-2, 3e-2, 1e5, 1e-6, 1e-15, 1e-9, 1e-8, 1e-18, 1e2, 1e-18, 1e-10, 1e-30, 1e-25, 1e4])
    X = X * 10.0 ** rng.uniform(-1, 1, 14)
    e = T * coop.K_GAS * coop.K_MP * (X @ INV) / (X @ MASS)
    return np.append(X, e)


def temperature(oracle, y):
    return y[14] * (y[:14] @ MASS) / (coop.K_GAS * coop.K_MP * (y[:14] @ INV))


def execute(gen, kind, regime, y, oracle, mult, seeds=()):
    pr = next(p for k, r, p in gen["progs"] if (k, r) == (kind, regime))
    V = start({**gen, "nv": gen["nva"]}, y, oracle)
    for r, m in enumerate(mult):
        V[gen["mult"] + r] = u(m)
    for i, s in enumerate(seeds):
        V[(gen["fbar"] if kind == "rhsvjp" else 0) + i] = u(s)
    words, ctl = coop.device_words(pr, pr["nv"])
    overlapped(words, ctl, V, oracle)
    return pr, V, np.array([d(fetch(V, o)) for o in pr["out"]])


REGIME_OF = [(150.0, 0), (350.0, 0), (350.0, 1), (800.0, 2), (1100.0, 3), (1500.0, 4), (3000.0, 5), (3000.0, 6),
             (9000.0, 0)]


@pytest.mark.parametrize("T,regime", REGIME_OF)
def test_forward_programs(programs, diff_oracle, oracle_port, T, regime):
    y = state(int(T) + regime, T)
    mult = np.exp(np.random.default_rng(regime).normal(0, 0.1, programs["nmult"]))
    for kind in ("jrhsp", "rhsp"):
        pr, V, f = execute(programs, kind, regime, y, oracle_port, mult)
        Tx = d(fetch(V, pr["T_out"]))
        assert same(f, diff_oracle.rhs(np.maximum(y[:14], 1e-100), Tx, mult))
        if kind == "jrhsp":
            assert same([-d(fetch(V, o)) for o in pr["jac_out"]], oracle_port.jac(y))


@pytest.mark.parametrize("T,regime", REGIME_OF)
def test_vector_jacobian_products(programs, diff_oracle, oracle_port, T, regime):
    D = diff_oracle
    rng = np.random.default_rng(int(T))
    y = state(int(T) + 1, T)
    y[9] = 0.0  # below the floor: no adjoint reaches it
    mult = np.exp(rng.normal(0, 0.1, programs["nmult"]))
    dy = rng.normal(size=15) * y
    dm = rng.normal(size=len(mult))
    X = np.maximum(y[:14], 1e-100)
    dX = np.where(y[:14] < 1e-100, 0.0, dy[:14])
    A, B = X @ MASS, X @ INV
    Tx = temperature(D, np.append(X, y[14]))
    dT = Tx * (dy[14] / y[14] + dX @ MASS / A - dX @ INV / B)

    f, df = D.rhs_jvp(X, Tx, mult, dX, dT, dm)
    fbar = rng.normal(size=15) / np.maximum(np.abs(f), 1e-30)
    _, _, out = execute(programs, "rhsvjp", regime, y, oracle_port, mult, fbar)
    lhs, terms = fbar @ df, np.concatenate([out[:15] * dy, out[15:] * dm])
    assert out[9] == 0.0
    assert abs(lhs - terms.sum()) <= 1e-10 * (np.abs(terms).sum() + np.abs(fbar * df).sum())

    J, dJ = D.jac_jvp(X, Tx, dX, dT)
    Jbar = rng.normal(size=(15, 15)) / np.maximum(np.abs(J), 1e-30)
    Jbar[J == 0.0] = 0.0
    _, _, out = execute(programs, "jacvjp", regime, y, oracle_port, mult, Jbar.ravel())
    lhs, terms = (Jbar * dJ).sum(), out * dy
    assert abs(lhs - terms.sum()) <= 1e-10 * (np.abs(terms).sum() + np.abs(Jbar * dJ).sum())
