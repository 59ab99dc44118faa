"""The vector-Jacobian programs (``gen/coop_adj.py``) against the straight-line derivative
code that the CPU oracle is compiled from: they claim its operations in its order, so
every value is equal to the last bit, at every temperature regime.  (A zero may have the
other sign: the straight-line code adds each contribution to a sum that starts at +0, the
programs start with the first contribution.)"""
import numpy as np
import pytest

from test_coop_diff_programs import INV, MASS, REGIME_OF, diff_oracle, execute, programs, state  # noqa: F401
from warp_reactor_gb300.gen import coop


def in_order(v):
    s = v[0]
    for x in v[1:]:
        s = s + x
    return s


def temperature(y):
    """T of a state, operation for operation as the programs' prologue has it."""
    X = np.maximum(y[:14], 1e-100)
    rho, sa = in_order(X * MASS), in_order(X)
    sg = in_order(X * coop.K_MP / rho * INV)
    sa = sa * (coop.K_MP / rho)
    return X, rho, y[14] / (sg / sa * coop.K_GAS * sa)


@pytest.mark.parametrize("T,regime", REGIME_OF)
def test_vector_jacobian_bits(programs, diff_oracle, oracle_port, T, regime):  # noqa: F811
    rng = np.random.default_rng(1000 + int(T))
    y = state(int(T) + 2, T)
    y[7] = 0.0  # below the floor
    mult = np.exp(rng.normal(0, 0.1, programs["nmult"]))
    X, rho, Tx = temperature(y)
    # T = e A / (R mp B): its adjoint reaches the state's fourteen densities and e
    c = in_order(X * INV) * (coop.K_GAS * coop.K_MP)

    def ybar(Xbar, Tbar):
        t = Tbar * (y[14] * rho / c)
        g = Xbar + t * (MASS / rho - INV / in_order(X * INV))
        return np.append(np.where(y[:14] < 1e-100, 0.0, g), Tbar * rho / c)

    f = diff_oracle.rhs(X, Tx, mult)
    fbar = rng.normal(size=15) / np.maximum(np.abs(f), 1e-30)
    Xbar, Tbar, mbar = diff_oracle.rhs_vjp(X, Tx, mult, fbar)
    _, _, out = execute(programs, "rhsvjp", regime, y, oracle_port, mult, fbar)
    assert np.array_equal(out, np.concatenate([ybar(Xbar, Tbar), mbar]))

    J = oracle_port.jac(y)
    Jbar = rng.normal(size=(15, 15)) / np.maximum(np.abs(J), 1e-30)
    Jbar[J == 0.0] = 0.0
    Xbar, Tbar = diff_oracle.jac_vjp(X, Tx, Jbar)
    _, _, out = execute(programs, "jacvjp", regime, y, oracle_port, mult, Jbar.ravel())
    assert np.array_equal(out, ybar(Xbar, Tbar))
