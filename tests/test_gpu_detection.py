"""Trouble detection at the edges of its fast test and of the ghost gather:
one limited step against the oracle, bit for bit, with tolerances around and
below one unit of the fast test, fluid at rest, states of large and small
magnitude, every boundary kind, and the smallest grids."""
import numpy as np
import pytest

from gpu_helpers import oracle_like

pytestmark = pytest.mark.gpu


def _state(scale, rest):
    def f(xyz, case):
        d = xyz.shape[0]
        x = xyz[0]
        s = sum(np.sin(2 * np.pi * (i + 1) * xyz[i]) for i in range(d))
        if case == 0:
            return scale * np.where(np.abs(x - 0.5) < 0.2, 1.5, 1.0 + 1e-7 * s)
        if case <= d:
            return np.zeros(x.shape) if rest else 0.3 * np.cos(2 * np.pi * x) + 1e-6 * case
        return scale * np.where(np.abs(x - 0.4) < 0.2, 1.2, 1.0)
    return f


CASES = [
    (1, (1,), 1, "periodic", 1e-5, 1.0, False), (1, (7,), 3, "reflective", 1e-5, 1.0, False),
    (2, (1, 1), 3, "gradfree", 1e-5, 1.0, False), (2, (5, 3), 2, "periodic", 2.0 ** -17, 1.0, False),
    (2, (4, 6), 3, "reflective", 1e-7, 1.0, True), (2, (3, 4), 3, "ic", 1e-3, 1e-30, False),
    (2, (6, 3), 1, "gradfree", 0.0, 1e30, True), (3, (2, 1, 3), 2, "reflective", 1e-5, 1.0, False),
    (3, (1, 2, 2), 1, "periodic", 1e-5, 1.0, True), (3, (2, 2, 1), 2, "ic", 1e-5, 1.0, False),
]


@pytest.mark.parametrize("ndim,N,p,bc,tol,scale,rest", CASES)
def test_limited_steps_match_oracle(ndim, N, p, bc, tol, scale, rest):
    from spd_gb300 import SDADER_Simulator
    s = SDADER_Simulator(p=p, N=N, init_fct=_state(scale, rest), update="FV", FB=True, tolerance=tol,
                         riemann_solver_sd="hllc", riemann_solver_fv="hllc", BC=((bc, bc),) * ndim,
                         min_rho=1e-40, max_rho=1e40, min_P=1e-40)
    o = oracle_like(s)
    for _ in range(2):
        s.compute_dt()
        o.compute_dt()
        assert s.dm.dt == o.dt
        s.perform_update()
        o.perform_update()
        np.testing.assert_array_equal(s.dm.troubles, o.troubles)
        np.testing.assert_array_equal(s.dm.theta, o.theta)
        np.testing.assert_array_equal(s.dm.U_sp, o.U_sp)
        np.testing.assert_array_equal(s.dm.W_cv, o.W_cv)
