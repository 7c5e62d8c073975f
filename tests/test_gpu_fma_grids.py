"""The fused multiply-add build on cell widths that are powers of two and on
ones that are not (the product build scales the derivative operator on the
former): one step from a smooth state within the specification's 1e-12 of the
product build, normwise per variable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    ((16,), 3, "FV", "llf", {}), ((12,), 4, "SD", "hllc", {}),
    ((8, 8), 3, "SD", "llf", {}), ((8, 10), 3, "FV", "hllc", {}), ((10, 16), 2, "FV", "lhllc", {}),
    ((8, 6), 3, "SD", "hllc", dict(viscosity=True, nu=1e-3)),
    ((4, 4, 4), 2, "FV", "hllc", {}), ((4, 3, 2), 4, "SD", "llf", {}),
]


def _smooth(xyz, case):
    d = xyz.shape[0]
    s = sum(np.sin(2 * np.pi * xyz[i] + 0.21 + 0.37 * i) for i in range(d))
    if case == 0:
        return 1.0 + 0.1 * s
    if case <= d:
        return 0.5 + 0.1 * case * np.cos(2 * np.pi * xyz[case - 1] + 0.53)
    return 1.0 + 0.05 * s


@pytest.mark.parametrize("case", CASES, ids=str)
def test_fused_build_step_on_any_cell_width(case):
    from spd_gb300 import SDADER_Simulator
    N, p, update, solver, kw = case
    kw = dict(p=p, N=N, init_fct=_smooth, update=update, FB=update == "FV", riemann_solver_sd=solver,
              riemann_solver_fv=solver, BC=(("periodic", "periodic"),) * len(N), verbose=False, **kw)
    a = SDADER_Simulator(**kw)
    f = SDADER_Simulator(fma=True, **kw)
    for s in (a, f):
        s.compute_dt()
        s.perform_update()
    U, F = a.dm.U_sp, f.dm.U_sp
    dev = max(float(np.max(np.abs(F[v] - U[v])) / np.max(np.abs(U[v]))) for v in range(U.shape[0]))
    moved = float(np.max(np.abs(U - SDADER_Simulator(**kw).dm.U_sp)))
    assert moved > 1e-4 and dev <= 1e-12, (moved, dev)
    a.close()
    f.close()
