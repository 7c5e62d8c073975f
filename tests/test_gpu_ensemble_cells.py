"""Packed ensembles at the largest blocks of the interior kernel, whose
launches within a step need different amounts of shared memory: bit-identical
to the instances stepped alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sim(p, m, N, seed):
    from spd_gb300 import SDADER_Simulator
    from spd_gb300.initial_conditions import kelvin_helmholtz, sine_wave
    init = kelvin_helmholtz(N[0], seed=seed) if len(N) == 2 else sine_wave
    return SDADER_Simulator(p=p, m=m, N=N, init_fct=init, update="FV", FB=True, riemann_solver_sd="hllc",
                            riemann_solver_fv="hllc", BC=(("periodic", "periodic"),) * len(N), verbose=False)


# (p, m, sizes, cells per block, None for the context's own)
@pytest.mark.parametrize("p, m, sizes, cells", [(3, 3, ((12, 12), (16, 16)), 64), (4, 4, ((10, 10), (8, 8)), 32),
                                                (4, 5, ((2, 2, 2), (3, 3, 3)), None)])
def test_packed_ensemble_at_large_blocks(p, m, sizes, cells):
    from spd_gb300 import SDADER_Ensemble
    sims = [_sim(p, m, N, 5 + i) for i, N in enumerate(sizes)]
    alone = [_sim(p, m, N, 5 + i) for i, N in enumerate(sizes)]
    steps = 2
    if cells is None:
        ens = SDADER_Ensemble(sims)
    else:
        # form and block are fixed: the probe's steps count
        ens = SDADER_Ensemble(sims, packed=False, nstreams=1)
        tuning = ens.autotune(streams=(), cpbs=(cells,), probe_launches=1, packed=(True,))
        assert not tuning["skipped"] and tuning["cells_per_block"] == cells
        steps += 2
    ens.perform_iterations(2)
    for s, a in zip(sims, alone):
        for _ in range(steps):
            a.compute_dt()
            a.perform_update()
        assert s.n_step == steps
        assert np.array_equal(s.dm.U_sp, a.dm.U_sp)
    ens.close()
