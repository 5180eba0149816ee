"""The coarse levels' sub-cycle in a thread-block cluster (wpf_coarse.cuh): grids
whose first cluster level is cut along x, y or z, has slabs of unequal size, short
last rows, a single plane or a single cell per row, or is one CTA's alone."""
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

SHAPES = [(3, 5, 7), (3, 1, 1), (47, 3, 2), (4, 2, 61), (5, 60, 7), (20, 18, 14), (33, 31, 29), (64, 20, 9),
          (96, 33, 17), (3, 90, 80)]


@pytest.mark.parametrize("nu", [1, 2, 3])
@pytest.mark.parametrize("shape", SHAPES)
def test_solve_matches_oracle(oracle_mod, shape, nu):
    from mizuho_edit_gb300.cases import make_case
    from mizuho_edit_gb300.sim import Simulation
    case = make_case(shape, log_var=1.0, corr_len=3.0, seed=sum(shape))
    ref = oracle_mod.OracleSim(case.params, case.permeab_rock, case.phase, case.concent)
    ref.calcPermeability()
    ref.solvePressure(oracle_mod.SOLVE_CG, 1e-14)
    # the residual bounds the error by about the condition number (n^2 times the
    # permeabilities' spread, below 1e5 here) times rtol
    for solver, rtol, bound in (("fp64", 1e-12, 1e-8), ("mixed", 1e-11, 1e-7)):
        with Simulation(case.params, case.permeab_rock, case.phase, case.concent, solver=solver, rtol=rtol,
                        smooth_sweeps=nu) as sim:
            sim.calcPermeability()
            st = sim.solvePressure()
            assert st.converged
            assert st.inner_iterations <= 60      # the cycle preconditions (unpreconditioned CG: hundreds)
            assert rel_l2(sim.download("pressure"), ref.pressure) < bound
