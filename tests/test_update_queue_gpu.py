"""The interface update of the mixed form: cells whose phase rate takes the FP64
form (the anisotropy guard) queue up within a block until they fill its warps.
From a rough state, where both kinds of cells abound, and from a smooth one,
where almost none queue, one step agrees with the form that keeps every cell's
rate in FP64."""
import numpy as np
import pytest

from test_gpu_parity import _case, _rough_state

pytestmark = pytest.mark.gpu


# interface cells: fewer than one block's threads, a few blocks' worth, more than the grid's
@pytest.mark.parametrize("rough", [True, False])
@pytest.mark.parametrize("n", [(5, 4, 3), (20, 14, 12), (33, 17, 9), (96, 80, 64)])
def test_queued_cells_match_fp64_rates(oracle_mod, n, rough):
    from mizuho_edit_gb300.sim import Simulation
    case = _case(n, seed=4, log_var=1.0, corr_len=3.0)
    if rough:
        case = _rough_state(case, seed=8)
    out = []
    for exact in (False, True):
        with Simulation(case.params, case.permeab_rock, case.phase, case.concent, solver="mixed", rtol=1e-10,
                        fp64_update=exact) as sim:
            before = sim.download("phase", "concent")
            sim.step()
            after = sim.download("phase", "concent")
            out.append([after[k] - before[k] for k in ("phase", "concent")])
    # FP32 rates: a relative 1e-7 per operation, some tens of operations, and
    # the pressure to 1e-10 times its condition; of the largest change
    for lo, hi in zip(*out):
        scale = np.max(np.abs(hi))
        assert np.max(np.abs(lo - hi)) <= 2e-5 * scale
