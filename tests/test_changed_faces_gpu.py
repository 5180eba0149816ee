"""calcPermeability lists the changed faces of a block of 32 x 4 x 2 cells and
the cells that they need: steps at extents around the block's, from a rough
state (nearly every face changes) and a smooth one (few do), follow the oracle.
So does the update's classification, which takes two cells of a row per thread:
odd, even and short rows."""
import pytest

from conftest import rel_l2
from test_gpu_parity import _case, _pair, _rough_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rough", [False, True])
@pytest.mark.parametrize("n", [(31, 3, 1), (32, 4, 2), (33, 5, 3), (63, 9, 4), (5, 40, 7)])
def test_steps_follow_the_oracle(oracle_mod, n, rough):
    case = _case(n, seed=21, log_var=1.0, corr_len=3.0)
    if rough:
        case = _rough_state(case, seed=22)
    ref, sim = _pair(case)
    with sim:
        for _ in range(4):
            sim.step()
            ref.step(oracle_mod.SOLVE_CG, 1e-14)
            if abs(ref.phase).max() > 2.0:   # a 5-cell domain: the oracle's first step already leaves [-1, 1]
                break
        f = sim.download("phase", "concent", "pressure")
    # the bounds of the comparison over 100 steps
    assert rel_l2(f["pressure"], ref.pressure) < 1e-10
    assert rel_l2(f["phase"], ref.phase) < 1e-9
    assert rel_l2(f["concent"], ref.concent) < 1e-9
