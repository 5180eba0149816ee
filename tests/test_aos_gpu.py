"""The interleaved arrays of a download (permeab, velocity) are written by one
kernel, into page-locked memory in place (16-byte pieces, or 8-byte ones when
the array is off that boundary) or wherever an ordinary array lives: the same
bits each way, and the oracle's values, at sizes around the kernel's tile of
512 cells."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(__file__))
from test_gpu_parity import _case, _pair, _rough_state
from test_host_io_gpu import Pinned

pytestmark = pytest.mark.gpu


# halo boxes of 150 cells (one partial tile), 512 + 28, and many odd tiles
@pytest.mark.parametrize("n", [(3, 4, 3), (7, 4, 8), (33, 17, 9), (20, 14, 12)])
def test_interleaved_download(oracle_mod, n):
    from mizuho_edit_gb300 import capi
    case = _rough_state(_case(n, seed=6, log_var=1.0, corr_len=3.0))
    ref, sim = _pair(case)
    with sim:
        ref.calcPermeability(); ref.solvePressure(oracle_mod.SOLVE_CG, 1e-14); ref.calcVelocity()
        sim.calcPermeability(); sim.solvePressure(); sim.calcVelocity()
        plain = sim.download("permeab", "velocity")
        # the bounds of the routine-by-routine comparison with the oracle
        err = np.max(np.abs(plain["permeab"] - ref.permeab)) / np.max(np.abs(ref.permeab))
        assert err < 1e-14
        assert np.linalg.norm(plain["velocity"] - ref.velocity) < 1e-10 * np.linalg.norm(ref.velocity)
        halo = sim.halo_shape
        for offset in (0, 8):
            k, v = Pinned(sim.L, (4,) + halo, 1, offset), Pinned(sim.L, (3,) + halo, 1, offset)
            try:
                k.arrays[0][:] = np.nan
                v.arrays[0][:] = np.nan
                capi.check(sim.L.wpf_download(sim.h, None, None, None, k.dp(0), v.dp(0), None, None),
                           "wpf_download")
                assert np.array_equal(k.arrays[0].view(np.int64), plain["permeab"].view(np.int64))
                assert np.array_equal(v.arrays[0].view(np.int64), plain["velocity"].view(np.int64))
            finally:
                k.free()
                v.free()
