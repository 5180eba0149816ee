"""The showProgress reductions at the edges of their walk: rows shorter than a warp,
one longer than a few, more rows than the blocks take in one go, single planes;
and the values that leave the integer sum (|phase| >= 2, Inf, NaN)."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(3, 1, 1), (5, 7, 3), (30, 4, 4), (31, 3, 9), (62, 5, 2), (129, 2, 3), (4, 130, 70), (200, 90, 70)]
KEYS = ("pv", "vcal", "rwhmax", "phase_max", "phase_min", "concent_max", "concent_min")


def _noalloc(p, ph, cc):
    import torch
    from mizuho_edit_gb300 import capi
    cp = capi.Params(p.nx, p.ny, p.nz, p.ix_ref, p.iy_ref, p.iz_ref, p.dx, p.epsilon, p.lambda_, p.porosity,
                     p.viscosity, p.diffusion, p.ral, p.rat, p.permeab_hole, p.alpha, p.tfac)
    t = [torch.from_numpy(np.ascontiguousarray(a.ravel(order="F"))).cuda() for a in (ph, cc)]
    d = capi.Diag()
    capi.check(capi.load().wpf_reduce_noalloc(C.byref(cp), C.c_void_p(t[0].data_ptr()), C.c_void_p(t[1].data_ptr()),
                                              C.byref(d), None), "wpf_reduce_noalloc")
    return d.as_dict()


@pytest.mark.parametrize("shape", SHAPES)
def test_reductions_match_oracle(oracle_mod, shape):
    from mizuho_edit_gb300.cases import grf, make_case
    from mizuho_edit_gb300.sim import Simulation
    case = make_case(shape, log_var=1.0, corr_len=2.0, seed=7)
    case.params.dx = 0.37
    case.phase = np.tanh(1.5 * grf(shape, 2.0, 8)) * 1.05
    case.concent = np.clip(0.5 + 0.5 * grf(shape, 3.0, 9), 0, 1)
    ref = oracle_mod.OracleSim(case.params, case.permeab_rock, case.phase, case.concent)
    # a pressure handed over: the reductions are the subject, and the overshooting
    # phase makes some permeabilities negative, which no solve is defined for
    pr = np.asfortranarray(np.random.default_rng(10).random(tuple(n + 2 for n in shape)))
    with Simulation(case.params, case.permeab_rock, case.phase, case.concent, solver="fp64") as sim:
        sim.upload(pressure=pr)
        sim.calcPermeability()
        got, f = sim.diagnostics(), sim.download("phase", "concent", "pressure")
        want = ref.diagnostics()
        other = _noalloc(case.params, f["phase"], f["concent"])
        # sums of at most 1.3e6 terms below 2: the compensated sum is off by 1e-16 of it, the exact one rounded once
        for k in KEYS:
            assert got[k] == pytest.approx(want[k], rel=1e-13, abs=1e-300), k
            assert other[k] == got[k], k
        assert got["pressure_ref"] == f["pressure"][case.params.ix_ref, case.params.iy_ref, case.params.iz_ref]
        K = sim.download("permeab")
        u = -K[1, 1, 1:-1, 1:-1] / case.params.viscosity * (f["pressure"][2, 1:-1, 1:-1] - f["pressure"][1, 1:-1, 1:-1])
        assert got["inlet_flux"] == pytest.approx(float(u.sum()) * case.params.dx, rel=1e-12)


@pytest.mark.parametrize("values", [(5.0, -3.5), (2.0, -2.0), (1e200, 1.0), (math.inf, 0.0), (math.nan, 0.5),
                                    (5e-324, -1e-310)])
def test_reductions_of_extreme_values(values):
    from mizuho_edit_gb300.cases import make_case
    p = make_case((6, 5, 4), log_var=0.0).params
    ph = np.full((8, 7, 6), 0.25, order="F")
    cc = np.zeros((8, 7, 6), order="F")
    ph[2, 3, 2], ph[4, 2, 3] = values
    inner = ph[1:-1, 1:-1, 1:-1]
    d = _noalloc(p, ph, cc)
    for key, terms, c in (("pv", 1.0 - inner, 0.5 * p.porosity), ("vcal", 1.0 + inner, 0.5 * (1 - p.porosity))):
        want = math.fsum(terms.ravel()) if np.isfinite(terms).all() else math.nan
        if math.isnan(want):
            assert math.isnan(d[key])
        else:
            assert d[key] == pytest.approx(c * p.dx ** 3 * want, rel=1e-13)
    # an infinite or undefined phase has no place in the maxima's range, as fmax has it
    fin = ph[~np.isnan(ph)]
    assert d["phase_max"] == fin.max() and d["phase_min"] == fin.min()
