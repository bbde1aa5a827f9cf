"""The time-step vote that the mixed mode takes from FP64 limits (the dt query,
and the CRKSPH step) is the FP64 limit to the last bit: with the gas at rest it
is cfl times the smallest h / nPerh / c of the state's own fields."""
import numpy as np
import pytest

from spheral_gb300 import problems

pytestmark = pytest.mark.gpu


def _rest(p):
    p.vel[:] = 0.0
    p.config.update(dt_min=0.0, dt_max=1.0e3, last_dt=1.0e3, dt_growth=2.0, cfl=1.0)
    return p


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("hydro", ["sph", "crksph"])
def test_dt_is_the_fp64_limit(native_lib, hydro, seed):
    from spheral_gb300.engine import DT_REASONS, Engine
    make = problems.random_box if hydro == "sph" else problems.crksph_box
    p = _rest(make(n_side=11 + 2 * seed, seed=seed))
    eng = Engine.from_problem(p, precision="fp32")
    eng.initialize()
    eng.sum_density()
    hinv, cs = eng.field("H")[:, 0], eng.field("soundSpeed")
    want = np.min(1.0 / hinv / p.nodelists[0]["nPerh"] / (cs + np.finfo(float).eps))
    dt, reason = eng.dt()[:2]
    assert dt == want and reason == DT_REASONS[0]
    if hydro == "crksph":   # the vote on the density sweep
        assert eng.step() == want
