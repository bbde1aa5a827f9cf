"""Both sides of the node counts where the sweeps change their lanes per node.
FP64: 30,000 nodes.  Mixed: the energy sweep (6,000 and 40,000, seen in a step),
the lean tensor pair sweep (15,000 and 25,000) and the CRKSPH sweeps (6,000,
25,000 and 35,000).  Against the FP64 oracle: 1e-12 for FP64 derivatives, 2e-5
for mixed ones, 5e-5 for the mixed state after a step."""
import numpy as np
import pytest

from spheral_gb300 import problems

from _parity import compare_fields

pytestmark = pytest.mark.gpu


def _both(oracle_mod, p, precision="fp32"):
    from spheral_gb300.engine import Engine
    eng, orc = Engine.from_problem(p, precision=precision), oracle_mod.Oracle(p)
    eng.initialize()
    orc.initialize()
    return eng, orc


def _box(n):
    side = int(np.ceil(n ** (1.0 / 3.0)))
    p = problems.random_box(n_side=side, seed=n % 89, nPerh=1.25, boundaries="open")
    keep = np.sort(np.random.default_rng(n).permutation(p.n)[:n])
    for k in ("pos", "vel", "mass", "rho", "eps", "H", "nodelist"):
        setattr(p, k, np.ascontiguousarray(getattr(p, k)[keep]))
    return p


@pytest.mark.parametrize("n", [29999, 30000])
def test_fp64_line(native_lib, oracle_mod, n):
    eng, orc = _both(oracle_mod, _box(n), "fp64")
    eng.evaluate_derivatives()
    orc.evaluate_derivatives()
    bad = compare_fields(eng, orc, ["DvDt", "DepsDt", "DvDx", "gradRho", "M", "massZerothMoment", "omegaGradh"], 1e-12)
    assert not bad, bad


@pytest.mark.parametrize("n", [5999, 6000, 39999, 40000])
def test_energy_lines(native_lib, oracle_mod, n):
    eng, orc = _both(oracle_mod, _box(n))
    for _ in range(2):
        a, b = eng.step(), orc.step()
        assert abs(a - b) <= 1e-5 * b
    bad = compare_fields(eng, orc, ["massDensity", "velocity", "specificThermalEnergy", "H"], 5e-5)
    assert not bad, bad


@pytest.mark.parametrize("shape", [(30, 20, 24), (30, 20, 26), (30, 20, 41), (30, 20, 42)])
def test_tensor_lines(native_lib, oracle_mod, shape):
    eng, orc = _both(oracle_mod, problems.stretched_box(*shape, seed=sum(shape)))
    eng.evaluate_derivatives()
    orc.evaluate_derivatives()
    bad = compare_fields(eng, orc, ["DvDt", "DepsDt", "DvDx", "massDensitySum", "DHDt", "Hideal", "massZerothMoment",
                                    "maxViscousPressure"], 2e-5)
    assert not bad, bad


@pytest.mark.parametrize("side", [18, 19, 29, 30, 32, 33])
def test_crk_lines(native_lib, oracle_mod, side):
    p = problems.crksph_box(n_side=side, seed=side, boundaries="reflecting" if side == 29 else "periodic")
    p.config.update(xsph=False)
    eng, orc = _both(oracle_mod, p)
    eng.sum_density()
    orc.sum_density()
    eng.evaluate_derivatives()
    orc.rk_corrections()
    orc.evaluate_derivatives()
    bad = compare_fields(eng, orc, ["massDensity", "DvDt", "DepsDt", "DvDx", "Hideal", "massZerothMoment",
                                    "rkCorrections"], 2e-5)
    assert not bad, bad
