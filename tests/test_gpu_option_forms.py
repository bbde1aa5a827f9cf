"""The mixed pair sweep with options read at run time (XSPH, compatible energy
off, several NodeLists, tensile correction, the Q's expansion options, other
kernels) and with plain sums, on both sides of every node count where its form
changes: 40,000, 58,368 and 150,000 nodes with isotropic H, 20,000 with tensor H,
and the smallest boxes.  Against the FP64 oracle within the mixed mode's bound
for derivatives, 2e-5 of the largest (FP32 rounding of pair terms that cancel)."""
import numpy as np
import pytest

from spheral_gb300 import problems

from _parity import compare_fields

pytestmark = pytest.mark.gpu

FIELDS = ["massDensitySum", "DvDt", "DepsDt", "DvDx", "gradRho", "M", "maxViscousPressure", "DHDt", "Hideal",
          "massZerothMoment"]
LIMITED = dict(viscosity="limited_monaghan_gingold", Cl=2.0, Cq=2.0)
OPTIONS = {
    "xsph": dict(xsph=True),
    "xsph_limited": dict(xsph=True, **LIMITED),
    "no_compat": dict(compatible_energy=False),
    "no_compat_limited": dict(compatible_energy=False, **LIMITED),
    "two_lists": {},
    "two_lists_limited": dict(LIMITED),
    "tensile": dict(eps_tensile=0.3),
    "expansion": dict(linear_in_expansion=True, quadratic_in_expansion=True),
    "kernel": dict(kernel="nbspline", kernel_order=3),
    "plain": {},
    "plain_limited": dict(LIMITED),
    "plain_kernel": dict(kernel="nbspline", kernel_order=3),
}


def _compare(oracle_mod, p, option):
    from spheral_gb300.engine import Engine
    p.config.update(OPTIONS[option])
    if option.startswith("two_lists"):
        p.nodelist = (p.pos[:, 1] > 0.5).astype(np.int32)
        p.nodelists = [p.nodelists[0], dict(p.nodelists[0], gamma=1.4)]
    if option == "tensile":
        p.eps[: p.n // 2] *= -0.2   # tension
    eng = Engine.from_problem(p, precision="fp32_plain" if option.startswith("plain") else "fp32")
    orc = oracle_mod.Oracle(p)
    for e in (eng, orc):
        e.initialize()
        e.evaluate_derivatives()
    bad = compare_fields(eng, orc, FIELDS, 2e-5)
    assert not bad, bad


def _box(n, boundaries):
    side = int(np.ceil(n ** (1.0 / 3.0) - 1e-9))
    p = problems.random_box(n_side=side, seed=n % 97, nPerh=1.25, boundaries=boundaries)
    keep = np.sort(np.random.default_rng(n).permutation(p.n)[:n])
    for k in ("pos", "vel", "mass", "rho", "eps", "H", "nodelist"):
        setattr(p, k, np.ascontiguousarray(getattr(p, k)[keep]))
    return p


@pytest.mark.parametrize("n", [1000, 39999, 40000, 58368, 58369])
@pytest.mark.parametrize("option", list(OPTIONS))
def test_isotropic_options(native_lib, oracle_mod, option, n):
    _compare(oracle_mod, _box(n, "reflecting" if n in (1000, 40000) else "open"), option)


@pytest.mark.parametrize("n", [149999, 150000])
@pytest.mark.parametrize("option", ["xsph_limited", "two_lists", "tensile", "kernel", "plain", "plain_limited"])
def test_isotropic_options_large(native_lib, oracle_mod, option, n):
    _compare(oracle_mod, _box(n, "open"), option)


@pytest.mark.parametrize("shape", [(16, 13, 11), (30, 20, 33), (30, 20, 34)])
@pytest.mark.parametrize("option", ["xsph", "xsph_limited", "no_compat", "no_compat_limited", "two_lists", "tensile",
                                    "expansion", "kernel", "plain"])
def test_tensor_options(native_lib, oracle_mod, option, shape):
    _compare(oracle_mod, problems.stretched_box(*shape, seed=sum(shape)), option)
