"""Gravity runs on a stream of its own beside the pair sweep; its profile scope
covers its own launches (some thirty, none below a microsecond), not what the
step still waits for once the pair sweep is done."""
import pytest

from spheral_gb300 import problems

pytestmark = pytest.mark.gpu


def test_gravity_scope_covers_its_launches(native_lib):
    from spheral_gb300.engine import Engine
    p = problems.evrard(n=40000, seed=1, opening=4.0)   # a short walk beside a long FP64 pair sweep
    eng = Engine.from_problem(p, precision="fp64")
    eng.initialize()
    eng.evaluate_derivatives()
    eng.profile(True)
    eng.profile_reset()
    for _ in range(4):
        eng.evaluate_derivatives()
    eng.profile(False)
    calls, ms = eng.profile_get("gravity")
    assert calls == 4 and ms / calls >= 0.03, (calls, ms)
