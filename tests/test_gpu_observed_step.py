"""A fresh context whose first observed run is a single step.  (The ring of
observables was taken as allocated for one step, and the read-back failed with
IBG_E_CUDA.)"""
import pytest

from ibisco_b200 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1], ids=["fp32", "fp64"])
def test_first_observed_run_of_one_step(sysdir, precision):
    g = native.System(native.Setup(sysdir("fluid")), precision)
    h = native.System(native.Setup(sysdir("fluid")), precision)
    g.set_state()
    h.set_state()
    (o,) = g.run(1, 1, observe=True)
    ref = h.step(1)
    assert o["STEP"] == 1
    assert o["V_NB1"] == pytest.approx(ref["V_NB1"], rel=1e-9)
