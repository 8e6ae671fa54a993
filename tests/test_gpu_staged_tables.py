"""Tables staged in shared memory by several contexts of one process: the
kernel's shared-memory limit is shared, so a context with small tables must not
take it away from one with large tables."""
import numpy as np
import pytest

from ibisco_b200 import native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1], ids=["fp32", "fp64"])
def test_contexts_with_staged_tables_of_different_sizes(tmp_path, prec):
    made = []
    for k, dr in enumerate((0.0002, 0.0005)):  # 6,001 and 2,401 rows: more than 48 kB both
        spec = synth.lj_fluid(n=1500, rho=8.0, seed=3, nsteps=10, dmin=0.42)
        spec.nb_tabs = [((1, 1), synth.lj_table("nb11", 0.47, 3.5, 1.2, dr))]
        g = native.System(native.Setup(synth.write_system(spec, str(tmp_path / str(k)))), prec)
        g.set_tuning(nb_tables_smem=1)
        assert g.tuning()["nb_tables_smem"] == 1
        g.set_state()
        made.append(g)
    staged = []
    for g in made:
        g.forces(1)
        staged.append(g.state64()["fxyz"])
    for g, f in zip(made, staged):
        g.set_tuning(nb_tables_smem=0)
        g.set_state()
        g.forces(1)
        if prec == 0:  # integer sums
            assert np.array_equal(g.state64()["fxyz"], f)
        else:  # FP64 atomics add in any order
            np.testing.assert_allclose(g.state64()["fxyz"], f, rtol=0, atol=1e-12 * np.abs(f).max())
