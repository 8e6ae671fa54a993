"""Pairs at the end of their nonbonded table on the FP64 path: a distance of
NDAT + 1 bins is past it (IBG_E_TABLE_RANGE), one of less is not.  The quotient
r/bin is a whole number there, which r times 1/bin can miss (with two of the
three bins it does)."""
import numpy as np
import pytest

from ibisco_b200 import native, synth
from oracle.oracle import Oracle, OracleError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("smem", [0, 1], ids=["tables_l1", "tables_smem"])
@pytest.mark.parametrize("dr,missed", [(0.0019, True), (0.001942, True), (0.002, False)])
def test_a_pair_on_the_end_of_its_table(tmp_path, dr, missed, smem):
    spec = synth.lj_fluid(n=8, rho=8.0, seed=1, nsteps=10, dmin=0.1)
    spec.nb_tabs = [((1, 1), synth.lj_table("nb11", 0.47, 3.5, 255 * dr, dr))]
    spec.pos = np.array([[0.0, y, z] for y in (-2.0, 2.0) for z in (-2.0, 2.0) for _ in (0, 1)])
    spec.vel[:] = 0.0
    spec.box = (9.0, 9.0, 9.0)
    d = synth.write_system(spec, str(tmp_path / "x"))
    s = native.Setup(d)
    b, nd = float(s.array("BINNB")[-1]), int(s.array("NDATNB")[-1])
    assert nd == 255 and (256 * b * (1.0 / b) < 256) == missed
    x, v, box = s.initial_state()
    g = native.System(s, native.IBG_PREC_FP64_PLAIN)
    g.set_tuning(nb_tables_smem=smem)
    o = Oracle(d)
    o.init(1)
    for last, inside in ((256, False), (np.nextafter(np.float32(256 * b), np.float32(0)) / b, True)):
        x = x.copy()
        x[1::2, 0] = np.array([200, 250, 230, last]) * b
        g.set_state(x, v, box)
        o.set_state(x, v, box, 1)
        if inside:
            og = g.forces(1)
            o.forces(1, 1)
            assert og["V_NB1"] == pytest.approx(o.obs(1)["V_NB1"], rel=1e-12)
        else:
            with pytest.raises(OracleError):
                o.forces(1, 1)
            with pytest.raises(native.IbiscoError) as e:
                g.forces(1)
            assert e.value.code == -9
