"""Pairs at the cutoff at the sizes where their handling changes.

A simple cubic lattice whose spacing divides the cutoff has six neighbours of
every particle at the cutoff (to rounding), which the FP32 kernel leaves to the
FP64 decision.  Lists of one slot per thread of k_nb_collect's grid take them
along there, whichever block the two slots belong to; a batch and a system
alone must agree bit for bit.  Against the FP64 path, which evaluates the
same decision in FP64: 1e-5 of the largest force, the bar of the parity tests.
"""
import numpy as np
import pytest

from ibisco_b200 import native, synth

pytestmark = pytest.mark.gpu


def lattice(m, tmp):
    n = m ** 3
    spec = synth.lj_fluid(n=n, rho=8.0, seed=3, nsteps=10, dmin=0.05, shifted=False)
    a = 0.4  # three spacings are the 1.2 nm cutoff
    spec.box = (m * a,) * 3
    g = np.arange(m) * a - 0.5 * m * a + 0.5 * a
    spec.pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    spec.vel = np.zeros((n, 3))
    rng = np.random.default_rng(m)
    keep = rng.random(n) < 0.02  # a few particles off their site, so that forces do not cancel
    spec.pos[keep] += 0.01
    return synth.write_system(spec, tmp)


@pytest.mark.parametrize("m", [11, 12, 17])
def test_pairs_at_the_cutoff_across_blocks(tmp_path, m):
    s = native.Setup(lattice(m, str(tmp_path / "x")))
    a, b, c = (native.System(s, p) for p in (0, 0, 1))
    for g in (a, b, c):
        g.set_state()
    oa, oc = a.forces(1), c.forces(1)
    fa, fc = a.state64()["fxyz"], c.state64()["fxyz"]
    assert np.abs(fa - fc).max() <= 1e-5 * np.abs(fc).max()
    assert oa["V_NB1"] == pytest.approx(oc["V_NB1"], rel=1e-5)
    a.set_state()
    a.run(1, 3)
    batch = native.Batch([b])
    batch.run(3)
    sa, sb = a.state64(), b.state64()
    for k in sa:
        assert np.array_equal(sa[k], sb[k]), k
    batch.close()
