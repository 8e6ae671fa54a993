"""Bonded terms where a rounding is amplified, against the oracle in FP64, whose
expressions the FP64 path restates operation by operation.

Where only lengths and sines that scale a force are divided by differently (one
reciprocal each), a force component differs by at most about a dozen roundings,
with the arc cosine's last bit a few 1e-15 of the largest force; the bar of
1e-12 leaves a margin of some hundred.
"""
import numpy as np
import pytest

from ibisco_b200 import native, synth
from oracle.oracle import Oracle

from conftest import rel_maxnorm

pytestmark = pytest.mark.gpu


def chains(pos, itype, ntypes, nper, **tabs):
    """Chains of nper beads at the given places in a 9 nm box, each farther
    from the others than the cutoff; without tables for them, the chains have
    no angles or torsions."""
    spec = synth.polymer_melt(nchains=1, nper=4, ntypes=ntypes, nsteps=10)
    n = len(pos)
    spec.pos, spec.vel, spec.itype = pos, np.zeros((n, 3)), itype
    spec.bonds = synth.chain_bonds(n // nper, nper)
    spec.molecules = [("chain", nper)] * (n // nper)
    spec.box = (9.0, 9.0, 9.0)
    spec.control = dict(spec.control, atoms=n)
    for k, v in tabs.items():
        setattr(spec, k, v)
    return spec


def test_torsions_next_to_straight_angles(tmp_path):
    """i-j-k, j-k-l or both within 1e-5 rad of straight: 1/sin of the angle from
    1 - cos^2 amplifies every rounding of the cosine by 1/sin^2 = 1e10."""
    rng = np.random.default_rng(5)
    pos = []
    for c in range(125):
        at = np.array([c % 5, c // 5 % 5, c // 25]) * 1.8 - 3.6
        u, v = rng.normal(size=3), rng.normal(size=3)
        u /= np.linalg.norm(u)
        v -= (v @ u) * u
        v /= np.linalg.norm(v)
        w = np.cross(u, v)
        b = 0.153
        phi = np.radians(rng.uniform(50, 130))
        side = np.cos(phi) * v + np.sin(phi) * w  # l's side of the axis, at the dihedral phi from i's
        s1, s2 = [(1e-5, 0.8), (0.8, 1e-5), (1e-5, 1e-5)][c % 3]
        j, k = -0.5 * b * u, 0.5 * b * u
        i = j - b * np.cos(s1) * u + b * np.sin(s1) * v
        l = k + b * np.cos(s2) * u + b * np.sin(s2) * side
        pos += [at + x for x in (i, j, k, l)]
    d = synth.write_system(chains(np.array(pos), np.ones(500, int), 1, 4), str(tmp_path / "x"))
    g = native.System(native.Setup(d), native.IBG_PREC_FP64_PLAIN)
    g.set_state()
    og = g.forces(1)
    o = Oracle(d)
    o.init(1)
    o.forces(1, 1)
    fo = o.state(1)["fxyz"]
    assert np.isfinite(fo).all() and np.abs(fo).max() > 1e5  # the sines are there
    assert rel_maxnorm(g.state64()["fxyz"], fo) < 1e-12
    assert og["V_TORSION1"] == pytest.approx(o.obs(1)["V_TORSION1"], rel=1e-12)


@pytest.mark.parametrize("prec", [0, 1], ids=["fp32", "fp64"])
def test_bonds_that_end_on_the_end_of_their_table(tmp_path, prec):
    """A bond of exactly NDAT + 1 bins counts as overextended, one of NDAT bins
    does not: the quotient length/bin is a whole number there, which the
    length times 1/bin can miss (with two of the three tables it does)."""
    bins = (0.0019, 0.001942, 0.002)
    at = [np.array([c % 4, c // 4, 0]) * 1.8 - 2.7 for c in range(12)]
    spec = chains(np.zeros((24, 3)), np.repeat(np.arange(12) % 3 + 1, 2), 3, 2, angle_tabs=[], torsion_tabs=[])
    spec.bond_tabs = [((t + 1, t + 1), synth.harmonic_bond_table(f"bond{t}", 0.3, 1.0e3, 255 * b, b))
                      for t, b in enumerate(bins)]
    for c in range(12):  # x = 0 for the first of each pair, so that the difference is exact
        spec.pos[2 * c] = spec.pos[2 * c + 1] = [0.0, at[c][0], at[c][1]]
    d = synth.write_system(spec, str(tmp_path / "x"))
    s = native.Setup(d)
    b, nd = s.array("BINB").astype(np.float64), s.array("NDATB")
    b, nd = b[-3:], nd[-3:]
    assert list(nd) == [255] * 3
    assert [256 * x * (1.0 / x) < 256 for x in b] == [True, True, False]
    x, v, box = s.initial_state()
    x = x.copy()
    for c in range(12):
        x[2 * c + 1, 0] = (256, 256, 255, 255)[c // 3] * b[c % 3]
    g = native.System(s, prec)
    g.set_state(x, v, box)
    o = Oracle(d)
    o.init(1)
    o.set_state(x, v, box, 1)
    og = g.forces(1)
    o.forces(1, 1)
    oo = o.obs(1)
    assert oo["BOND_OVEREXT"] == 6
    assert og["BOND_OVEREXT"] == 6
    assert og["V_BOND1"] == pytest.approx(oo["V_BOND1"], rel=1e-12)
