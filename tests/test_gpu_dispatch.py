"""The variants of the nonbonded kernel, the list build and the step graphs, at
the sizes and forms where the host passes from one to another.

* tables on one grid against tables looked up by their descriptor: forces
  within 1e-5 (max-norm) of the FP64 path, the bar of the parity tests, and the
  same bits as slice lists, whose kernel always looks the descriptor up;
* lists from units of cells: identical to the oracle's, order included;
* ten steps per graph against single steps: the same bits.
"""
import numpy as np
import pytest

from ibisco_b200 import native, synth
from oracle.oracle import Oracle

from conftest import rel_maxnorm

pytestmark = pytest.mark.gpu


def typed_fluid(ntypes, fine, long, tmp, n=1500):
    """LJ fluid of several types; `fine` tables have half the others' bin and
    `long` ones reach twice as far."""
    spec = synth.lj_fluid(n=n, rho=8.0, seed=ntypes, nsteps=20, dmin=0.42)
    spec.types = [(f"T{t}", 0.072, "A") for t in range(1, ntypes + 1)]
    spec.itype = 1 + np.arange(n) % ntypes
    pairs = [(a, b) for a in range(1, ntypes + 1) for b in range(a, ntypes + 1)]
    spec.nb_tabs = [((a, b), synth.lj_table(f"nb{a}_{b}", 0.45 + 0.002 * (a + b), 2.0,
                                            2.4 if k < long else 1.2, 0.001 if k < fine else 0.002))
                    for k, (a, b) in enumerate(pairs)]
    return synth.write_system(spec, tmp)


@pytest.mark.parametrize("ntypes,fine,long", [(1, 0, 0), (2, 1, 0), (3, 0, 2), (8, 0, 0), (8, 35, 0), (9, 0, 0)])
def test_tables_on_one_grid_or_several(tmp_path, ntypes, fine, long):
    s = native.Setup(typed_fluid(ntypes, fine, long, str(tmp_path / "x")))
    a, slices, ref, staged = (native.System(s, p) for p in (0, 0, 1, 1))
    slices.set_list_form(native.LIST_PER_SLICE)
    for g in (a, slices, ref, staged):
        g.set_state()
    staged.set_tuning(nb_tables_smem=1)
    oa, os_, orf = a.forces(1), slices.forces(1), ref.forces(1)
    staged.forces(1)
    fa, fr = a.state64()["fxyz"], ref.state64()["fxyz"]
    assert np.array_equal(fa, slices.state64()["fxyz"])
    assert rel_maxnorm(fa, fr) < 1e-5
    assert rel_maxnorm(staged.state64()["fxyz"], fr) < 1e-9
    assert oa["V_NB1"] == pytest.approx(orf["V_NB1"], rel=1e-5)
    assert oa["V_NB1"] == pytest.approx(os_["V_NB1"], rel=1e-5)


@pytest.mark.parametrize("prec", [0, 1], ids=["fp32", "fp64"])
@pytest.mark.parametrize("m", [3, 4, 12])
def test_lists_from_cells_of_every_size(tmp_path, m, prec):
    """Boxes of m^3 cells with 0 to 97 particles each: units with a remainder,
    full ones, several per cell, neighbours through every face of the box."""
    sizes = [0, 1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 97]
    rng = np.random.default_rng(m)
    ncell = m ** 3
    if m < 12:
        cnt = np.array([sizes[k % len(sizes)] for k in range(ncell)])
    else:  # cells enough for a whole cell per unit: mostly few particles
        cnt = np.where(np.arange(ncell) % 29 == 0, rng.choice(sizes, ncell), rng.integers(0, 6, ncell))
    w = 1.43  # cell width, a little above the list radius of 1.4 nm
    cell = np.repeat(np.arange(ncell), cnt)
    at = np.stack([cell % m, cell // m % m, cell // (m * m)], -1)
    n = len(cell)
    spec = synth.lj_fluid(n=8, rho=8.0, seed=1, nsteps=10, dmin=0.1)
    order = rng.permutation(n)
    spec.pos = ((at + 0.005 + 0.99 * rng.random((n, 3))) * w - 0.5 * m * w)[order]
    spec.vel = np.zeros((n, 3))
    spec.itype = np.ones(n, int)
    spec.bonds = [[] for _ in range(n)]
    spec.molecules = [("bead", 1)] * n
    spec.box = (m * w,) * 3
    spec.control["atoms"] = n
    d = synth.write_system(spec, str(tmp_path / "x"))
    g = native.System(native.Setup(d), prec)
    g.set_state()
    o = Oracle(d)
    o.init(prec)
    lg, ng = g.neighbour_list(0)
    lo, no = o.neighbour_list(0, prec)
    np.testing.assert_array_equal(ng, no)
    np.testing.assert_array_equal(lg, lo)


@pytest.mark.parametrize("name", ["melt", "mix5_mts", "mix_npt", "hybrid"])
def test_groups_of_steps_equal_single_steps(sysdir, name):
    """A run launches whole groups of ten steps as one graph once their sequence
    has come before; steps launched one by one give the same bits, whatever the
    runs' lengths."""
    s = native.Setup(sysdir(name))
    a, b = native.System(s), native.System(s)
    a.set_state()
    b.set_state()
    first, oa = 1, []
    for n in (40, 9, 1, 31, 10, 19):
        oa += a.run(first, n, observe=True)
        first += n
    ob = [b.run(k, 1, observe=True)[0] for k in range(1, first)]
    assert oa == ob
    sa, sb = a.state64(), b.state64()
    for k in sa:
        assert np.array_equal(sa[k], sb[k]), k
