"""Two borders of the list build: storage outgrown inside a ten-step graph, and
whole-cell units whose candidates do not fit one stage."""
import numpy as np
import pytest

from ibisco_b200 import native, synth
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def test_storage_outgrown_inside_a_group_of_steps(tmp_path):
    """A fluid that flows together, lists every five steps.  The storage is set
    to what the lists need up to step 60, and outgrown later, at a step whose
    group of ten (61.., 71.., ...) is launched as one graph: the rest of that
    group must do nothing, and the run goes on from the step that aborted with
    the bits of single steps over storage that never ran out."""
    spec = synth.lj_fluid(n=3000, rho=3.0, seed=5, nsteps=200, dmin=0.42, shifted=True, dt=0.005)
    spec.control["update_neighbour_list"] = 5
    spec.vel = spec.vel - 0.7 * spec.pos
    s = native.Setup(synth.write_system(spec, str(tmp_path / "x")))
    steps = 130
    one, g = native.System(s), native.System(s)
    one.set_state()
    one.run(1, 34)
    native.lib().ibg_set_list_rows(one._h, 100)
    need = {}
    o1 = []
    for k in range(35, steps + 1):
        o1 += one.run(k, 1, observe=True)
        if k % 5 == 0:
            need[k] = -(-int(one.neighbour_counts(0).max()) // 8)
    rows = max(v for k, v in need.items() if k <= 60)
    later = [k for k in sorted(need) if need[k] > rows]
    assert rows < 100 and later and later[0] <= 120  # inside a whole group of the run below
    g.set_state()
    g.run(1, 34)
    grown = g.timing()["list_growths"]
    native.lib().ibg_set_list_rows(g._h, rows)
    og = g.run(35, steps - 34, observe=True)
    assert g.timing()["list_growths"] > grown
    assert og == o1
    a, b = g.state64(), one.state64()
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("prec", [0, 1], ids=["fp32", "fp64"])
def test_dense_cells_among_many(tmp_path, prec):
    """12^3 cells, so that a unit is a whole cell; 5^3 neighbouring ones hold 120
    to 130 particles each (14 of them 1,680 and more candidates, several stages
    for each of a cell's groups of 32), the others up to three."""
    m, w = 12, 1.43
    rng = np.random.default_rng(17 + prec)
    ijk = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    dense = ((ijk - 9) % m < 5).all(1)  # across the box's faces
    cnt = np.where(dense, rng.integers(120, 131, m ** 3), rng.integers(0, 4, m ** 3))
    at = np.repeat(ijk, cnt, 0)
    n = len(at)
    spec = synth.lj_fluid(n=8, rho=8.0, seed=1, nsteps=10, dmin=0.1)
    spec.pos = ((at + 0.005 + 0.99 * rng.random((n, 3))) * w - 0.5 * m * w)[rng.permutation(n)]
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
