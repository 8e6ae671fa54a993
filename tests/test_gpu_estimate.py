"""The memory estimate made before a context exists against what it then holds.

The serving loop admits jobs by the estimate.  Everything but the list storage
is known from the descriptor, so beside that storage the estimate may not fall
below what a context holds with its state set, and may exceed it by the 2 MB
added for small arrays, 64 kB per bonded table and a quarter (bonds are counted
from both ends, tables of a list by the longest one)."""
import numpy as np
import pytest

from ibisco_b200 import native, synth

pytestmark = pytest.mark.gpu


def long_tables():
    """1,500 beads of eight types: 36 tables of 24,001 rows on one grid."""
    spec = synth.lj_fluid(n=1500, rho=8.0, seed=3, nsteps=10, dmin=0.42)
    spec.types = [(f"T{t}", 0.072, "A") for t in range(1, 9)]
    spec.itype = 1 + np.arange(1500) % 8
    spec.nb_tabs = [((a, b), synth.lj_table(f"nb{a}_{b}", 0.45, 2.0, 1.2, 0.00005))
                    for a in range(1, 9) for b in range(a, 9)]
    return spec


SYSTEMS = {
    "tables": long_tables,
    "melt": lambda: synth.polymer_melt(nchains=400, nper=100, seed=2, nsteps=10),
    "cg": lambda: synth.cg_melt(nchains=800, nper=200, nsteps=10),
    "hybrid": lambda: synth.hybrid_melt(n_atomistic=60, n_cg=60, nmono=40, seed=13, nsteps=10),
}


@pytest.mark.parametrize("prec", [0, 1], ids=["fp32", "fp64"])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_estimate_covers_what_a_context_holds(tmp_path, name, prec):
    spec = SYSTEMS[name]()
    s = native.Setup(synth.write_system(spec, str(tmp_path / "x")))
    _, _, box = s.initial_state()
    est = native.lib().ibg_estimate_bytes(s.desc(), prec, native._fp(box))
    for key, rl in (("ATOM", "neighbour_list_cutoff"), ("BEAD", "bead_neighbour_list_cutoff")):
        n = len(s.array(key))
        half = n / float(np.prod(box.astype(np.float64))) * 2.0 / 3.0 * np.pi * spec.control[rl] ** 3
        est -= n * 32 * (np.ceil((half * 1.25 + 8) / 8) * 1.25 + 2)
    g = native.System(s, prec)
    g.set_state()
    g.forces(1)
    native.lib().ibg_set_list_rows(g._h, 1)
    held = native.lib().ibg_device_bytes(g._h)
    for key in ("ATOM", "BEAD"):
        held -= (len(s.array(key)) + 3) // 4 * 128
    bonded = sum(len(s.array(k)) for k in ("NDATB", "NDATAN", "NDATT", "NDATO"))
    print(f"{name} prec {prec}, lists apart: estimate {est / 1e6:.2f} MB, held {held / 1e6:.2f} MB")
    assert held <= est <= 1.25 * held + 2 * 2 ** 20 + 65536 * bonded
