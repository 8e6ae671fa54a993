"""Source invariants of the kernels that raise a step's skip flag (CPU only).

A list build raises the flag when a slot outgrows the storage, while other
blocks of the same launch may only be starting.  Threads of such a block that
read the flag one by one can disagree, and a warp that left would be missing
from the work its block shares through shared memory.  So a block of a list
build reads the flag together.

The kernels that take the pairs at the cutoff raise it when there are more of
them than their buffer holds.  Every thread that reads the count must then
leave by the same branch, whatever the flag says: the count is not cleared in
the launch, and the branch holds no barrier."""
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
with open(os.path.join(ROOT, "ibisco_b200", "csrc", "ibg_kernels.cuh")) as f:
    SOURCE = re.sub(r"//[^\n]*", "", f.read())


def body(name: str) -> str:
    m = re.search(r"\b%s\([^;{]*\{\n(.*?)\n\}\n" % name, SOURCE, re.S)
    assert m, f"{name} not found"
    return m.group(1)


@pytest.mark.parametrize("kernel", ["k_list_build_warp", "k_list_build_thread", "k_list_build_slices"])
def test_a_list_build_block_reads_the_flag_together(kernel):
    b = body(kernel)
    assert "sc->skip = 1" in b  # it raises the flag
    assert "__syncthreads_or(sc->skip ||" in body("build_idle")
    assert b.count("if (build_idle(sc, always)) return;") == 1
    assert not re.search(r"sc->skip(?! = 1)", b)  # and reads it nowhere else


@pytest.mark.parametrize("kernel", ["k_nb_near", "k_nb_collect"])
def test_an_overflow_of_the_cutoff_pairs_leaves_without_a_barrier(kernel):
    assert "sc->skip = 1" in body("near_overflow")
    assert "near_n" not in body("near_overflow")
    branches = re.findall(r"if \(\w+ > \(unsigned\)A\.near_cap\) \{(.*?)\n\s*\}\n", body(kernel), re.S)
    assert len(branches) == 1
    assert "near_overflow(" in branches[0] and branches[0].rstrip().endswith("return;")
    assert "__sync" not in branches[0]
