"""Every kernel that may be launched programmatically opens with its wait (CPU
only): the ones whose launch takes a condition too, not only a literal true.
The same source invariant as in test_launch_invariants.py, over all launches."""
import re

import pytest

from test_launch_invariants import _body_opening, _read

HOST = re.sub(r"//[^\n]*", "", _read("ibg_device.cu"))


def programmatic():
    names = set(re.findall(r"launch_pdl\(c,\s*(k_\w+)", HOST))
    for condition, name in re.findall(r"launch_on\([\w>.\-]+,\s*([^,]+),\s*(k_\w+|nb_kernel)", HOST):
        if condition.strip() != "false":
            names.add(name)
    return sorted((names - {"nb_kernel"}) | {"k_nonbonded", "k_nonbonded_f32", "k_nonbonded_slices"})


def test_the_conditional_launches_are_among_them():
    assert {"k_positions", "k_move", "k_cell_assign", "k_finalize", "k_nb_collect"} <= set(programmatic())


@pytest.mark.parametrize("name", programmatic())
def test_a_programmatic_kernel_waits_first(name):
    opening = _body_opening(_read("ibg_kernels.cuh"), name)
    assert opening and opening[-1] == "pdl_wait();", opening
    assert all(line.startswith(("using ", "constexpr ")) for line in opening[:-1]), opening
