"""Where a run captures its graphs of ten steps (CPU only: the source's order).

Capturing and instantiating one takes as long as ten to forty of its replays
save.  So it belongs where the device has work meanwhile: behind enough queued
steps of the run, or between the run's queued read-back and the host's wait."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_groups_are_captured_while_the_device_works():
    with open(os.path.join(ROOT, "ibisco_b200", "csrc", "ibg_device.cu")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    m = re.search(r"static int run_steps\(.*?\n\}\n", src, re.S)
    run = m.group(0)
    assert run.count("capture(c, &") == 2  # a group's, in take, and a step's
    takes = [m.start() for m in re.finditer(r"\btake\(", run)]
    assert len(takes) == 2
    assert run[:takes[0]].endswith("if (!it->second.exec && k - begin >= kAhead) ")
    queued = run.index("cudaMemcpyAsync(c->hsc")
    waits = run.index("cudaStreamSynchronize", queued)
    assert queued < takes[1] < waits
    assert "cudaEventQuery(c->run_ev[1])" in run[queued:takes[1]]
