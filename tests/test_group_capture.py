"""Where a run captures its graphs of ten steps (CPU only: the source's order).

Capturing and instantiating one takes as long as ten to forty of its replays
save.  It must not stand between two steps of a run: it belongs after the run's
read-back is queued and before the host waits for it, while the device works."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_groups_are_captured_while_the_device_works():
    with open(os.path.join(ROOT, "ibisco_b200", "csrc", "ibg_device.cu")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    m = re.search(r"static int run_steps\(.*?\n\}\n", src, re.S)
    run = m.group(0)
    groups = [x.start() for x in re.finditer(r"capture\(c, &\w+->second\.launches|capture\(c, &ch\.launches", run)]
    assert len(groups) == 1  # one place
    queued = run.index("cudaMemcpyAsync(c->hsc")
    waits = run.index("cudaStreamSynchronize", queued)
    assert queued < groups[0] < waits
    assert "cudaEventQuery(c->run_ev[1])" in run[queued:groups[0]]
