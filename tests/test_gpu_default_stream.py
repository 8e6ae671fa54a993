"""A context's results do not depend on what runs on the default stream.

A context works on non-blocking streams, which the default stream does not
order.  Its state, flags and buffers must therefore be set on its own stream
(or waited for), not by small copies or memsets on the default stream that are
still on their way when the first kernels run.  Here the default stream is
kept busy (a bounded spin of about 20 ms) while a state is set, the list
storage grows in mid-run and the observable ring is allocated; the trajectory
must be the one of an idle device, bit for bit.
"""
import numpy as np
import pytest

from ibisco_b200 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [native.IBG_PREC_FP32_FIXED])
@pytest.mark.parametrize("system", ["melt", "hybrid"])
def test_busy_default_stream_changes_nothing(sysdir, system, precision):
    torch = pytest.importorskip("torch")
    setup = native.Setup(sysdir(system))
    got = []
    for busy in (False, True):
        g = native.System(setup, precision)
        spin = (lambda: torch.cuda._sleep(40_000_000)) if busy else (lambda: None)
        torch.zeros(1, device="cuda")
        spin()
        g.set_state()
        spin()
        g.run(1, 9)
        native.lib().ibg_set_list_rows(g._h, 1)  # step 10 rebuilds the lists: the storage grows there
        spin()
        obs = g.run(10, 11, observe=True)
        got.append((g.state64(), obs))
        g.close()
    (a, oa), (b, ob) = got
    for k in a:
        assert np.array_equal(a[k], b[k]), k
    assert oa == ob
