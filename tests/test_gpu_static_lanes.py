"""ibg_nonbonded_static at the sizes where its split of the work changes: a
single particle, lists shorter and longer than the lanes that share one, and
list counts on both sides of the rule that picks the lanes per particle.

The reference is the same sum over the same list in FP64.  A pair's REAL*4
force carries at most ~10 roundings of 6e-8 relative (difference, minimum
image, square root, division, interpolation); near the cutoff r/bin is ~600, so
the weight's share is up to 600 * 6e-8 of one table step.  1e-5 of the largest
force, the tolerance of the other tests of this entry point, covers both.
Two calls in a row have to agree bit for bit (the scratch is left clean), also
after a call that ended with an error.
"""
import ctypes

import numpy as np
import pytest

from ibisco_b200 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nneb", [(1, 0), (2, 1), (9, 8), (40, 33), (257, 64), (44999, 20), (45000, 20), (60011, 7)])
def test_static_lanes(n, nneb):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    box = np.float32(max(4.0, (n / 8.0) ** (1 / 3)))
    x = ((rng.random((n, 3)) - 0.5) * box).astype(np.float32)
    rc = np.float32(1.2)
    ld, bin_ = 612, np.float32(0.002)
    r = (np.arange(ld) * bin_).astype(np.float32)
    force = (5.0 * np.cos(3.0 * r)).astype(np.float32)
    pot = (2.0 * np.sin(2.0 * r)).astype(np.float32)
    maxnab = nneb + 3
    lst = np.zeros((n, maxnab), np.int32)
    for a in range(n):
        lst[a, :nneb] = 1 + (a + 1 + rng.permutation(max(n - 1, 1))[:nneb]) % n if n < 1000 else \
            1 + (a + 1 + np.arange(nneb)) % n
    nn = np.full(n, nneb, np.int32)
    i = np.repeat(np.arange(n), nneb)
    j = lst[:, :nneb].ravel().astype(np.int64) - 1
    d = x[i].astype(np.float64) - x[j]
    d -= float(box) * np.round(d / float(box))
    rr = np.sqrt((d * d).sum(1))
    ok = rr * rr < float(rc * rc)
    i, j, d, rr = i[ok], j[ok], d[ok], rr[ok]
    k = (rr / float(bin_)).astype(int)
    al = (rr - r[k]) / float(bin_)
    fij = force[k] * (1 - al) + force[k + 1].astype(np.float64) * al
    vij = pot[k] * (1 - al) + pot[k + 1].astype(np.float64) * al
    ref = np.zeros((n, 3))
    np.add.at(ref, i, fij[:, None] * d)
    np.add.at(ref, j, -fij[:, None] * d)

    def up(a, dt):
        return torch.from_numpy(np.ascontiguousarray(a, dt)).cuda()

    t = dict(x=up(x, np.float32), ty=up(np.ones(n), np.int32), lab=up(np.ones(n), np.int32),
             idx=up(np.arange(1, n + 1), np.int32), lst=up(lst, np.int32), nn=up(nn, np.int32), map=up([1], np.int32),
             r=up(r, np.float32), f=up(force, np.float32), v=up(pot, np.float32), b=up([bin_], np.float32),
             nd=up([ld - 3], np.int32))
    bad = up(np.full(n, 7), np.int32)  # a type outside 1..ntype
    err = ctypes.create_string_buffer(256)
    got = []
    for types in (t["ty"], bad, t["ty"]):
        fx = torch.full((n, 3), float("nan"), dtype=torch.float64, device="cuda")
        sums = torch.full((9,), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        p = lambda a: ctypes.c_void_p(a.data_ptr())  # noqa: E731
        rc_ = native.lib().ibg_nonbonded_static(
            n, n, p(t["x"]), p(types), p(t["lab"]), p(t["idx"]), p(t["lst"]), maxnab, p(t["nn"]), 1, p(t["map"]), 1,
            ld, p(t["r"]), p(t["f"]), p(t["v"]), p(t["b"]), p(t["nd"]),
            np.full(3, box, np.float32).ctypes.data_as(ctypes.c_void_p), ctypes.c_float(rc * rc), p(fx), p(sums), None,
            err, 256)
        if types is bad:
            assert rc_ == (native.STATUS_CODE["IBG_E_MISSING_TABLE"] if len(i) else 0)
            continue
        assert rc_ == 0, err.value
        got.append((fx.cpu().numpy(), sums.cpu().numpy()))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    scale = max(np.abs(ref).max(), 1e-30)
    assert np.abs(got[0][0] - ref).max() <= 1e-5 * scale
    assert abs(got[0][1][0] - vij.sum()) <= 1e-5 * max(np.abs(vij).sum(), 1e-30)
