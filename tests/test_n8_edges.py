"""8-neighbour graphs at the edges of their tiles (32x32 relabel tiles, 32x8
push tiles), with sinks nearer and farther than the first iteration's height
limit, and paths that cross tiles by their corners."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]


def _check(dp, dn, penalty, arrs):
    import oracle as O
    from test_n8 import DIRS, _gpu8

    label, smin, smax, r = _gpu8(dp, dn, penalty, arrs)
    o = O.solve8(dp, dn, penalty=penalty, arrays=None if arrs is None else [arrs[k] for k in DIRS])
    assert r["flow"] == o["flow"]
    assert np.array_equal(smin, o["smin"]) and np.array_equal(smax, o["smax"])
    assert np.array_equal(label, o["smax"].astype(np.int32))


@pytest.mark.parametrize("w,h", [(3, 3), (7, 33), (31, 8), (32, 32), (33, 9), (34, 40), (64, 7), (65, 65), (66, 34), (130, 97)])
@pytest.mark.parametrize("arrays", [False, True])
def test_sizes(w, h, arrays):
    from test_n8 import DIRS

    rng = np.random.default_rng(w * 1000 + h)
    dp = rng.integers(0, 90, (h, w)).astype(np.int32)
    dn = rng.integers(0, 90, (h, w)).astype(np.int32)
    arrs = {k: (rng.integers(0, 30, (h, w)) * (rng.random((h, w)) < 0.8)).astype(np.int32) for k in DIRS}
    _check(dp, dn, 17, arrs if arrays else None)


@pytest.mark.parametrize("dist", [1, 7, 8, 9, 10, 11, 31, 32, 33, 36, 70])
@pytest.mark.parametrize("near", [False, True])
def test_sink_at_distance(dist, near):
    """Only diagonal edges lead from the source row to the sink row `dist`
    below; `near`: random terms beside them too."""
    from test_n8 import DIRS

    h, w = dist + 20, 150
    dp, dn = np.zeros((h, w), np.int32), np.zeros((h, w), np.int32)
    dp[5, 20:60] = 40
    dn[5 + dist, :] = 37
    rng = np.random.default_rng(dist)
    arrs = {k: np.zeros((h, w), np.int32) for k in DIRS}
    arrs["downright"][:] = 11
    arrs["downleft"][:] = rng.integers(0, 9, (h, w))
    if near:
        dp[:, 110:] = rng.integers(0, 90, (h, 40))
        dn[:, 110:] = rng.integers(0, 90, (h, 40))
        for k in DIRS:
            arrs[k][:, 110:] = rng.integers(0, 25, (h, 40))
    _check(dp, dn, 0, arrs)


@pytest.mark.parametrize("rounds", [1, 2, 8])
@pytest.mark.parametrize("w,h,penalty", [(70, 45, 60), (200, 150, 100)])
def test_many_relabels(w, h, penalty, rounds):
    """Sources on one side and sinks on the other: far flow, so that the solve
    goes past its third relabel."""
    import gcfg
    import oracle as O
    from gpu_util import dev

    rng = np.random.default_rng(w + rounds)
    dp = (rng.integers(0, 90, (h, w)) * (np.arange(w) < w // 3)).astype(np.int32)
    dn = (rng.integers(0, 90, (h, w)) * (np.arange(w) > w // 2)).astype(np.int32)
    gw = gcfg.GC_Init8(w, h, dev(dp), dev(dn), penalty)
    gcfg.GC_SetSchedule8(gw, rounds, 3)
    label = np.zeros((h, w), np.int32)
    r = gcfg.GC_Optimize8(gw, label)
    gcfg.GC_End8(gw)
    o = O.solve8(dp, dn, penalty=penalty, arrays=None)
    if rounds == 1:
        assert r["global_relabels"] > 3
    assert r["flow"] == o["flow"] and np.array_equal(label, o["smax"].astype(np.int32))
