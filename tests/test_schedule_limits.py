"""Schedule settings accept any count from 1 up: very large ones, which a
caller passes for "until nothing is left", solve as any other does."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

import gcfg  # noqa: E402
import oracle as O  # noqa: E402
from gpu_util import dev, gpu_solve  # noqa: E402

INT_MAX = (1 << 31) - 1


def _terms(H, W, seed):
    """Random terms under a strong penalty: a graph of some ten relabels."""
    rng = np.random.default_rng(seed)
    dp, dn = (rng.integers(0, 220, (H, W)).astype(np.int32) for _ in range(2))
    dp[:H // 3] += 120
    dn[-H // 3:] += 150
    return dp, dn


@pytest.mark.parametrize("schedule", [(2, INT_MAX), (1, 1 << 30), (2, 1 << 16)])
def test_sweeps_per_visit(schedule):
    dp, dn = _terms(150, 160, 1)
    o = O.solve(dp, dn, penalty=300)
    label, smin, smax, res = gpu_solve(dp, dn, penalty=300, schedule=schedule)
    assert res["global_relabels"] > 4  # past the iterations that keep the count as it was given
    assert res["flow"] == o["flow"]
    assert np.array_equal(smin, o["smin"]) and np.array_equal(smax, o["smax"])
    assert np.array_equal(label, o["smax"].astype(np.int32))


@pytest.mark.parametrize("rounds", [1, INT_MAX, 1 << 30])
def test_tile_rounds_per_relabel_8(rounds):
    dp, dn = _terms(60, 70, 2)
    o = O.solve8(dp, dn, penalty=100)
    gw = gcfg.GC_Init8(70, 60, dev(dp), dev(dn), 100)
    gcfg.GC_SetSchedule8(gw, rounds, 0)
    label = np.zeros((60, 70), np.int32)
    res = gcfg.GC_Optimize8(gw, label)
    gcfg.GC_End8(gw)
    assert res["flow"] == o["flow"]
    assert np.array_equal(label, o["smax"].astype(np.int32))
    assert res["push_rounds"] <= 3 * min(rounds, 1 << 12) * res["global_relabels"]
