"""Handles that change streams while earlier work is still queued elsewhere."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

import gcfg  # noqa: E402
import oracle as O  # noqa: E402
from gpu_util import dev  # noqa: E402


def test_graph_made_behind_other_work_then_moved():
    """A handle made without terms while the default stream is busy (some 50 ms),
    then used on a stream of its own, which does not wait for the default one."""
    rng = np.random.default_rng(5)
    H, W = 90, 130
    dp, dn = (rng.integers(0, 90, (H, W)).astype(np.int32) for _ in range(2))
    o = O.solve(dp, dn, penalty=15)
    d = dev(dp), dev(dn)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        torch.cuda._sleep(100_000_000)
        gw = gcfg.GC_Init(W, H, None, None, 15)
        gcfg.GC_SetStream(gw, side)
        gcfg.GC_SetDataterms(gw, *d)
        gcfg.GC_SetGraph(gw)
        label = np.zeros((H, W), np.int32)
        res = gcfg.GC_Optimize(gw, label)
        gcfg.GC_End(gw)
        assert res["flow"] == o["flow"]
        assert np.array_equal(label, o["smax"].astype(np.int32))
