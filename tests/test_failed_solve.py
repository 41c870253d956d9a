"""A solve that ends at its iteration cap: an error, the caller's labels left
alone, and a handle that solves the same graph once it may work enough."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

import gcfg  # noqa: E402
import oracle as O  # noqa: E402
from gpu_util import dev  # noqa: E402


@pytest.mark.parametrize("pinned", [False, True])
def test_labels_left_alone(pinned):
    """One row of pixels, source and sink 2000 apart: with one sweep per visit
    and one push round per relabel flow moves at most four pixels in an
    iteration (two in the first three), some 260 in the 66 that there are."""
    H, W = 3, 2040
    dp, dn = np.zeros((H, W), np.int32), np.zeros((H, W), np.int32)
    dp[1, 10], dn[1, 2010] = 50, 40
    gw = gcfg.GC_Init(W, H, dev(dp), dev(dn), 30)
    label = torch.full((H, W), 77, dtype=torch.int32)
    label = (label.pin_memory() if pinned else label).numpy()
    gcfg.GC_SetSchedule(gw, 1, 1)
    with pytest.raises(gcfg.GcfgError) as err:
        gcfg.GC_Optimize(gw, label)
    assert "iteration cap" in str(err.value)
    assert (label == 77).all()
    gcfg.GC_SetSchedule(gw, 2, 64)
    gcfg.GC_SetGraph(gw)
    res = gcfg.GC_Optimize(gw, label)
    gcfg.GC_End(gw)
    o = O.solve(dp, dn, penalty=30)
    assert res["flow"] == o["flow"] == 30
    assert np.array_equal(label, o["smax"].astype(np.int32))
