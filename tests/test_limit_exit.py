"""A tile's BFS that ends at the height limit with its last levels: they reach
the tile's border columns, whose heights the neighbour tile pushes by."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]


@pytest.mark.parametrize("dist", [*range(4, 14), *range(33, 42)])
@pytest.mark.parametrize("right", [False, True])
def test_border_heights_at_the_limit(dist, right):
    """Sinks `dist` columns inside one tile, excess next to it in the
    neighbour tile (32 tile rows, so that many warps run this at once)."""
    import oracle as O
    from gpu_util import gpu_solve

    H, W = 32 * 32, 32 * 4
    dp, dn = np.zeros((H, W), np.int32), np.zeros((H, W), np.int32)
    rng = np.random.default_rng(dist)
    src, sink = (63, 63 + dist) if not right else (64, 64 - dist)  # columns beside the border of tiles 1 and 2
    dp[:, src] = rng.integers(1, 50, H)
    dn[:, sink] = rng.integers(1, 50, H)
    kw = {k: (rng.integers(0, 30, (H, W)) * (rng.random((H, W)) < 0.9)).astype(np.int32)
          for k in ("up", "down", "left", "right")}
    o = O.solve(dp, dn, **kw)
    for _ in range(3):
        label, smin, smax, res = gpu_solve(dp, dn, **kw)
        assert res["flow"] == o["flow"]
        assert np.array_equal(smin, o["smin"]) and np.array_equal(smax, o["smax"])
        assert np.array_equal(label, o["smax"].astype(np.int32))
