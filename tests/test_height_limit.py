"""The solver's height limit: sinks nearer and farther than the limits of the
first outer iterations (9 and 36 steps), alone and beside near ones."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]


def _check(dp, dn, **kw):
    import oracle as O
    from gpu_util import gpu_solve

    label, smin, smax, res = gpu_solve(dp, dn, **kw)
    o = O.solve(dp, dn, **kw)
    assert res["flow"] == o["flow"]
    assert np.array_equal(smin, o["smin"]) and np.array_equal(smax, o["smax"])
    assert np.array_equal(label, o["smax"].astype(np.int32))


@pytest.mark.parametrize("dist", [1, 7, 8, 9, 10, 11, 12, 13, 31, 32, 33, 34, 35, 36, 37, 39, 40, 100, 200])
@pytest.mark.parametrize("near", [False, True])
def test_sink_at_distance(dist, near):
    """A source column and a sink column `dist` apart; `near`: also a corner
    of random terms, so that the limited iterations have work."""
    H, W = 45, dist + 75
    dp, dn = np.zeros((H, W), np.int32), np.zeros((H, W), np.int32)
    dp[:, 5] = 40
    dn[:, 5 + dist] = 37
    if near:
        rng = np.random.default_rng(dist)
        dp[:, -50:-5] = rng.integers(0, 90, (H, 45))
        dn[:, -50:-5] = rng.integers(0, 90, (H, 45))
    _check(dp, dn, penalty=23)


@pytest.mark.parametrize("seed", range(4))
def test_far_sinks_behind_weak_edges(seed):
    """Random capacities (some zero) with few sinks: distances of all sizes."""
    rng = np.random.default_rng(seed)
    H, W = 150, 170
    dp = np.where(rng.random((H, W)) < 0.3, rng.integers(1, 60, (H, W)), 0).astype(np.int32)
    dn = np.where(rng.random((H, W)) < 0.004, rng.integers(1, 900, (H, W)), 0).astype(np.int32)
    kw = {k: (rng.integers(0, 25, (H, W)) * (rng.random((H, W)) < 0.85)).astype(np.int32)
          for k in ("up", "down", "left", "right")}
    _check(dp, dn, **kw)


@pytest.mark.parametrize("seed", range(3))
def test_easy_and_hard_images_in_one_solve(seed):
    """Images that end at their first termination check beside images that
    need several: each image's check is its own."""
    import gcfg
    import oracle as O
    from gpu_util import dev

    rng = np.random.default_rng(seed)
    ims = [(int(rng.integers(20, 200)), int(rng.integers(20, 200)), lam)
           for lam in (1.0, 20000.0, 50.0, 2000.0, 10.0, 100000.0, 200.0, 5000.0)]
    data = [O.generate(3, w, h, seed * 100 + i) for i, (w, h, _) in enumerate(ims)]
    rgb, scrib = (dev(np.concatenate([d[k].reshape(-1) for d in data])) for k in (0, 1))
    smin, smax = torch.zeros_like(scrib), torch.zeros_like(scrib)
    bs = gcfg.BatchSolver(len(ims), scrib.numel())
    flows, _ = bs.run([w for w, _, _ in ims], [h for _, h, _ in ims], [lam for *_, lam in ims], rgb, scrib, smin, smax)
    bs.close()
    a, b, off = smin.cpu().numpy(), smax.cpu().numpy(), 0
    for (w, h, lam), (im, sc), flow in zip(ims, data, flows):
        o = O.segment(im, sc, lam)
        assert flow == o["flow"]
        assert np.array_equal(a[off:off + w * h].reshape(h, w), o["smin"])
        assert np.array_equal(b[off:off + w * h].reshape(h, w), o["smax"])
        off += w * h
