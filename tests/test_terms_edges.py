"""t-links and n-links at the edges of their blocks: widths and heights around
the 32-pixel blocks, pixel counts around the chunk sizes, and scribbles that
are full, dense, sparse or in strips."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]


def _scrib(kind, h, w, rng):
    if kind == "full":
        return rng.integers(1, 3, (h, w)).astype(np.uint8)
    if kind == "dense":
        return rng.integers(0, 3, (h, w)).astype(np.uint8)
    if kind == "sparse":
        return ((rng.random((h, w)) < 0.02) * rng.integers(1, 3, (h, w))).astype(np.uint8)
    s = np.zeros((h, w), np.uint8)
    s[: min(10, h)] = 2
    s[:, max(0, w - 7):] = 1
    s[h // 2, ::3] = 3  # not a class: counts for neither
    return s


@pytest.mark.parametrize("w,h", [(1, 1), (2, 1), (1, 33), (31, 4), (32, 32), (33, 31), (64, 16), (1023, 1), (41, 25),
                                 (2049, 1), (4097, 2), (511, 513), (515, 1031), (2100, 2001)])
@pytest.mark.parametrize("kind", ["full", "dense", "sparse", "strips"])
def test_terms(w, h, kind):
    import gcfg
    import oracle as O
    from gpu_util import dev

    rng = np.random.default_rng(w * 7 + h)
    rgb = rng.integers(0, 256, (h, w, 3)).astype(np.uint8)
    scrib = _scrib(kind, h, w, rng)
    dp, dn, *links = [torch.full((h, w), -7, dtype=torch.int32, device="cuda") for _ in range(6)]
    off = 1 + (w + h) % 3  # odd addresses of the image and the scribbles
    pad = torch.zeros(3 * w * h + 8, dtype=torch.uint8, device="cuda")
    pad[off:off + 3 * w * h] = dev(rgb.reshape(-1))
    spad = torch.zeros(w * h + 8, dtype=torch.uint8, device="cuda")
    spad[off:off + w * h] = dev(scrib.reshape(-1))
    d_rgb, d_scrib = pad[off:off + 3 * w * h], spad[off:off + w * h]
    gcfg.tlinks(d_rgb, d_scrib, dp, dn)
    odp, odn = O.tlinks(rgb, scrib)
    assert np.array_equal(dp.cpu().numpy(), odp) and np.array_equal(dn.cpu().numpy(), odn)
    gcfg.nlinks(d_rgb, w, h, 50.0, *links)
    for got, want in zip(links, O.nlinks(rgb, 50.0)):
        assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("w,h", [(64, 64), (511, 513), (515, 1031), (2100, 2001)])
def test_segment_in_each_chunk_size(w, h):
    import oracle as O
    from gpu_util import gpu_segment

    rgb, scrib = O.generate(3, w, h, w)
    smin, smax, res = gpu_segment(rgb, scrib, 50.0)
    ref = O.segment(rgb, scrib, 50.0)
    assert res["flow"] == ref["flow"]
    assert np.array_equal(smin, ref["smin"]) and np.array_equal(smax, ref["smax"])


def test_terms_in_the_largest_chunks():
    """More than 2^24 pixels."""
    test_terms(4111, 4099, "sparse")


@pytest.mark.parametrize("n", [1, 7, 97, 1000, 4099, 70001, 999983])
def test_tlinks_near_rounding_ties(n):
    """Tables of images of one colour and of two: their entries 10 ln(N / k)
    take all places between two integers."""
    import gcfg
    import oracle as O
    from gpu_util import dev

    rgb = np.full((n, 1, 3), 40, np.uint8)
    rgb[: n // 3] = 200
    scrib = np.full((n, 1), 1, np.uint8)
    scrib[::2] = 2
    dp, dn = [torch.zeros((n, 1), dtype=torch.int32, device="cuda") for _ in range(2)]
    gcfg.tlinks(dev(rgb), dev(scrib), dp, dn)
    odp, odn = O.tlinks(rgb, scrib)
    assert np.array_equal(dp.cpu().numpy(), odp) and np.array_equal(dn.cpu().numpy(), odn)
