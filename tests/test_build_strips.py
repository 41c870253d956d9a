"""The image -> graph build at the edges of its strips and kinds of tile:
sizes with no, one and many tiles inside the image border, on both sides of
the tile count where the strips change, odd byte addresses, weights beyond the
fast rounding's range and a constant image."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

SIZES = [(3, 3), (32, 33), (33, 65), (65, 65), (66, 66), (67, 98), (97, 66), (98, 99), (130, 34), (71, 300),
         (1024, 1024), (1025, 1056)]


# (a large image with so large a lambda runs into the solver's iteration cap)
@pytest.mark.parametrize("w,h,lam", [(w, h, lam) for w, h in SIZES for lam in (30.0, 5.0e6, "constant")
                                     if lam != 5.0e6 or w * h < 100000])
def test_image_graph_against_array_graph(w, h, lam):
    """The same graph built from the image and from the t-link and n-link
    arrays that the stand-alone calls write (checked against the oracle in
    the small sizes) has the same flow, energy and cuts."""
    import gcfg
    import oracle as O
    from gpu_util import dev, gpu_solve

    rgb, scrib = O.generate(3, w, h, w + h)
    if lam == "constant":
        rgb, lam = np.full_like(rgb, 90), 25.0
    off = (w + h) % 4
    pad = torch.zeros(3 * w * h + 4, dtype=torch.uint8, device="cuda")
    pad[off:off + 3 * w * h] = dev(rgb.reshape(-1))
    d_rgb, d_scrib = pad[off:off + 3 * w * h], dev(scrib)
    smin, smax = [torch.zeros((h, w), dtype=torch.uint8, device="cuda") for _ in range(2)]
    res = gcfg.Segmenter(w, h).run(d_rgb, d_scrib, w, h, lam, smin, smax)

    dp, dn, up, down, left, right = [torch.zeros((h, w), dtype=torch.int32, device="cuda") for _ in range(6)]
    gcfg.tlinks(d_rgb, d_scrib, dp, dn)
    gcfg.nlinks(d_rgb, w, h, lam, up, down, left, right)
    a = [t.cpu().numpy() for t in (dp, dn, up, down, left, right)]
    _, amin, amax, ares = gpu_solve(a[0], a[1], 0, *a[2:])
    assert res["flow"] == ares["flow"] and res["ref_energy"] == ares["ref_energy"]
    assert np.array_equal(smin.cpu().numpy(), amin) and np.array_equal(smax.cpu().numpy(), amax)
    if w * h < 100000:
        ref = O.segment(rgb, scrib, lam)
        assert res["flow"] == ref["flow"]
        assert np.array_equal(amin, ref["smin"]) and np.array_equal(amax, ref["smax"])
