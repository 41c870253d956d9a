"""The workloads this library is measured on, through its public entry points.

A case is one call (or the short sequence of calls) that a program using the
library makes: an image cut out of device memory, an image cut from host
memory, a batch of uneven images, a stream of host batches, the graph API of
the reference with either neighbourhood, the data term by itself, and a
server's burst of new images and scribble edits.  Inputs are made on the GPU
from the seed alone, with the statistics of the configured synthetic families:
noisy coloured ellipses (foreground N((200, 60, 60)), background
N((60, 120, 200))), or small discs on a striped background, a 20x20
foreground scribble at the centre and a 10-pixel background border strip.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "gc-fg_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import gcfg  # noqa: E402

FG = (200.0, 60.0, 60.0)
BG = (60.0, 120.0, 200.0)
NBINS = 4096


def listed():
    return [
        # interactive cut of a thumbnail: latency of one small solve
        dict(name="seg_256", kind="seg", image="ellipse", w=256, h=256, lam=50.0),
        # a video frame / photo, the ordinary single-image call
        dict(name="seg_1080", kind="seg", image="multi", w=1920, h=1080, lam=50.0),
        # odd size, strong smoothing: several global relabels
        dict(name="seg_odd", kind="seg", image="multi", w=1237, h=823, lam=200.0),
        # the largest single image: thousands of small objects
        dict(name="seg_4096", kind="seg", image="blobs", w=4096, h=4096, lam=100.0),
        # a photo that starts and ends in host memory
        dict(name="seg_host", kind="seg_host", image="multi", w=2048, h=1536, lam=10.0),
        # the main workload: many uneven images in one solve
        dict(name="batch_256", kind="batch", n=256, lo=64, hi=1024, shapes=1, lam=50.0),
        # two host batches in flight, as a data pipeline feeds them
        dict(name="batch_stream", kind="stream", n=48, lo=64, hi=1024, shapes=2, lam=50.0),
        # the reference's graph API, handle kept, new terms for each frame
        dict(name="graph_loop", kind="graph", w=1024, h=768, penalty=20, arrays=False, keep=True),
        # the reference's applications: init, optimise, end, per-direction arrays
        dict(name="graph_once", kind="graph", w=641, h=479, penalty=0, arrays=True, keep=False),
        # the reference built with the 8-neighbourhood
        dict(name="graph8", kind="graph8", w=640, h=480, penalty=600, arrays=False),
        # the data term alone: t-links and n-links for a caller's own solver
        dict(name="terms", kind="terms", image="multi", w=1279, h=853, lam=50.0),
        # a server's burst: new images of mixed sizes, then edits of each
        dict(name="serve", kind="serve", sides="256,256,256,256,256,256,1024,1024,1024,2048", edits=8, lam=50.0),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """Width and height: side log-uniform in [lo, hi], aspect in [0.5, 2]."""
    s = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a = rng.uniform(0.5, 2.0)
    return max(40, int(round(s * math.sqrt(a)))), max(40, int(round(s / math.sqrt(a))))


def draw(rng):
    kind = rng.choice(["seg", "seg", "seg", "seg_host", "batch", "stream", "graph", "graph8", "terms", "serve"])
    lam = rng.choice([10.0, 50.0, 100.0, 200.0])
    if kind in ("seg", "seg_host"):
        image = rng.choice(["ellipse", "multi", "blobs"])
        w, h = _size(rng, 64, 2800 if image != "blobs" else 3600)
        return dict(kind=kind, image=image, w=w, h=h, lam=lam)
    if kind == "batch":
        return dict(kind=kind, n=_logint(rng, 2, 200), lo=rng.choice([48, 64, 100]), hi=rng.choice([256, 700, 1024]),
                    shapes=rng.randrange(1 << 20), lam=50.0)
    if kind == "stream":
        return dict(kind=kind, n=_logint(rng, 2, 48), lo=64, hi=rng.choice([300, 1024]),
                    shapes=rng.randrange(1 << 20), lam=50.0)
    if kind == "graph":
        w, h = _size(rng, 64, 1500)
        return dict(kind=kind, w=w, h=h, penalty=rng.choice([5, 20, 60]), arrays=rng.random() < 0.5,
                    keep=rng.random() < 0.5)
    if kind == "graph8":
        w, h = _size(rng, 64, 1100)
        return dict(kind=kind, w=w, h=h, penalty=rng.choice([20, 100, 600]), arrays=rng.random() < 0.5)
    if kind == "terms":
        w, h = _size(rng, 64, 3000)
        return dict(kind=kind, image=rng.choice(["ellipse", "multi"]), w=w, h=h, lam=lam)
    n = rng.randint(3, 10)
    sides = ",".join(str(rng.choice([256, 256, 256, 333, 1024, 1000])) for _ in range(n))
    return dict(kind="serve", sides=sides, edits=rng.randint(1, 8), lam=lam)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _scribbles(w, h):
    s = torch.zeros((h, w), dtype=torch.uint8, device="cuda")
    s[:10] = 2
    s[max(0, h - 10):] = 2
    s[:, :10] = 2
    s[:, max(0, w - 10):] = 2
    y0, x0 = max(0, h // 2 - 10), max(0, w // 2 - 10)
    s[y0:y0 + 20, x0:x0 + 20] = 1
    return s


def _image(kind, w, h, rng, gen):
    """(rgb uint8 [h, w, 3], scribbles uint8 [h, w]) on the GPU."""
    xs = torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
    ys = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
    sd_fg, sd_bg, stripe = 20.0, 25.0, None
    if kind == "blobs":
        n = max(4, int(2000 * (w * h) / 16777216.0))
        bx = torch.rand(n, generator=gen, device="cuda") * w
        by = torch.rand(n, generator=gen, device="cuda") * h
        r = 3.0 + 12.0 * torch.rand(n, generator=gen, device="cuda")
        bx[0], by[0], r[0] = w // 2, h // 2, 15.0
        off = torch.arange(-16, 17, device="cuda")
        px = (bx.floor().long()[:, None, None] + off[None, None, :]).expand(n, 33, 33)
        py = (by.floor().long()[:, None, None] + off[None, :, None]).expand(n, 33, 33)
        hit = (px - bx[:, None, None]) ** 2 + (py - by[:, None, None]) ** 2 <= (r * r)[:, None, None]
        hit &= (px >= 0) & (py >= 0) & (px < w) & (py < h)
        fg = torch.zeros(w * h, dtype=torch.bool, device="cuda")
        fg[(py * w + px)[hit]] = True
        fg = fg.view(h, w)
        sd_bg = 40.0
        stripe = 30.0 * torch.sin(xs * (2.0 * math.pi / 17.0))
    else:
        # one centred ellipse that scales with the image
        ax, ay = 80.0 * w / 256.0, 60.0 * h / 256.0
        if kind == "multi":
            ax, ay = 80.0 * max(1.0, w / 1920.0), 60.0 * max(1.0, h / 1080.0)
            sd_fg = sd_bg = 30.0
        fg = ((xs - w // 2) / ax) ** 2 + ((ys - h // 2) / ay) ** 2 <= 1.0
        if kind == "multi":
            s = min(1.0, min(w, h) / 1080.0)
            for _ in range(3):
                cx, cy = rng.uniform(0, w), rng.uniform(0, h)
                ea, eb = rng.uniform(40, 200) * s, rng.uniform(40, 200) * s
                fg |= ((xs - cx) / ea) ** 2 + ((ys - cy) / eb) ** 2 <= 1.0
    noise = torch.randn((h, w, 3), generator=gen, device="cuda")
    m = fg[..., None]
    mean = torch.where(m, torch.tensor(FG, device="cuda"), torch.tensor(BG, device="cuda"))
    if stripe is not None:
        mean = mean + torch.where(m, torch.zeros((), device="cuda"), stripe[..., None])
    noise *= torch.where(m, sd_fg, sd_bg)
    rgb = (mean + noise + 0.5).floor_().clamp_(0, 255).to(torch.uint8)
    return rgb, _scribbles(w, h)


def _gens(seed):
    return random.Random(seed), torch.Generator(device="cuda").manual_seed(seed)


def _shapes(case):
    rng = random.Random(case["shapes"])
    return [_size(rng, case["lo"], case["hi"]) for _ in range(case["n"])]


def _packed(case, seed):
    rng, gen = _gens(seed)
    sizes = _shapes(case)
    imgs = [_image("ellipse", w, h, rng, gen) for w, h in sizes]
    rgb = torch.cat([a.reshape(-1) for a, _ in imgs])
    scrib = torch.cat([b.reshape(-1) for _, b in imgs])
    return ([w for w, _ in sizes], [h for _, h in sizes], [case["lam"]] * len(sizes), rgb, scrib)


def _tlinks64(rgb, scrib):
    """Histogram t-links of an image (numpy, 64 bits): dp, dn int32."""
    c = rgb.reshape(-1, 3).astype(np.int64) >> 4
    bins = (c[:, 0] << 8) | (c[:, 1] << 4) | c[:, 2]
    s = scrib.reshape(-1)
    out = []
    for cls in (2, 1):  # dp from the background model, dn from the foreground's
        hist = np.bincount(bins[s == cls], minlength=NBINS)
        p = (hist + 1.0) / float(hist.sum() + NBINS)
        out.append(np.floor(10.0 * -np.log(p) + 0.5).astype(np.int32)[bins])
    return out


def _nlinks64(rgb, lam):
    """Contrast n-links (numpy, 64 bits): up, down, left, right int32 [h, w]."""
    a = rgb.astype(np.int64)
    dh = ((a[:, 1:] - a[:, :-1]) ** 2).sum(-1)
    dv = ((a[1:] - a[:-1]) ** 2).sum(-1)
    s2 = float(dh.sum() + dv.sum()) / (dh.size + dv.size)
    wh, wv = [np.floor(lam * np.exp(-d / (2.0 * s2)) + 0.5).astype(np.int32) if s2 > 0
              else np.full(d.shape, int(math.floor(lam + 0.5)), np.int32) for d in (dh, dv)]
    up, down, left, right = (np.zeros(rgb.shape[:2], np.int32) for _ in range(4))
    right[:, :-1] = wh
    left[:, 1:] = wh
    down[:-1] = wv
    up[1:] = wv
    return up, down, left, right


def _graph_inputs(case, seed, diag):
    """Device t-links (histogram model) and, if asked for, edge arrays."""
    rng, gen = _gens(seed)
    w, h = case["w"], case["h"]
    rgb, scrib = _image("multi", w, h, rng, gen)
    c = (rgb.view(-1, 3).long() >> 4)
    bins = (c[:, 0] << 8) | (c[:, 1] << 4) | c[:, 2]
    s = scrib.view(-1)
    dp, dn = [torch.floor(-10.0 * torch.log((torch.bincount(bins[s == k], minlength=NBINS) + 1).double()
                                            / float(int((s == k).sum()) + NBINS)) + 0.5).int()[bins].contiguous()
              for k in (2, 1)]
    edges = {}
    if case["arrays"]:
        a = rgb.int()

        def link(dy, dx):
            d = torch.full((h, w), 1 << 20, dtype=torch.int32, device="cuda")
            y0, y1 = max(0, -dy), h - max(0, dy)
            x0, x1 = max(0, -dx), w - max(0, dx)
            d[y0:y1, x0:x1] = ((a[y0:y1, x0:x1] - a[y0 + dy:y1 + dy, x0 + dx:x1 + dx]) ** 2).sum(-1)
            return (50.0 * torch.exp(d.double() / -5400.0) + 0.5).int().contiguous()

        edges = dict(up=link(-1, 0), down=link(1, 0), left=link(0, -1), right=link(0, 1))
        if diag:
            edges.update(upleft=link(-1, -1), upright=link(-1, 1), downleft=link(1, -1), downright=link(1, 1))
    return dp, dn, edges


def prepare(case, seed):
    k = case["kind"]
    st = dict(case=case)
    if k in ("seg", "seg_host"):
        w, h = case["w"], case["h"]
        rng, gen = _gens(seed)
        rgb, scrib = _image(case["image"], w, h, rng, gen)
        smin, smax = (torch.zeros((h, w), dtype=torch.uint8, device="cuda") for _ in range(2))
        if k == "seg_host":
            rgb, scrib, smin, smax = (t.cpu().pin_memory() for t in (rgb, scrib, smin, smax))
        st.update(rgb=rgb, scrib=scrib, smin=smin, smax=smax, seg=gcfg.Segmenter(w, h))
    elif k == "batch":
        ws, hs, lams, rgb, scrib = _packed(case, seed)
        st.update(ws=ws, hs=hs, lams=lams, rgb=rgb, scrib=scrib, smin=torch.zeros_like(scrib),
                  smax=torch.zeros_like(scrib), bs=gcfg.BatchSolver(len(ws), scrib.numel()))
    elif k == "stream":
        bufs = []
        for j in range(2):  # the second batch: other images of the same sizes
            ws, hs, lams, rgb, scrib = _packed(case, 2 * seed + j)
            bufs.append([t.cpu().pin_memory() for t in (rgb, scrib, torch.zeros_like(scrib), torch.zeros_like(scrib))])
        st.update(ws=ws, hs=hs, lams=lams, bufs=bufs, bs=gcfg.BatchSolver(len(ws), scrib.numel()))
    elif k == "graph":
        dp, dn, edges = _graph_inputs(case, seed, False)
        w, h = case["w"], case["h"]
        st.update(dp=dp, dn=dn, edges=edges, label=torch.zeros((h, w), dtype=torch.int32).pin_memory().numpy())
        if case["keep"]:
            st["gw"] = gcfg.GC_Init(w, h, None, None, case["penalty"])
    elif k == "graph8":
        dp, dn, edges = _graph_inputs(case, seed, True)
        w, h = case["w"], case["h"]
        st.update(dp=dp, dn=dn, edges=edges, label=torch.zeros((h, w), dtype=torch.int32).pin_memory().numpy(),
                  gw=gcfg.GC_Init8(w, h, dp, dn, case["penalty"], **edges),
                  smin=torch.zeros((h, w), dtype=torch.uint8, device="cuda"))
    elif k == "terms":
        w, h = case["w"], case["h"]
        rng, gen = _gens(seed)
        rgb, scrib = _image(case["image"], w, h, rng, gen)
        st.update(rgb=rgb, scrib=scrib,
                  out=[torch.zeros((h, w), dtype=torch.int32, device="cuda") for _ in range(6)])
    else:
        rng, gen = _gens(seed)
        sides = [int(x) for x in case["sides"].split(",")]
        # packed host label maps: both cuts after the first solves, both after the edits
        total = sum(s * s for s in sides)
        cuts = [torch.zeros(total, dtype=torch.uint8).pin_memory() for _ in range(4)]
        reqs, at = [], 0
        for s in sides:
            rgb, scrib = _image("multi", s, s, rng, gen)
            reqs.append([t.cpu().pin_memory() for t in (rgb, scrib)] + [c[at:at + s * s] for c in cuts])
            at += s * s
        edits = [dict(target=i, x=rng.randrange(sides[i] - 15), y=rng.randrange(sides[i] - 15), size=15,
                      cls=rng.choice([1, 2])) for i in range(min(case["edits"], len(sides)))]
        st.update(reqs=reqs, edits=edits, cuts=cuts, srv=gcfg.Server(
            mem_cap_bytes=1 << 30, lanes=2, max_batch_images=64, max_batch_tiles=1 << 14, max_sessions=64))
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(st):
    case = st["case"]
    k = case["kind"]
    if k in ("seg", "seg_host"):
        call = st["seg"].run if k == "seg" else st["seg"].run_host
        r = call(st["rgb"], st["scrib"], case["w"], case["h"], case["lam"], st["smin"], st["smax"])
        return dict(flow=r["flow"], energy=r["ref_energy"], smin=st["smin"], smax=st["smax"])
    if k == "batch":
        flows, _ = st["bs"].run(st["ws"], st["hs"], st["lams"], st["rgb"], st["scrib"], st["smin"], st["smax"])
        return dict(flows=flows, smin=st["smin"], smax=st["smax"])
    if k == "stream":
        bs = st["bs"]
        tk = [bs.submit_host(st["ws"], st["hs"], st["lams"], *b) for b in st["bufs"]]
        flows = [bs.wait(t)[0] for t in tk]
        return dict(flows=flows, cuts=[b[2:] for b in st["bufs"]])
    if k == "graph":
        if case["keep"]:
            gw = st["gw"]
            gcfg.GC_SetDataterms(gw, st["dp"], st["dn"])
            if case["arrays"]:
                gcfg.GC_SetEdges(gw, **st["edges"])
            gcfg.GC_SetGraph(gw)
        else:
            gw = gcfg.GC_Init(case["w"], case["h"], st["dp"], st["dn"], case["penalty"], **st["edges"])
        r = gcfg.GC_Optimize(gw, st["label"])
        if not case["keep"]:
            gcfg.GC_End(gw)
        return dict(flow=r["flow"], energy=r["ref_energy"], label=st["label"])
    if k == "graph8":
        gw = st["gw"]
        gcfg.GC_SetGraph8(gw)
        r = gcfg.GC_Optimize8(gw, st["label"])
        gcfg.GC_GetCuts8(gw, st["smin"], None)
        return dict(flow=r["flow"], energy=r["ref_energy"], label=st["label"], smin=st["smin"])
    if k == "terms":
        dp, dn, *links = st["out"]
        gcfg.tlinks(st["rgb"], st["scrib"], dp, dn)
        gcfg.nlinks(st["rgb"], case["w"], case["h"], case["lam"], *links)
        return dict(pos=dp, neg=dn, links=links)
    srv = st["srv"]
    news = [srv.submit_new(r[0], r[1], case["lam"], r[2], r[3]) for r in st["reqs"]]
    edits = [srv.submit_edit(news[e["target"]][1], e["x"], e["y"], e["size"], e["cls"], st["reqs"][e["target"]][4],
                             st["reqs"][e["target"]][5]) for e in st["edits"]]
    res = [srv.wait(t) for t, _ in news] + [srv.wait(t) for t, _ in edits]
    for _, sid in news:
        srv.release(sid)
    return dict(status=np.array([r["status"] for r in res]), flows=np.array([r["flow"] for r in res]),
                cuts=st["cuts"])


# ---------------------------------------------------------------------------
# what a pass cannot do without, and exact values
# ---------------------------------------------------------------------------

def work(case):
    """Each input read once and each output written once.  The operations
    counted are the ones every pixel needs whatever the solver: squared
    differences to two neighbours, two histogram or table look-ups, one
    comparison per cut; the flow computation itself depends on the image."""
    k = case["kind"]
    if k in ("seg", "seg_host"):
        px = case["w"] * case["h"]
        return dict(bytes=6 * px, flops=20 * px)
    if k in ("batch", "stream"):
        px = sum(w * h for w, h in _shapes(case)) * (2 if k == "stream" else 1)
        return dict(bytes=6 * px, flops=20 * px)
    if k in ("graph", "graph8"):
        px = case["w"] * case["h"]
        d = 8 if k == "graph8" else 4
        out = 5 if k == "graph8" else 4
        return dict(bytes=(8 + out + (4 * d if case["arrays"] else 0)) * px, flops=2 * d * px)
    if k == "terms":
        px = case["w"] * case["h"]
        return dict(bytes=(4 + 24) * px, flops=30 * px)
    sides = [int(x) for x in case["sides"].split(",")]
    px = sum(s * s for s in sides)
    edit = sum(s * s for s in sides[:case["edits"]])
    return dict(bytes=6 * px + 2 * edit, flops=20 * (px + edit))


def exact(case, seed):
    """t-links and n-links in 64 bits; the cuts and flows are integers that
    are compared for equality."""
    if case["kind"] != "terms":
        return None
    rng, gen = _gens(seed)
    rgb, scrib = (t.cpu().numpy() for t in _image(case["image"], case["w"], case["h"], rng, gen))
    dp, dn = _tlinks64(rgb, scrib)
    h, w = scrib.shape
    return dict(pos=dp.reshape(h, w), neg=dn.reshape(h, w), links=list(_nlinks64(rgb, case["lam"])))
