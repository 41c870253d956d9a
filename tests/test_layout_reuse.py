"""Handles that are used for batches of other sizes in between: captured
graphs, the layout kept on the device and the tables behind it follow."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

import gcfg  # noqa: E402
import oracle as O  # noqa: E402


class _Batch:
    def __init__(self, sizes, seed, lam=50.0):
        data = [O.generate(3, w, h, seed + i) for i, (w, h) in enumerate(sizes)]
        self.W, self.H = [w for w, _ in sizes], [h for _, h in sizes]
        self.lam = [lam] * len(sizes)
        self.rgb, self.scrib = (np.concatenate([d[k].reshape(-1) for d in data]) for k in (0, 1))
        self.dev = [torch.from_numpy(a).cuda() for a in (self.rgb, self.scrib)]
        self.out = [torch.zeros(self.scrib.size, dtype=torch.uint8, device="cuda") for _ in range(2)]
        cuts = [O.segment(im, sc, lam) for im, sc in data]
        self.flows = [c["flow"] for c in cuts]
        self.cuts = [np.concatenate([c[k].reshape(-1) for c in cuts]) for k in ("smin", "smax")]

    def check(self, flows, cuts):
        assert list(flows) == self.flows
        for a, b in zip(cuts, self.cuts):
            assert np.array_equal(a, b)

    def run(self, bs):
        for o in self.out:
            o.fill_(7)
        flows, _ = bs.run(self.W, self.H, self.lam, *self.dev, *self.out)
        self.check(flows, [o.cpu().numpy() for o in self.out])


def _few_and_many():
    """A few images, and many small ones with more tiles, chunks and images
    than a handle made for the few has room for (1 pixel past a tile each way)."""
    return _Batch([(150, 90), (65, 200), (33, 40)], 7000), _Batch([(33, 33)] * 60, 7100)


def test_captured_graph_after_the_buffers_grew():
    few, many = _few_and_many()
    bs = gcfg.BatchSolver(len(few.W), few.scrib.size)
    bs.set_graph(True)
    few.run(bs)
    few.run(bs)
    assert bs.graph_info()["captures"] == 1 and bs.graph_info()["replays"] == 2
    many.run(bs)
    few.run(bs)  # every array has moved: the first graph must not be replayed
    assert bs.graph_info()["captures"] == 3
    for b in (many, few, many, few):
        b.run(bs)
    assert bs.graph_info()["captures"] == 3
    bs.close()


def test_the_same_layout_after_another_one():
    few, many = _few_and_many()
    other = _Batch([(150, 90), (65, 200), (33, 40)], 7200)  # the sizes of `few`, other images
    weak = _Batch([(150, 90), (65, 200), (33, 40)], 7000, lam=3.0)  # and other lambdas
    bs = gcfg.BatchSolver(64, max(few.scrib.size, many.scrib.size))
    for b in (few, few, other, many, few, weak, weak, other, many, many, few):
        b.run(bs)
    bs.close()


def test_stream_changed_between_runs_of_one_layout():
    few, _ = _few_and_many()
    other = _Batch([(150, 90), (65, 200), (33, 40)], 7200)
    bs = gcfg.BatchSolver(len(few.W), few.scrib.size)
    torch.cuda.synchronize()
    for stream in (None, torch.cuda.Stream(), torch.cuda.Stream(), None):
        if stream is not None:
            stream.wait_stream(torch.cuda.current_stream())
        bs.set_stream(stream if stream is not None else torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            other.run(bs)
            few.run(bs)
    bs.close()


@pytest.mark.parametrize("graph", [False, True])
def test_growth_while_a_batch_is_in_flight(graph):
    """The second set of host tables and staging buffers is made, and every
    device array moves, while the first batch is on its way."""
    few, many = _few_and_many()
    big = _Batch([(400, 300), (90, 500)], 7300)
    bs = gcfg.BatchSolver(len(few.W), few.scrib.size)
    bs.set_graph(graph)
    pinned = {id(b): [torch.from_numpy(a).pin_memory().numpy() for a in (b.rgb, b.scrib)] for b in (few, many, big)}

    def submit(b):
        out = [torch.full((b.scrib.size,), 7, dtype=torch.uint8).pin_memory().numpy() for _ in range(2)]
        return b, out, bs.submit_host(b.W, b.H, b.lam, *pinned[id(b)], *out)

    def collect(flight):
        b, out, ticket = flight
        b.check(bs.wait(ticket)[0], out)

    flight = submit(few)
    for b in (many, big, few, few, many, few, big, big):
        nxt = submit(b)
        collect(flight)
        flight = nxt
    collect(flight)
    few.run(bs)
    bs.close()
