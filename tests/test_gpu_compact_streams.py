"""Compactions of one context on several streams at once, and captured ones
replayed between others: every call's counts are its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


class Bitmap:
    def __init__(self, n, seed, share):
        rng = np.random.default_rng(seed)
        self.n = n
        self.rows = np.unique(rng.integers(0, n, int(n * share)))
        words = np.zeros((n + 31) // 32, np.uint32)
        np.bitwise_or.at(words, self.rows >> 5, np.uint32(0x80000000) >> (self.rows & 31).astype(np.uint32))
        self.bm = torch.from_numpy(words.view(np.int32)).cuda()
        self.out = torch.zeros(len(self.rows) + 8, dtype=torch.int32, device="cuda")
        self.cnt = torch.zeros(1, dtype=torch.int64, device="cuda")

    def clear(self):
        self.out.fill_(-1)
        self.cnt.fill_(-1)

    def run(self, ctx, stream):
        ctx.bitmap_rows_async(self.bm.data_ptr(), self.n, self.out.data_ptr(), self.out.numel(), self.cnt.data_ptr(),
                              stream.cuda_stream)

    def check(self):
        assert int(self.cnt.item()) == len(self.rows)
        got = self.out.cpu().numpy().view(np.uint32)
        assert np.array_equal(got[:len(self.rows)], self.rows.astype(np.uint32))
        assert (got[len(self.rows):] == 0xFFFFFFFF).all()


@pytest.fixture
def own_ctx():
    import rtscan_b200 as R
    c = R.Context(0)
    yield c
    c.close()


def test_compactions_on_many_streams(own_ctx):
    maps = [Bitmap(n, i, share) for i, (n, share) in
            enumerate([(200_000, 0.5), (90_000_000, 0.02), (170_000_000, 0.005), (33, 0.3), (60_000_000, 0.05)])]
    streams = [torch.cuda.Stream() for _ in maps]
    for _ in range(4):
        for m in maps:
            m.clear()
        torch.cuda.synchronize()
        for m, s in zip(maps, streams):
            m.run(own_ctx, s)
        torch.cuda.synchronize()
        for m in maps:
            m.check()


def test_captured_compactions(own_ctx):
    """Two graphs and plain calls (one of which grows the context's buffer)
    side by side."""
    maps = [Bitmap(3_000_000, 1, 0.1), Bitmap(40_000_000, 2, 0.02), Bitmap(150_000_000, 3, 0.005)]
    streams = [torch.cuda.Stream() for _ in maps]
    graphs = []
    for m in maps[:2]:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            m.run(own_ctx, torch.cuda.current_stream())
        graphs.append(g)
    for _ in range(3):
        for m in maps:
            m.clear()
        torch.cuda.synchronize()
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        maps[2].run(own_ctx, streams[2])
        torch.cuda.synchronize()
        for m in maps:
            m.check()
    del graphs
