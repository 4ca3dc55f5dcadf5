"""Very wide rows beside many output channels, whose stages do not share one
ring of the direct kernel: batches and served bursts give every problem the
result that it has by itself."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

# n, c, h, w, k: neither of the first two fits a ring with the third, nor with one another
SHAPES = [(1, 64, 800, 800, 64), (2, 24, 9, 1080, 40), (8, 256, 14, 14, 256), (3, 16, 7, 7, 40), (1, 8, 5, 760, 300)]


def _tensors(shapes, seed):
    """Integers whose every product and sum is exact in fp32: the direct
    kernel's result is the rounded exact one, whatever the order."""
    g = torch.Generator().manual_seed(seed)
    out = []
    for n, c, h, w, k in shapes:
        x = torch.randint(-2, 3, (n, c, h, w), generator=g).half()
        f = torch.randint(-1, 2, (k, c, 3, 3), generator=g).half()
        out.append((x.cuda(), f.cuda(), torch.full((n, k, h, w), float("nan"), dtype=torch.float16, device="cuda")))
    return out


def _problem(wg, t, shape):
    return wg.make_problem(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), *shape)


def _by_name(wg, t, shape, algo):
    y = torch.zeros_like(t[2])
    op = wg.Conv2d(_problem(wg, (t[0], t[1], y), shape), wg.default_options(algo=algo))
    assert op.algo == algo
    op(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert op.check_device()[0] == wg.OK
    op.destroy()
    return y


def test_batch(wg):
    ts = _tensors(SHAPES, 5)
    want = [_by_name(wg, t, s, wg.ALGO_DIRECT) for t, s in zip(ts, SHAPES)]
    exact = torch.nn.functional.conv2d(ts[2][0].double(), ts[2][1].double(), padding=1).half()
    assert torch.equal(want[2], exact)
    b = wg.Batch([_problem(wg, t, s) for t, s in zip(ts, SHAPES)], wg.default_options(algo=wg.ALGO_DIRECT))
    assert 1 < b.launches(True) < len(SHAPES)   # queues of several problems where their stages fit
    s = torch.cuda.current_stream().cuda_stream
    for _ in range(2):   # launches, then the recorded graph
        for t in ts:
            t[2].fill_(float("nan"))
        b.run(s)
        torch.cuda.synchronize()
        assert b.check_device()[0] == wg.OK
        for i, (t, w) in enumerate(zip(ts, want)):
            assert torch.equal(t[2], w), i
    b.destroy()


@pytest.mark.parametrize("slots,max_batch", [(1, 16), (3, 2)])
def test_served_burst(wg, slots, max_batch):
    """Each request's output is that of the kernel its layer runs by itself:
    the direct one, or F(2x3) (no layer here runs F(4x3))."""
    ts = _tensors(SHAPES, 6)
    want = [[_by_name(wg, t, s, a) for a in (wg.ALGO_DIRECT, wg.ALGO_2X3)] for t, s in zip(ts, SHAPES)]
    srv = wg.Server(hbm_budget_bytes=4 << 30, slots=slots, max_batch=max_batch)
    layers = [srv.add_layer(s[1], s[4], s[2], s[3], t[1].data_ptr()) for t, s in zip(ts, SHAPES)]
    for order in ([0, 1, 2, 3, 4], [2, 0, 4, 1, 3]):
        for t in ts:
            t[2].fill_(float("nan"))
        torch.cuda.synchronize()
        srv.replay([layers[i] for i in order], [SHAPES[i][0] for i in order], [0.0] * len(order),
                   [ts[i][0].data_ptr() for i in order], [ts[i][2].data_ptr() for i in order])
        for i, (t, w) in enumerate(zip(ts, want)):
            assert torch.equal(t[2], w[0]) or torch.equal(t[2], w[1]), i
    srv.destroy()
