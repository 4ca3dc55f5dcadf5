"""Direct convolution kernel (algorithm 5): bit-exact on integer inputs.

Inputs are integers in [-2, 2] and filters in {-1, 0, 1}, so every product and
every partial sum below 2^24 is exact in the fp32 accumulator whatever the
summation order, and the one rounding to the output type is that of the exact
integer: the result equals the rounded 64-bit convolution bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _run(wg, n, c, h, w, k, pad, nhwc=False, bf16=False, bn=0):
    dt = torch.bfloat16 if bf16 else torch.float16
    g = torch.Generator().manual_seed(n + 3 * c + 5 * h + 7 * w + 11 * k)
    x = torch.randint(-2, 3, (n, c, h, w), generator=g).double()
    f = torch.randint(-1, 2, (k, c, 3, 3), generator=g).double()
    want = torch.nn.functional.conv2d(x, f, padding=pad).to(dt)
    xd = x.to(dt).cuda()
    if nhwc:
        xd = xd.permute(0, 2, 3, 1).contiguous()
    oh, ow = want.shape[2:]
    fd = f.to(dt).cuda()
    guard = 64   # values past the output that must stay as they are
    size = n * k * oh * ow
    y = torch.full((size + guard,), 7.0, dtype=dt, device="cuda")
    prob = wg.make_problem(xd.data_ptr(), fd.data_ptr(), y.data_ptr(), n, c, h, w, k, pad[0], pad[1])
    op = wg.Conv2d(prob, wg.default_options(algo=wg.ALGO_DIRECT, layout_nhwc=int(nhwc), io_bf16=int(bf16), gemm_bn=bn))
    assert op.algo == wg.ALGO_DIRECT and op.launches_per_call == 1
    s = torch.cuda.current_stream().cuda_stream
    op(s)
    op(s)
    torch.cuda.synchronize()
    st, site = op.check_device()
    assert st == wg.OK, site
    op.destroy()
    got = y[:size].cpu().reshape((n, oh, ow, k) if nhwc else (n, k, oh, ow))
    if nhwc:
        got = got.permute(0, 3, 1, 2)
    assert torch.equal(got, want), (got.double() - want.double()).abs().max()
    assert bool((y[size:] == 7.0).all())


@pytest.mark.parametrize("shape,pad", [
    ((1, 1, 1, 1, 1), (1, 1)), ((1, 3, 7, 7, 5), (1, 1)), ((1, 8, 3, 3, 4), (0, 0)), ((2, 5, 14, 14, 27), (1, 1)),
    ((1, 16, 56, 56, 64), (1, 1)), ((3, 17, 13, 9, 33), (0, 1)), ((2, 40, 9, 31, 31), (1, 0)), ((5, 24, 7, 7, 65), (2, 2)),
    ((1, 130, 20, 20, 257), (1, 1)), ((40, 33, 7, 7, 40), (1, 1)), ((1, 12, 4, 5, 7), (3, 5)), ((1, 2, 2, 2, 3), (64, 64)),
    ((2, 16, 3, 300, 20), (1, 1)), ((1, 20, 5, 700, 8), (1, 1)), ((16, 64, 33, 31, 96), (1, 1)),
    ((300, 16, 5, 5, 16), (0, 0)), ((8, 256, 28, 28, 512), (1, 1)),
])
def test_exact_on_integers(wg, shape, pad):
    _run(wg, *shape, pad)


@pytest.mark.parametrize("bn,mb", [(32, 1), (32, 2), (32, 4), (32, 8), (64, 1), (64, 2), (64, 4), (96, 1), (96, 2), (128, 1),
                                   (128, 2), (160, 1), (192, 1), (224, 1), (256, 1)])
@pytest.mark.parametrize("w", [30, 31])
def test_every_tile(wg, bn, mb, w):
    # bn channels x mb x 128 positions; even rows are read as pixel pairs, odd ones singly
    _run(wg, 3, 48, 29, w, 300, (1, 1), bn=bn + 512 * mb)
    _run(wg, 40, 20, 5, w - 20, 33, (1, 1), bn=bn + 512 * mb)


def test_whole_rounds_and_a_tail(wg):
    # 96 tiles of 256 positions and more: 76 in one round, the others in smaller items
    _run(wg, 20, 32, 40, 40, 256, (1, 1), bn=256)
    _run(wg, 20, 32, 40, 41, 256, (1, 1), bn=256, nhwc=True)


@pytest.mark.parametrize("shape,pad", [((1, 8, 5, 5, 8), (1, 1)), ((3, 24, 13, 17, 20), (0, 0)), ((2, 64, 56, 56, 96), (1, 1)),
                                       ((1, 40, 6, 240, 33), (1, 2)), ((20, 136, 7, 7, 72), (2, 1))])
def test_channels_last(wg, shape, pad):
    _run(wg, *shape, pad, nhwc=True)


@pytest.mark.parametrize("shape,tile", [((200, 16, 28, 28, 256), 0), ((300, 24, 14, 14, 40), 32 + 512), ((5, 40, 90, 90, 64), 32 + 512),
                                        ((64, 8, 30, 30, 32), 32 + 1024)])
def test_channels_last_many_items(wg, shape, tile):
    # 3 to 13 items per CTA pair: both item tables are filled again and again, by
    # items of one chunk (fewer than the producer groups) to three
    _run(wg, *shape, (1, 1), nhwc=True, bn=tile)


@pytest.mark.parametrize("shape,nhwc,tile", [
    ((2, 64, 6, 1000, 40), False, 0), ((1, 80, 4, 1080, 40), False, 0), ((12, 96, 40, 40, 256), True, 256 + 512),
    ((19, 296, 32, 32, 280), True, 0), ((5, 312, 56, 56, 720), True, 0), ((1, 80, 12, 400, 70), True, 0),
    ((8, 200, 64, 64, 64), True, 64 + 512 * 2)])
def test_fewest_stages(wg, shape, nhwc, tile):
    # windows or filter tiles that leave the rings little more than their fewest stages
    _run(wg, *shape, (1, 1), nhwc=nhwc, bn=tile)


@pytest.mark.parametrize("shape", [(1, 3, 8, 8, 5), (4, 72, 28, 28, 130)])
def test_bf16(wg, shape):
    _run(wg, *shape, (1, 1), bf16=True)


def test_filter_files(wg, tmp_path, monkeypatch):
    """A tuned plan that runs the direct kernel stands for its Winograd
    algorithm: it saves that algorithm's filter (of the weights it was first
    called with), and runs that algorithm from a loaded one.  A plan asked for
    direct by name keeps its own files."""
    n, c, h, w, k = 2, 24, 18, 20, 40
    g = torch.Generator().manual_seed(5)
    x = (torch.rand((n, c, h, w), generator=g) * 2 - 1).half().cuda()
    f = (torch.randn((k, c, 3, 3), generator=g) / 15).half().cuda()
    s = torch.cuda.current_stream().cuda_stream

    def plan(weights, algo):
        y = torch.zeros((n, k, h, w), dtype=torch.float16, device="cuda")
        prob = wg.make_problem(x.data_ptr(), weights.data_ptr(), y.data_ptr(), n, c, h, w, k)
        op = wg.Conv2d(prob, wg.default_options(algo=algo))
        op._keep = (weights, y)
        return op, y

    def garbage():
        return torch.full_like(f, 7.0)

    by_name, yd = plan(f, wg.ALGO_DIRECT)
    by_name(s)
    own = str(tmp_path / "direct")
    by_name.save(own)
    again, ya = plan(garbage(), wg.ALGO_DIRECT)
    again.load(own)
    again(s)
    torch.cuda.synchronize()
    assert torch.equal(ya, yd)
    try:
        for algo in (wg.ALGO_4X3, wg.ALGO_2X3, wg.ALGO_2X3_FUSED, wg.ALGO_4X3_ROW):
            tune = tmp_path / f"tune{algo}"
            tune.write_text(f"{n} {c} {h} {w} {k} 1 1 0 0 0 {algo + 16} 0 0.1\n")
            monkeypatch.setenv("WG_CONV2D_TUNE_FILE", str(tune))
            wg.lib().conv2d_autotune_clear()
            named, yn = plan(f, algo)
            named(s)
            path = str(tmp_path / f"f{algo}")
            named.save(path)
            mine = f.clone()
            a, y = plan(mine, wg.ALGO_AUTO)
            assert a.algo == algo and a.direct and a.launches_per_call == 1
            a(s)
            torch.cuda.synchronize()
            assert torch.equal(y, yd)
            mine.fill_(7.0)          # the plan keeps the weights of its first call
            path2 = str(tmp_path / f"a{algo}")
            a.save(path2)
            assert open(path, "rb").read() == open(path2, "rb").read()
            b, yb = plan(garbage(), wg.ALGO_AUTO)
            b.load(path)
            assert b.algo == algo and not b.direct
            b(s)
            torch.cuda.synchronize()
            assert torch.equal(yb, yn), algo
            with pytest.raises(wg.Conv2dError):
                again.load(path)
            with pytest.raises(wg.Conv2dError):
                a.load(own)
    finally:
        wg.lib().conv2d_autotune_clear()


def test_one_queue_of_many_problems(wg, tmp_path, monkeypatch):
    """A batch whose problems all run the direct kernel: one launch, exact on
    integers, from one pixel to several rounds of items, odd and even rows."""
    shapes = [(1, 3, 1, 1, 1), (2, 16, 7, 7, 40), (20, 32, 40, 40, 256), (3, 17, 13, 9, 33), (1, 64, 56, 56, 64),
              (1, 20, 5, 300, 8), (40, 33, 7, 7, 300)]
    tune = tmp_path / "tune"
    tune.write_text("".join(f"{n} {c} {h} {w} {k} 1 1 0 0 0 {wg.ALGO_2X3 + 16} 0 0.1\n" for n, c, h, w, k in shapes))
    monkeypatch.setenv("WG_CONV2D_TUNE_FILE", str(tune))
    wg.lib().conv2d_autotune_clear()
    g = torch.Generator().manual_seed(3)
    try:
        probs, keep = [], []
        for n, c, h, w, k in shapes:
            x = torch.randint(-2, 3, (n, c, h, w), generator=g).double()
            f = torch.randint(-1, 2, (k, c, 3, 3), generator=g).double()
            want = torch.nn.functional.conv2d(x, f, padding=1).half()
            xd, fd = x.half().cuda(), f.half().cuda()
            y = torch.zeros((n, k, h, w), dtype=torch.float16, device="cuda")
            probs.append(wg.make_problem(xd.data_ptr(), fd.data_ptr(), y.data_ptr(), n, c, h, w, k))
            keep.append((xd, fd, y, want))
        b = wg.Batch(probs, wg.default_options(algo=wg.ALGO_AUTO))
    finally:
        wg.lib().conv2d_autotune_clear()
    assert b.launches(True) == 1 and b.launches(False) == len(shapes)
    s = torch.cuda.current_stream().cuda_stream
    for _ in range(3):   # direct launches, then the recorded graph
        for _, _, y, _ in keep:
            y.zero_()
        b.run(s)
        torch.cuda.synchronize()
        st, site = b.check_device()
        assert st == wg.OK, site
        for i, (_, _, y, want) in enumerate(keep):
            assert torch.equal(y.cpu(), want), i
    b.destroy()


def test_served_layers_of_an_older_file(wg, tmp_path):
    """A layer file without the direct kernel's filters (they follow the
    others) still loads, and its layers run the Winograd transform; a file cut
    inside them is refused."""
    c, k, h = 64, 96, 14
    g = torch.Generator().manual_seed(8)
    wt = (torch.randn((k, c, 3, 3), generator=g) / 24).half().cuda()
    x = (torch.rand((3, c, h, h), generator=g) * 2 - 1).half().cuda()

    def run(server, layer):
        y = torch.zeros((3, k, h, h), dtype=torch.float16, device="cuda")
        torch.cuda.synchronize()
        server.submit(layer, 3, x.data_ptr(), y.data_ptr())
        server.wait_all()
        return y.cpu()

    a = wg.Server(hbm_budget_bytes=1 << 28)
    a.add_layer(c, k, h, h, wt.data_ptr())
    path = tmp_path / "layers"
    a.save_layers(str(path))
    ya = run(a, 0)
    f2 = wg.Server(hbm_budget_bytes=1 << 28, algo=wg.ALGO_2X3)
    f2.add_layer(c, k, h, h, wt.data_ptr())
    y2 = run(f2, 0)
    raw = path.read_bytes()
    cut = raw.rindex(b"WGCSRVD1")
    older, broken = tmp_path / "older", tmp_path / "broken"
    older.write_bytes(raw[:cut])
    broken.write_bytes(raw[:-2])
    b = wg.Server(hbm_budget_bytes=1 << 28)
    assert torch.equal(run(b, b.load_layers(str(path))[0]), ya)
    assert torch.equal(run(b, b.load_layers(str(older))[0]), y2)
    with pytest.raises(wg.Conv2dError):
        b.load_layers(str(broken))
    for server in (a, f2, b):
        server.destroy()
