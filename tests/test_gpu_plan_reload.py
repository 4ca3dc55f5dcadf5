"""A filter file loaded into a tuned plan that runs the direct kernel: calls run
the file's filter from then on, and what the caller took from the plan before
(a captured graph, a copy of the param blob) stays usable."""
import ctypes

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

N, C, H, W, K = 2, 24, 18, 20, 40


def _filter(seed):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn((K, C, 3, 3), generator=g) / 15).half().cuda()


def _plan(wg, x, f, algo):
    y = torch.zeros((N, K, H, W), dtype=torch.float16, device="cuda")
    op = wg.Conv2d(wg.make_problem(x.data_ptr(), f.data_ptr(), y.data_ptr(), N, C, H, W, K), wg.default_options(algo=algo))
    op._keep = (x, f, y)
    return op, y


def _result(wg, x, f, algo):
    op, y = _plan(wg, x, f, algo)
    op(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    op.destroy()
    return y


def _same(a, b):
    torch.cuda.synchronize()
    return torch.equal(a, b)


@pytest.fixture
def tuned(wg, tmp_path, monkeypatch):
    """Tunes the shape by a file: this algorithm, and the direct kernel for calls."""
    def tune(algo):
        path = tmp_path / f"tune{algo}"
        path.write_text(f"{N} {C} {H} {W} {K} 1 1 0 0 0 {algo + 16} 0 0.1\n")
        monkeypatch.setenv("WG_CONV2D_TUNE_FILE", str(path))
        wg.lib().conv2d_autotune_clear()
    yield tune
    wg.lib().conv2d_autotune_clear()


@pytest.mark.parametrize("algo", [0, 1, 2, 4])
def test_what_was_taken_before_a_load_stays_usable(wg, tmp_path, tuned, algo):
    g = torch.Generator().manual_seed(9)
    x = (torch.rand((N, C, H, W), generator=g) * 2 - 1).half().cuda()
    f1, f2, f3 = _filter(1), _filter(2), _filter(3)
    saved, named = str(tmp_path / "f2"), {}
    other, named[2] = _plan(wg, x, f2, algo)
    other(torch.cuda.current_stream().cuda_stream)
    other.save(saved)
    named[3] = _result(wg, x, f3, algo)
    direct = {1: _result(wg, x, f1, wg.ALGO_DIRECT), 3: _result(wg, x, f3, wg.ALGO_DIRECT)}
    tuned(algo)
    weights = f1.clone()
    op, y = _plan(wg, x, weights, wg.ALGO_AUTO)
    s = torch.cuda.current_stream().cuda_stream
    op(s)
    assert op.direct and _same(y, direct[1])
    own = op.workspace_bytes
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        op(torch.cuda.current_stream().cuda_stream)
    copy = (ctypes.c_ubyte * len(op.param)).from_buffer_copy(op.param)
    for bad in (saved[:-2], str(tmp_path / "cut")):   # no file, a cut one: nothing changes
        if bad.endswith("cut"):
            open(bad, "wb").write(open(saved, "rb").read()[:-8])
        with pytest.raises(wg.Conv2dError):
            op.load(bad)
        assert op.direct and op.workspace_bytes == own
    op.load(saved)
    assert op.algo == algo and not op.direct and op.workspace_bytes > own
    junk = [torch.full((1 << 20,), 7.0, dtype=torch.float16, device="cuda") for _ in range(8)]   # freed memory would be taken
    # the graph: the kernel and filter it was captured with; calls and copies of the blob: the file's filter
    y.zero_()
    graph.replay()
    assert _same(y, direct[1])
    y.zero_()
    op(s)
    assert _same(y, named[2])
    y.zero_()
    wg._check(wg.lib().conv2d_fp16_ex(ctypes.cast(copy, ctypes.c_void_p), ctypes.c_void_p(s)))
    assert _same(y, named[2])
    after = torch.cuda.CUDAGraph()
    with torch.cuda.graph(after):
        op(torch.cuda.current_stream().cuda_stream)
    y.zero_()
    after.replay()
    assert _same(y, named[2])
    # refreshed weights reach calls and both graphs; saving and loading again is in place
    weights.copy_(f3)
    op.refresh_filter(s)
    for run, want in ((lambda: op(s), named[3]), (graph.replay, direct[3]), (after.replay, named[3])):
        y.zero_()
        run()
        assert _same(y, want)
    both = op.workspace_bytes
    again = str(tmp_path / "again")
    op.save(again)
    op.load(saved)
    y.zero_()
    after.replay()
    assert _same(y, named[2])
    op.load(again)
    y.zero_()
    op(s)
    assert _same(y, named[3]) and op.workspace_bytes == both
    assert op.check_device()[0] == wg.OK
    del junk, graph, after
    op.destroy()
    other.destroy()
