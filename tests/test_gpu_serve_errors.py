"""Served requests that cannot be launched: reported as failed, with the others
of their batch computed and the server usable."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

# c, k, h, w: an ordinary layer, and rows too wide for every kernel of the server
GOOD, WIDE = (64, 96, 14, 14), (8, 8, 4, 2400)


def _layer(srv, dims, seed):
    c, k, h, w = dims
    g = torch.Generator().manual_seed(seed)
    f = (torch.randn((k, c, 3, 3), generator=g) / (9 * c) ** 0.5).half().cuda()
    return srv.add_layer(c, k, h, w, f.data_ptr()), f


def _request(dims, n, seed):
    c, k, h, w = dims
    g = torch.Generator().manual_seed(seed)
    x = (torch.rand((n, c, h, w), generator=g) * 2 - 1).half().cuda()
    return x, torch.full((n, k, h, w), float("nan"), dtype=torch.float16, device="cuda")


@pytest.mark.parametrize("order", ["GWG", "WGW", "W", "WW"])
@pytest.mark.parametrize("by_replay", [True, False])
def test_failed_requests_are_reported(wg, order, by_replay):
    srv = wg.Server(slots=2, max_batch=16, hbm_budget_bytes=1 << 28)
    good, fg = _layer(srv, GOOD, 1)
    wide, fw = _layer(srv, WIDE, 2)
    x, want = _request(GOOD, 3, 3)
    torch.cuda.synchronize()
    srv.replay([good], [3], [0.0], [x.data_ptr()], [want.data_ptr()])
    assert bool(torch.isfinite(want).all())
    reqs = [(good, 3, x, torch.full_like(want, float("nan"))) if o == "G" else (wide, 1, *_request(WIDE, 1, 4)) for o in order]
    torch.cuda.synchronize()
    ids = []
    with pytest.raises(wg.Conv2dError):
        if by_replay:
            srv.replay([r[0] for r in reqs], [r[1] for r in reqs], [0.0] * len(reqs), [r[2].data_ptr() for r in reqs],
                       [r[3].data_ptr() for r in reqs])
        else:
            ids = [srv.submit(r[0], r[1], r[2].data_ptr(), r[3].data_ptr()) for r in reqs]
            srv.wait_all()
    for o, rid in zip(order, ids):
        assert srv.poll(rid)[0] == (1 if o == "G" else -2)
    for o, r in zip(order, reqs):
        assert torch.equal(r[3], want) if o == "G" else bool(r[3].isnan().all())
    # reported once; workspaces given back; later requests as before
    srv.wait_all()
    assert srv.stats()["arena_used_bytes"] == 0
    y = torch.full_like(want, float("nan"))
    torch.cuda.synchronize()
    srv.replay([good], [3], [0.0], [x.data_ptr()], [y.data_ptr()])
    assert torch.equal(y, want)
    srv.destroy()
