"""The kernel that a served layer runs, by the width of its rows: each request's
output is, bit for bit, that of the expected algorithm called by name."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

DIRECT, F2, F4 = 5, 1, 0


@pytest.mark.parametrize("c,k,h,w,algo", [
    (64, 64, 9, 900, DIRECT), (64, 64, 9, 902, F2), (40, 32, 5, 1080, F2), (32, 40, 5, 1080, DIRECT), (8, 8, 5, 1079, DIRECT),
    (256, 64, 9, 801, DIRECT), (256, 64, 9, 803, F2), (256, 256, 10, 900, DIRECT), (128, 128, 14, 640, DIRECT),
    (128, 128, 14, 642, F4), (128, 128, 15, 639, DIRECT), (128, 128, 15, 641, F4), (256, 256, 16, 604, DIRECT),
    (256, 256, 16, 606, F4), (256, 256, 16, 349, DIRECT), (256, 256, 16, 351, F4), (256, 512, 14, 426, DIRECT),
    (256, 512, 14, 428, F4), (40, 24, 6, 1400, F2)])
def test_rows(wg, c, k, h, w, algo):
    g = torch.Generator().manual_seed(w)
    x = (torch.rand((2, c, h, w), generator=g) * 2 - 1).half().cuda()
    f = (torch.randn((k, c, 3, 3), generator=g) / (9 * c) ** 0.5).half().cuda()
    got, want = (torch.zeros((2, k, h, w), dtype=torch.float16, device="cuda") for _ in range(2))
    op = wg.Conv2d(wg.make_problem(x.data_ptr(), f.data_ptr(), want.data_ptr(), 2, c, h, w, k), wg.default_options(algo=algo))
    assert op.algo == algo
    op(torch.cuda.current_stream().cuda_stream)
    srv = wg.Server(hbm_budget_bytes=1 << 30)
    layer = srv.add_layer(c, k, h, w, f.data_ptr())
    torch.cuda.synchronize()
    srv.replay([layer], [2], [0.0], [x.data_ptr()], [got.data_ptr()])
    assert torch.equal(got, want)
    op.destroy()
    srv.destroy()
