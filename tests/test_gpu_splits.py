"""Work splits that depend on the sizes: the GEMM's tile and pairing, and the
F(4x3) input transform's blocks of channels and tile rows."""
import numpy as np
import pytest

import oracle as O
from test_gpu_parity import _dev_array, opts_for, run

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


# (N, C, HW, K): N images of one F(4x3) tile (four F(2x3) ones); single-CTA
# items, then CTA pairs with 2, 3 and 5 blocks of 128 tiles (an odd one leaves
# half a pair empty), channel remainders of the 128- and 256-wide blocks, and
# depths around the 64-channel stages
GEMM_SIZES = [(128, 16, 4, 600), (129, 8, 4, 129), (129, 24, 4, 600), (257, 72, 4, 257), (385, 64, 4, 160), (600, 100, 4, 300),
              (33, 520, 8, 512), (520, 130, 3, 96), (300, 40, 5, 385)]


@pytest.mark.parametrize("bn", [0, 128, 256])
@pytest.mark.parametrize("n,c,h,k", GEMM_SIZES)
@pytest.mark.parametrize("algo,mfp32,bf16", [(0, 0, 0), (0, 1, 0), (1, 0, 0), (1, 0, 1)])
def test_gemm_tiles_agree_bit_for_bit(wg, algo, mfp32, bf16, n, c, h, k, bn):
    """Each accumulator adds the same products, 16 channels at a time, in the
    same order whatever the tile, so every tile gives the bits of the 32-wide
    single-CTA one (which the oracle tests cover)."""
    x, wt = O.uniform_inputs(n + k, n, c, h, h, k)
    dt = torch.bfloat16 if bf16 else torch.float16
    xd, wd = torch.from_numpy(x).cuda().to(dt), torch.from_numpy(wt).cuda().to(dt)
    got = []
    for b in (32, bn):
        y, op = wg.conv2d_torch(xd, wd, 1, 1, opts_for(wg, algo, m_fp32=mfp32, gemm_bn=b))
        torch.cuda.synchronize()
        st, site = op.check_device()
        assert st == wg.OK, site
        got.append(y.view(torch.int16).cpu())
        op.destroy()
    assert torch.equal(got[0], got[1])


# blocks of 24 and 32 channels with a remainder of C, one to nine tile rows,
# and groups of eight tiles that end inside a row
@pytest.mark.parametrize("n,c,h,w", [(64, 100, 14, 14), (100, 50, 7, 7), (40, 172, 10, 22), (54, 81, 11, 9), (45, 101, 1, 35),
                                     (40, 157, 34, 1), (58, 82, 2, 2), (3, 20, 9, 16)])
def test_input_transform_blocks(wg, monkeypatch, n, c, h, w):
    """V read back against its restatement: one fp16 rounding of an fp32 result
    (whose error the sum of |terms| bounds)."""
    monkeypatch.setenv("WG_CONV2D_KEEP_WORKSPACE", "1")
    x, wt = O.uniform_inputs(n + w, n, c, h, w, 8)
    _, op = run(wg, x, wt, 1, 1, opts_for(wg, 0))
    E, cp = 36, (c + 7) // 8 * 8
    P = n * -(-h // 4) * -(-w // 4)
    Pp = (P + 7) // 8 * 8
    V = _dev_array(wg, op.blob_pointers()[1], E * Pp * cp, np.float16).reshape(E, cp // 8, Pp, 8).transpose(0, 2, 1, 3)
    V = V[:, :P].reshape(E, P, cp).astype(np.float64)
    ref = O.input_transform(x.astype(np.float64), 4, 1, 1, "F4")
    B = np.abs(O.XFORMS["F4"][1])
    terms = np.einsum("ir,pcrs,js->ijpc", B, np.abs(O.input_tiles(x.astype(np.float64), 4, 1, 1)), B, optimize=True)
    assert np.all(V[:, :, c:] == 0)
    assert np.all(np.abs(V[:, :, :c] - ref) <= np.abs(ref) * 2.0 ** -10 + terms.reshape(E, P, c) * 2.0 ** -20)


@pytest.mark.parametrize("algo", [0, 1, 5])
@pytest.mark.parametrize("n,k", [(1, 64), (10, 64), (11, 64), (13, 64), (13, 136)])
def test_host_chunks_around_the_threshold(wg, algo, n, k):
    """409,600 bytes of copies per image: one chunk below 4 MB (10 images), two
    from there on unless one direction (k = 136: the output) has more than two
    thirds; the result of each is that of the device call, bit for bit."""
    c, h = 64, 40
    x, wt = O.uniform_inputs(n, n, c, h, h, k)
    xt, wtt = torch.from_numpy(x).cuda(), torch.from_numpy(wt).cuda()
    y = torch.empty((n, k, h, h), dtype=torch.float16, device="cuda")
    op = wg.Conv2d(wg.make_problem(xt.data_ptr(), wtt.data_ptr(), y.data_ptr(), n, c, h, h, k), opts_for(wg, algo))
    s = torch.cuda.current_stream().cuda_stream
    op(s)
    torch.cuda.synchronize()
    want = y.cpu()
    hin, hout = torch.from_numpy(x).pin_memory(), torch.zeros(want.shape, dtype=torch.float16).pin_memory()
    for _ in range(2):
        hout.zero_()
        op.host(hin.data_ptr(), hout.data_ptr(), s)
        assert torch.equal(hout.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("n,h,algo", [(40, 13, 5), (21, 14, 5), (10, 20, 5), (11, 20, 0), (4, 29, 5), (5, 28, 5), (6, 28, 0)])
def test_server_picks_per_request(wg, n, h, algo):
    """512 -> 512 channels: F(4x3) where its tiles fit the output and there are
    4,096 output pixels, else direct; the bits are those of a call by name."""
    c = k = 512
    g = torch.Generator().manual_seed(n + h)
    x = (torch.rand((n, c, h, h), generator=g) * 2 - 1).half().cuda()
    f = (torch.randn((k, c, 3, 3), generator=g) / 68).half().cuda()
    want, op = wg.conv2d_torch(x, f, 1, 1, opts_for(wg, algo))
    assert op.algo == algo
    y = torch.zeros_like(want)
    torch.cuda.synchronize()
    server = wg.Server(hbm_budget_bytes=1 << 30)
    layer = server.add_layer(c, k, h, h, f.data_ptr())
    server.replay([layer], [n], [0.0], [x.data_ptr()], [y.data_ptr()])
    torch.cuda.synchronize()
    assert torch.equal(y.view(torch.int16), want.view(torch.int16))
