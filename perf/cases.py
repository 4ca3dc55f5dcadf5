"""What the operator's users have it do: 3x3 stride-1 convolutions through the
public calls, as cases that can be timed and checked.

A case is one of
  plan   a layer planned once (getkernelInfo_ex) and called on device tensors
         (conv2d_fp16_ex): NCHW fp16, channels-last fp16 or bf16 end to end;
  host   the same layer called on pinned host buffers (conv2d_fp16_host);
  batch  many uneven layers planned together and run as one group
         (conv2d_batch_run);
  serve  resident layers behind the request loop (conv2d_server_replay, every
         request arriving at once).
Sizes are those of the benchmark's workloads and of the reference benchmark's
shapes, or generic.  Activations are uniform in [-1, 1] (normal where the
precision study has them so), filters normal with standard deviation
1/sqrt(9 C), as the benchmark draws them.
"""
import importlib
import math

import torch

wg = importlib.import_module("dcu-winograd-conv2d_gb300")

# 24 uneven layers "n,c,h,k" (input h x h, pad 1), the benchmark's batched workload
BATCH24 = ("16,512,56,512;4,256,28,64;1,64,56,256;128,64,14,64;32,256,28,256;4,512,28,256;2,512,28,128;8,256,112,256;"
           "32,64,28,64;128,256,14,64;4,256,112,64;16,256,56,512;1,256,112,512;1,64,112,512;128,128,14,64;4,128,56,512;"
           "64,64,7,512;16,256,14,256;4,64,112,128;4,64,56,512;2,256,56,128;32,64,28,256;4,64,28,512;1,64,112,256")
# 16 resident layers "c,h,k", the benchmark's serving workload
LAYERS16 = ("512,56,512;256,7,256;128,14,128;256,7,256;64,14,64;512,28,256;128,112,256;256,14,128;512,28,128;"
            "64,56,256;512,7,128;64,56,256;256,14,64;512,7,256;512,28,128;512,28,256")


def _layer(kind, n, c, h, w, k, pad_h=1, pad_w=1, dtype="f16", layout="nchw", rule="auto", normal=False):
    return {"kind": kind, "n": n, "c": c, "h": h, "w": w, "k": k, "pad_h": pad_h, "pad_w": pad_w, "dtype": dtype,
            "layout": layout, "rule": rule, "normal": normal}


def listed():
    return [
        # one image of a small layer: an interactive call, where launches and latency count
        dict(_layer("plan", 1, 64, 56, 56, 64), name="one image 64x56x56 to 64"),
        # small images in a modest batch (one of the reference benchmark's shapes)
        dict(_layer("plan", 32, 256, 14, 14, 256), name="32x256x14x14 to 256"),
        # large images, few channels (reference benchmark)
        dict(_layer("plan", 16, 64, 128, 128, 64), name="16x64x128x128 to 64"),
        # the benchmark's headline layer
        dict(_layer("plan", 32, 256, 56, 56, 256), name="32x256x56x56 to 256"),
        # wide channels, the precision study's layer
        dict(_layer("plan", 32, 512, 28, 28, 512, normal=True), name="32x512x28x28 to 512"),
        # odd sizes throughout: padding in every dimension, nothing aligned
        dict(_layer("plan", 5, 100, 61, 45, 75), name="ragged 5x100x61x45 to 75"),
        # two large images with the reference's own selection rule, as a caller who wants its algorithms asks for it
        dict(_layer("plan", 2, 640, 64, 64, 640, rule="reference"), name="2x640x64x64 to 640 by rule"),
        # channels-last activations
        dict(_layer("plan", 32, 128, 56, 56, 128, layout="nhwc"), name="nhwc 32x128x56x56 to 128"),
        # bf16 tensors end to end
        dict(_layer("plan", 32, 256, 28, 28, 256, dtype="bf16"), name="bf16 32x256x28x28 to 256"),
        # activations that live in host memory: copy in, convolve, copy out
        dict(_layer("host", 16, 128, 28, 28, 128), name="host 16x128x28x28 to 128"),
        # a network's worth of uneven layers in one grouped run
        {"kind": "batch", "layers": BATCH24, "name": "batch of 24 layers"},
        # a burst of mixed requests on resident layers
        {"kind": "serve", "layers": LAYERS16, "requests": 24, "max_n": 32, "name": "burst of 24 requests"},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["plan"] * 9 + ["host", "batch", "serve"])
    if kind == "batch":
        rows, left = [], 300e9
        for _ in range(rng.randint(4, 20)):
            n, c, h, k = _log_int(rng, 1, 64), rng.choice([64, 128, 256, 512]), rng.choice([7, 14, 28, 56]), rng.choice(
                [64, 128, 256, 512])
            if _flops(n, c, h, h, k, 1, 1) < left:
                left -= _flops(n, c, h, h, k, 1, 1)
                rows.append("%d,%d,%d,%d" % (n, c, h, k))
        return {"kind": "batch", "layers": ";".join(rows)}
    if kind == "serve":
        rows = ["%d,%d,%d" % (rng.choice([64, 128, 256, 512]), rng.choice([7, 14, 28, 56]), rng.choice([64, 128, 256, 512]))
                for _ in range(rng.randint(2, 8))]
        return {"kind": "serve", "layers": ";".join(rows), "requests": rng.randint(4, 24), "max_n": rng.randint(2, 16)}
    while True:
        form = rng.choice(["f16", "f16", "f16", "bf16", "nhwc"])
        n, c, h, k = _log_int(rng, 1, 128), _log_int(rng, 3, 1280), _log_int(rng, 7, 128), _log_int(rng, 4, 1280)
        w = h if rng.random() < 0.5 else _log_int(rng, 7, 128)
        if rng.random() < 0.6:
            c, k = max(16, c // 16 * 16), max(16, k // 16 * 16)
        if form == "nhwc":
            c, k = max(16, c // 16 * 16), max(16, k // 16 * 16)
        pad = rng.choice([(1, 1)] * 6 + [(0, 0), (2, 2), (0, 1), (1, 0)])
        flops = _flops(n, c, h, w, k, *pad)
        if 1e6 < flops < 118e9 and n * h * w * max(c, k) < 60e6:
            return _layer(kind, n, c, h, w, k, pad[0], pad[1], "bf16" if form == "bf16" else "f16",
                          "nhwc" if form == "nhwc" and kind == "plan" else "nchw",
                          "reference" if form == "f16" and kind == "plan" and rng.random() < 0.1 else "auto",
                          rng.random() < 0.3)


def _flops(n, c, h, w, k, ph, pw):
    """Direct-convolution operations."""
    return 18.0 * n * k * (h + 2 * ph - 2) * (w + 2 * pw - 2) * c


def _shapes(case):
    """The convolutions of a case: (n, c, h, w, k, pad_h, pad_w) each."""
    if case["kind"] == "batch":
        rows = [tuple(int(v) for v in r.split(",")) for r in case["layers"].split(";")]
        return [(n, c, h, h, k, 1, 1) for n, c, h, k in rows]
    if case["kind"] == "serve":
        rows = [tuple(int(v) for v in r.split(",")) for r in case["layers"].split(";")]
        return [(n, rows[li][0], rows[li][1], rows[li][1], rows[li][2], 1, 1) for li, n in _requests(case)]
    return [(case["n"], case["c"], case["h"], case["w"], case["k"], case["pad_h"], case["pad_w"])]


def _requests(case):
    """(layer, images) of each request, spread over the layers and the batch sizes."""
    count = case["layers"].count(";") + 1
    return [((7 * i + i // count) % count, 1 + (11 * i + 5) % case["max_n"]) for i in range(case["requests"])]


def work(case):
    """Input, filter and output once each; the operations are those of the
    least-multiplying algorithm on the path, F(4x3): 36 products for 16 outputs."""
    nbytes = flops = 0.0
    seen = set()
    for i, (n, c, h, w, k, ph, pw) in enumerate(_shapes(case)):
        oh, ow = h + 2 * ph - 2, w + 2 * pw - 2
        nbytes += 2.0 * n * (c * h * w + k * oh * ow)
        layer = _requests(case)[i][0] if case["kind"] == "serve" else i
        if layer not in seen:
            nbytes += 18.0 * k * c
            seen.add(layer)
        flops += 72.0 * n * (oh * ow / 16.0) * c * k
    return {"bytes": nbytes, "flops": flops}


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _activation(g, n, c, h, w, dtype, normal):
    if normal:
        x = torch.randn((n, c, h, w), generator=g, device="cuda")
    else:
        x = torch.rand((n, c, h, w), generator=g, device="cuda") * 2 - 1
    return x.to(dtype)


def _filter(g, k, c, dtype):
    return (torch.randn((k, c, 3, 3), generator=g, device="cuda") / math.sqrt(9 * c)).to(dtype)


def _tensors(case, seed):
    """(activations, filters) of the case, one pair per convolution; the
    requests of one served layer share its filter."""
    g = _generator(seed)
    dtype = torch.bfloat16 if case.get("dtype") == "bf16" else torch.float16
    xs, ws, layers = [], [], {}
    for i, (n, c, h, w, k, _, _) in enumerate(_shapes(case)):
        xs.append(_activation(g, n, c, h, w, dtype, case.get("normal", False)))
        layer = _requests(case)[i][0] if case["kind"] == "serve" else i
        if layer not in layers:
            layers[layer] = _filter(g, k, c, dtype)
        ws.append(layers[layer])
    return xs, ws


def prepare(case, seed):
    xs, ws = _tensors(case, seed)
    shapes = _shapes(case)
    state = {"kind": case["kind"], "x": xs, "w": ws}
    if case["kind"] == "batch":
        ys = [torch.empty((n, k, h + 2 * p - 2, w + 2 * q - 2), dtype=torch.float16, device="cuda")
              for n, c, h, w, k, p, q in shapes]
        torch.cuda.synchronize()
        problems = [wg.make_problem(x.data_ptr(), f.data_ptr(), y.data_ptr(), *s)
                    for x, f, y, s in zip(xs, ws, ys, shapes)]
        return dict(state, y=ys, op=wg.Batch(problems))
    if case["kind"] == "serve":
        rows = [tuple(int(v) for v in r.split(",")) for r in case["layers"].split(";")]
        requests = _requests(case)
        ys = [torch.empty((n, k, h, w), dtype=torch.float16, device="cuda") for n, c, h, w, k, p, q in shapes]
        torch.cuda.synchronize()
        server = wg.Server(hbm_budget_bytes=8 << 30)
        index = {}
        for (layer, _), f in zip(requests, ws):
            if layer not in index:
                c, h, k = rows[layer]
                index[layer] = server.add_layer(c, k, h, h, f.data_ptr())
        return dict(state, y=ys, op=server, layers=[index[layer] for layer, _ in requests],
                    images=[n for _, n in requests], arrivals=[0.0] * len(requests),
                    ins=[x.data_ptr() for x in xs], outs=[y.data_ptr() for y in ys])
    n, c, h, w, k, p, q = shapes[0]
    x, f, nhwc = xs[0], ws[0], case["layout"] == "nhwc"
    oh, ow = h + 2 * p - 2, w + 2 * q - 2
    if nhwc:
        x = x.permute(0, 2, 3, 1).contiguous()
    y = torch.empty((n, oh, ow, k) if nhwc else (n, k, oh, ow), dtype=x.dtype, device="cuda")
    torch.cuda.synchronize()
    options = {}
    if case["rule"] == "reference":
        options["algo"] = wg.ALGO_REFERENCE
    if nhwc:
        options["layout_nhwc"] = 1
    if case["dtype"] == "bf16":
        options["io_bf16"] = 1
    op = wg.Conv2d(wg.make_problem(x.data_ptr(), f.data_ptr(), y.data_ptr(), n, c, h, w, k, p, q),
                   wg.default_options(**options) if options else None)
    state.update(x=x, w=f, y=y, op=op)
    if case["kind"] == "host":
        state.update(host_x=x.cpu().pin_memory(), host_y=torch.empty(y.shape, dtype=y.dtype, pin_memory=True))
    return state


def run(state):
    op = state["op"]
    if state["kind"] == "serve":
        op.replay(state["layers"], state["images"], state["arrivals"], state["ins"], state["outs"])
        return state["y"]
    stream = torch.cuda.current_stream().cuda_stream
    if state["kind"] == "host":
        op.host(state["host_x"].data_ptr(), state["host_y"].data_ptr(), stream)
        return state["host_y"]
    if state["kind"] == "batch":
        op.run(stream)
    else:
        op(stream)
    return state["y"]


def _conv64(x, f, ph, pw):
    """Direct convolution in 64 bits: one matrix product per filter tap."""
    n, c, h, w = x.shape
    k = f.shape[0]
    oh, ow = h + 2 * ph - 2, w + 2 * pw - 2
    taps = f.double().permute(2, 3, 0, 1).contiguous()
    y = torch.empty((n, k, oh * ow), dtype=torch.float64, device=x.device)
    step = max(1, int(2e8 // (8 * c * (h + 2) * (w + 2))))
    for i in range(0, n, step):
        xp = torch.nn.functional.pad(x[i:i + step].double(), (pw, pw, ph, ph))
        acc = None
        for r in range(3):
            for s in range(3):
                part = torch.matmul(taps[r, s], xp[:, :, r:r + oh, s:s + ow].reshape(-1, c, oh * ow))
                acc = part if acc is None else acc.add_(part)
        y[i:i + step] = acc
    return y.reshape(n, k, oh, ow)


def exact(case, seed):
    xs, ws = _tensors(case, seed)
    out = [_conv64(x, f, s[5], s[6]) for x, f, s in zip(xs, ws, _shapes(case))]
    if case["kind"] in ("batch", "serve"):
        return out
    y = out[0]
    if case["layout"] == "nhwc":
        y = y.permute(0, 2, 3, 1).contiguous()
    return y.cpu() if case["kind"] == "host" else y
