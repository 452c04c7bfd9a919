"""Filters wider than one tap at output heights that fill no tile (a tile is as many padded rows of one image as fit 128 GEMM rows, the last
one may hang over the image): the bottleneck, whose 3 x 3 and last 1 x 1 convolution are one kernel, and a bf16 3 x 3 convolution
with a residual on its own. Compared with f64.

Tolerances: Y is rounded by 2^-8; intermediates keep 2^-17, and a tensor-core sum cuts off at most 2^-23 of its magnitude for each 16-deep
step, twice, at most 72 steps: three convolutions stay below 2^-13 of the same chain over magnitudes."""
import pytest

from deepforge_b200 import dfgpu, graphs, runtime

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def run(doc, buffers, y):
    exe = runtime.compile_graph(doc)
    workspace = torch.empty(max(exe.workspace_size, 1), dtype=torch.uint8, device="cuda")
    exe.execute({uid: b.data_ptr() for uid, b in {**buffers, 7: y}.items()}, workspace.data_ptr())
    torch.cuda.synchronize()
    assert dfgpu.device_status() == 0
    return exe


def conv(x, w, pad):   # NHWC, KRSC, f64 on the CPU
    return torch.nn.functional.conv2d(x.permute(0, 3, 1, 2), w.permute(0, 3, 1, 2), padding=pad).permute(0, 2, 3, 1)


@pytest.mark.parametrize("n,h,w", [(1, 7, 7), (2, 11, 11), (3, 13, 13), (1, 17, 9), (2, 23, 23), (1, 31, 60), (1, 5, 126), (2, 53, 53), (40, 19, 19), (1, 1, 1), (1, 2, 125)])
def test_bottleneck(n, h, w):
    g = torch.Generator(device="cuda").manual_seed(h * 67 + w)
    randn = lambda *shape, std=1.0: (torch.randn(*shape, device="cuda", generator=g) * std).to(torch.bfloat16)
    x, w1, w2, w3 = randn(n, h, w, 256), randn(64, 1, 1, 256, std=256 ** -0.5), randn(64, 3, 3, 64, std=(9 * 64) ** -0.5), randn(256, 1, 1, 64, std=64 ** -0.5)
    b1, b2 = randn(64, std=0.1), randn(64, std=0.1)
    y = torch.full((n, h, w, 256), float("nan"), dtype=torch.bfloat16, device="cuda")
    exe = run(graphs.c2_bottleneck(n, h, w), {1: x, 2: w1, 3: b1, 4: w2, 5: b2, 6: w3}, y)
    assert len(exe.steps()) == 2 or not 7 <= w <= 56   # (wider: one window and the filters do not fit the shared memory)
    fx, f1, f2, f3, fb1, fb2 = (t.double().cpu() for t in (x, w1, w2, w3, b1, b2))
    want = conv(torch.relu(conv(torch.relu(conv(fx, f1, 0) + fb1), f2, 1) + fb2), f3, 0) + fx
    weight = conv(conv(conv(fx.abs(), f1.abs(), 0) + fb1.abs(), f2.abs(), 1) + fb2.abs(), f3.abs(), 0) + fx.abs()
    error, bound = (y.double().cpu() - want).abs(), 2.0 ** -8 * want.abs() + 2.0 ** -13 * weight
    assert bool(torch.all(error <= bound)), float((error / bound).max())


@pytest.mark.parametrize("n,h,w", [(1, 11, 11), (2, 13, 20), (1, 53, 53)])
def test_convolution_with_residual(n, h, w):
    g = torch.Generator(device="cuda").manual_seed(h)
    x, f, r = (torch.randn(*shape, device="cuda", generator=g).to(torch.bfloat16) for shape in ((n, h, w, 64), (128, 3, 3, 64), (n, h, w, 128)))
    y = torch.full((n, h, w, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    dims = lambda c: [n, c, h, w]
    tensors = [graphs.tensor(1, "X", dims(64), "BFLOAT16", graphs.nhwc(dims(64))), graphs.tensor(2, "W", [128, 64, 3, 3], "BFLOAT16", graphs.nhwc([128, 64, 3, 3])),
               graphs.tensor(3, "R", dims(128), "BFLOAT16", graphs.nhwc(dims(128))), graphs.tensor(5, "c", dims(128), strides=graphs.nhwc(dims(128)), virtual=True),
               graphs.tensor(7, "Y", dims(128), "BFLOAT16", graphs.nhwc(dims(128)))]
    nodes = [graphs.conv_node("conv", 1, 2, 5), graphs.pointwise_node("add", "ADD", 5, 7, 3)]
    run(graphs.document("conv_rows", nodes, tensors, io="BFLOAT16"), {1: x, 2: f, 3: r}, y)
    fx, ff, fr = (t.double().cpu() for t in (x, f, r))
    want, weight = conv(fx, ff, 1) + fr, conv(fx.abs(), ff.abs(), 1) + fr.abs()
    assert bool(torch.all((y.double().cpu() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -13 * weight))
