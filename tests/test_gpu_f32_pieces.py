"""The f32 contractions that AUTO picks by size: the flat reduction of the one-launch tensor-core kernel (channels in fours, 1 x 1 to
5 x 5 filters, either layout of B), three bf16 pieces multiplied pair by pair (large matrix products) and the kernel for
few rows. Compared with f64.

Tolerances: a tensor-core sum cuts off what an f32 does not hold, at most 2^-23 of sum |x w| for each 16-deep step (twice:
among a step's products and against what has been summed up), and the pieces leave out products below 2^-23; on the CUDA cores every one of
K additions and products rounds by at most 2^-24."""
import numpy as np
import pytest

from deepforge_b200 import dfgpu, graphs, runtime

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def pieces_bound(depth):
    return (2 * (-(-depth // 16) + 12) + 8) * 2.0 ** -23   # (12: a rank's last unit is padded to 64, and eight ranks are added)


def run(doc, buffers, out):
    exe = runtime.compile_graph(doc)
    workspace = torch.empty(max(exe.workspace_size, 1), dtype=torch.uint8, device="cuda")
    exe.execute({uid: b.data_ptr() for uid, b in {**buffers, **out}.items()}, workspace.data_ptr())
    torch.cuda.synchronize()
    assert dfgpu.device_status() == 0
    return exe


@pytest.mark.parametrize("n,c,k,h,w,r", [(1, 4, 4, 8, 8, 1), (1, 12, 20, 9, 11, 3), (2, 8, 28, 17, 13, 3), (1, 76, 68, 10, 9, 5), (3, 16, 64, 8, 16, 1), (1, 60, 128, 15, 15, 1),
                                         (2, 124, 12, 30, 30, 5), (4, 20, 64, 32, 32, 3), (1, 64, 64, 56, 56, 3)])
def test_conv_flat_reduction(n, c, k, h, w, r):
    g = torch.Generator(device="cuda").manual_seed(c * 131 + r)
    x, f = torch.randn(n, h, w, c, device="cuda", generator=g), torch.randn(k, r, r, c, device="cuda", generator=g)
    y = torch.full((n, h, w, k), float("nan"), device="cuda")
    doc = graphs.c1_conv("nhwc", n, c, h, w, k, r, r // 2)
    uid = {t["name"]: t["uid"] for t in doc["tensors"].values()}
    names = sorted(uid.values())
    run(doc, {names[0]: x, names[1]: f}, {names[2]: y})
    conv = lambda a, b: torch.nn.functional.conv2d(a.double().cpu().permute(0, 3, 1, 2), b.double().cpu().permute(0, 3, 1, 2), padding=r // 2).permute(0, 2, 3, 1)
    assert torch.all((y.double().cpu() - conv(x, f)).abs() <= pieces_bound(c * r * r) * conv(x.abs(), f.abs()))


@pytest.mark.parametrize("m,k,n", [(1, 4, 4), (1, 4232, 1688), (2, 132, 36), (3, 128, 32), (4, 1000, 64), (5, 127, 100), (8, 130, 2052), (9, 8192, 48), (16, 260, 4096),   # few rows
                                   (17, 64, 64), (100, 120, 68), (131, 100, 76), (500, 8, 1024),                                                                       # flat, shallow
                                   (129, 516, 4100), (1000, 130, 2052), (2047, 100, 257), (255, 4100, 640), (4097, 68, 130)])                                          # pieces
@pytest.mark.parametrize("b_k_major", [False, True])
def test_matmul(m, k, n, b_k_major):
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n)
    tensors = [graphs.tensor(1, "A", [m, k]), graphs.tensor(2, "B", [k, n], strides=[1, k] if b_k_major else [n, 1]), graphs.tensor(3, "bias", [1, n]), graphs.tensor(4, "C", [m, n]),
               graphs.tensor(5, "p", [m, n], virtual=True), graphs.tensor(6, "q", [m, n], virtual=True)]
    nodes = [graphs.matmul_node("matmul", 1, 2, 5), graphs.pointwise_node("bias", "ADD", 5, 6, 3), graphs.pointwise_node("relu", "RELU_FWD", 6, 4)]
    a, b, bias = (torch.randn(count, device="cuda", generator=g) for count in (m * k, k * n, n))
    for shift in (0, 1):   # operands on and off the 16-byte boundaries
        held = [torch.empty(t.numel() + 4, device="cuda")[shift:shift + t.numel()].copy_(t) for t in (a, b)]
        c = torch.full((m * n,), float("nan"), device="cuda")
        run(graphs.document("f32", nodes, tensors), {1: held[0], 2: held[1], 3: bias}, {4: c})
        fa, fb = a.view(m, k).double(), (b.view(n, k).t() if b_k_major else b.view(k, n)).double()
        want, weight = torch.relu(fa @ fb + bias.double()), fa.abs() @ fb.abs()
        bound = max(pieces_bound(k), k * 2.0 ** -24) * weight + 2.0 ** -23 * (weight + bias.abs().double())
        assert torch.all((c.view(m, n).double() - want).abs() <= bound), float(((c.view(m, n).double() - want).abs() / bound).max())


@pytest.mark.parametrize("m,k,n", [(3, 300, 64), (200, 100, 64), (1000, 130, 2052)])
def test_matmul_with_an_infinity(m, k, n):
    """inf and NaN come out where an f32 product puts them."""
    a, b = torch.ones(m, k, device="cuda"), torch.ones(k, n, device="cuda")
    a[1, k - 1], b[5, 7] = float("inf"), float("nan")
    c = torch.zeros(m, n, device="cuda")
    tensors = [graphs.tensor(1, "A", [m, k]), graphs.tensor(2, "B", [k, n]), graphs.tensor(4, "C", [m, n])]
    run(graphs.document("f32", [graphs.matmul_node("matmul", 1, 2, 4)], tensors), {1: a, 2: b}, {4: c})
    want = np.full((m, n), float(k), np.float32)
    want[1, :], want[:, 7] = np.inf, np.nan
    assert np.array_equal(c.cpu().numpy(), want, equal_nan=True)


@pytest.mark.parametrize("depth", [4, 8, 12, 20])
@pytest.mark.parametrize("conv", [True, False])
def test_shallow_reductions_are_f32_additions(depth, conv):
    """A handful of products: one rounding each, in order (a product and a sum in f64, rounded to f32, is that but for double roundings)."""
    g = torch.Generator(device="cuda").manual_seed(depth)
    rows, k = 400, 64
    x, f = torch.randn(rows, depth, device="cuda", generator=g), torch.randn(k, depth, device="cuda", generator=g)
    y = torch.full((rows, k), float("nan"), device="cuda")
    if conv:
        doc = graphs.c1_conv("nhwc", 1, depth, 20, 20, k, 1, 0)
    else:
        doc = graphs.document("f32", [graphs.matmul_node("matmul", 1, 2, 3)], [graphs.tensor(1, "A", [rows, depth]), graphs.tensor(2, "B", [depth, k], strides=[1, depth]), graphs.tensor(3, "C", [rows, k])])
    run(doc, {1: x, 2: f}, {3: y})
    want = torch.zeros(rows, k, device="cuda")
    for i in range(depth):
        want = (x[:, i : i + 1].double() * f[:, i].double() + want.double()).float()
    assert float((y == want).float().mean()) > 0.999


@pytest.mark.parametrize("n,c,k,h,w,r", [(1, 5, 3, 4, 5, 1), (2, 20, 24, 56, 12, 1), (1, 23, 33, 9, 11, 1), (1, 24, 44, 16, 10, 1), (1, 96, 31, 8, 8, 1), (4, 22, 100, 64, 64, 1), (1, 8, 40, 30, 41, 3),
                                         (3, 14, 65, 33, 31, 3), (1, 3, 64, 65, 66, 5)])
@pytest.mark.parametrize("layout", ["nhwc", "nchw"])
@pytest.mark.parametrize("shift", [0, 1])
def test_conv_shallow_reduction(n, c, k, h, w, r, layout, shift):
    """The whole depth at once: one chain below 24 products, else sums of eight, of four of them and of those. Depths that are no eights,
    pixels and channels that are no tiles, operands off the 16-byte boundary."""
    g = torch.Generator(device="cuda").manual_seed(c * 131 + r)
    x, f = torch.randn(n, c, h, w, device="cuda", generator=g), torch.randn(k, c, r, r, device="cuda", generator=g)
    place = lambda t: torch.zeros(t.numel() + shift, device="cuda")[shift:].copy_((t.permute(0, 2, 3, 1) if layout == "nhwc" else t).reshape(-1))
    y = torch.full((n * k * h * w,), float("nan"), device="cuda")
    doc = graphs.c1_conv(layout, n, c, h, w, k, r, r // 2)
    run(doc, {1: place(x), 2: place(f)}, {3: y})
    y = y.view(n, h, w, k).permute(0, 3, 1, 2) if layout == "nhwc" else y.view(n, k, h, w)
    conv = lambda a, b: torch.nn.functional.conv2d(a.double().cpu(), b.double().cpu(), padding=r // 2)
    assert torch.all((y.double().cpu() - conv(x, f)).abs() <= max(c * r * r * 2.0 ** -24, pieces_bound(c * r * r)) * conv(x.abs(), f.abs()))


@pytest.mark.parametrize("n,c,k,h,w,r,stride,dilation,reverse", [(1, 5, 3, 4, 5, 1, 1, 1, False), (2, 20, 24, 28, 12, 1, 1, 1, False), (1, 5, 33, 19, 21, 3, 2, 1, False), (1, 7, 40, 17, 13, 3, 1, 2, True), (3, 13, 65, 40, 41, 3, 1, 1, False),
                                                                 (2, 8, 43, 87, 56, 1, 1, 1, False), (4, 3, 100, 96, 97, 3, 1, 1, False), (9, 3, 7, 80, 83, 3, 1, 1, True)])
@pytest.mark.parametrize("layout", ["nhwc", "nchw"])
@pytest.mark.parametrize("io", ["FLOAT", "HALF", "BFLOAT16"])
def test_conv_shallow_fused_and_in_sixteen_bits(n, c, k, h, w, r, stride, dilation, reverse, layout, io):
    """Bias, ReLU and a residual behind it, every element type, tiles of 32 and of 64 (the last but one), of 32 for few channels (the last).
    Products of 16-bit values are exact in f32; C of them are added up in f32 and the operands behind, and Y is rounded once."""
    dtype, rounding = {"FLOAT": (torch.float32, 2.0 ** -24), "HALF": (torch.float16, 2.0 ** -11), "BFLOAT16": (torch.bfloat16, 2.0 ** -8)}[io]
    g = torch.Generator(device="cuda").manual_seed(c * 131 + k)
    pad, strides = dilation * (r // 2), graphs.nhwc if layout == "nhwc" else graphs.contiguous
    p, q = ((size + 2 * pad - dilation * (r - 1) - 1) // stride + 1 for size in (h, w))
    dims = {1: [n, c, h, w], 2: [k, c, r, r], 3: [1, k, 1, 1], 4: [n, k, p, q], 5: [n, k, p, q]}
    tensors = [graphs.tensor(uid, f"t{uid}", d, io, strides(d)) for uid, d in dims.items()] + [graphs.tensor(uid, f"v{uid}", dims[5], "FLOAT", strides(dims[5]), virtual=True) for uid in (6, 7, 8)]
    nodes = [graphs.conv_node("conv", 1, 2, 6, (pad, pad), stride=(stride, stride), dilation=(dilation, dilation), mode="CONVOLUTION" if reverse else "CROSS_CORRELATION"), graphs.pointwise_node("bias", "ADD", 6, 7, 3),
             graphs.pointwise_node("relu", "RELU_FWD", 7, 8), graphs.pointwise_node("residual", "ADD", 8, 5, 4)]
    values = {uid: torch.randn(dims[uid], device="cuda", generator=g).to(dtype) for uid in (1, 2, 3, 4)}
    place = lambda t: (t.permute(0, 2, 3, 1) if layout == "nhwc" else t).contiguous().reshape(-1)
    y = torch.full((n * k * p * q,), float("nan"), device="cuda", dtype=dtype)
    run(graphs.document("conv", nodes, tensors, io=io), {uid: place(t) for uid, t in values.items()}, {5: y})
    y = (y.view(n, p, q, k).permute(0, 3, 1, 2) if layout == "nhwc" else y.view(n, k, p, q)).double().cpu()
    x, f, bias, residual = (t.double().cpu() for t in values.values())
    f = f.flip(2, 3) if reverse else f
    conv = lambda a, b: torch.nn.functional.conv2d(a, b, padding=pad, stride=stride, dilation=dilation)
    want, weight = torch.relu(conv(x, f) + bias) + residual, conv(x.abs(), f.abs()) + bias.abs() + residual.abs()
    depth = c * r * r
    assert torch.all((y - want).abs() <= rounding * want.abs() + max((depth + 3) * 2.0 ** -24, pieces_bound(depth)) * weight)
