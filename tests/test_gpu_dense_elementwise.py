"""POINTWISE on dense tensors with broadcast operands, counts and pointers that fall on no quad, axes stored in another order; the
16-bit activations over their whole range; packed dequantize at block shapes and sizes that fill no unit. Compared with torch.

Tolerances: additions and products of stored values are rounded once (exact match); 16-bit activations are within one step
of the correctly rounded value (2^-7 relative for bf16, 2^-10 for f16) plus 3e-7 absolute where the formula cancels (the
f32 reference formulas carry as much); dequantized values are exact."""
import math

import pytest

from deepforge_b200 import dfgpu, graphs, runtime

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TORCH = {"FLOAT": torch.float32, "BFLOAT16": torch.bfloat16, "HALF": torch.float16}


def execute(doc, pack):
    exe = runtime.compile_graph(doc)
    exe.execute({uid: x.data_ptr() for uid, x in pack.items()})
    torch.cuda.synchronize()
    assert dfgpu.device_status() == 0


@pytest.mark.parametrize("io", ["FLOAT", "BFLOAT16", "HALF"])
@pytest.mark.parametrize("dims,b_dims", [([37, 129], [1, 129]), ([64, 256], [1, 256]), ([64, 256], [256]), ([33, 40], [33, 1]), ([5, 7], [1, 1]), ([1, 3], [1, 3]), ([9, 4, 5], [1, 4, 5]),
                                         ([9, 4, 5], [9, 1, 1]), ([9, 4, 5], [9, 4, 1]), ([9, 4, 5], [9, 1, 5]), ([3, 4099], [3, 4099]), ([1000, 1023], [1, 1023])])
@pytest.mark.parametrize("offset", [0, 1])
def test_broadcast_counts_and_pointers(io, dims, b_dims, offset):
    g = torch.Generator(device="cuda").manual_seed(len(dims) + dims[-1])
    values = lambda d: torch.randn(math.prod(d) + offset, device="cuda", generator=g).to(TORCH[io])[offset:]
    a, b, out = values(dims), values(b_dims), torch.full((math.prod(dims) + 8 + offset,), 7.0, device="cuda").to(TORCH[io])[offset:]
    tensors = [graphs.tensor(1, "A", dims, io), graphs.tensor(2, "B", b_dims, io), graphs.tensor(3, "O", dims, io)]
    execute(graphs.document("dense", [graphs.pointwise_node("add", "ADD", 1, 3, 2)], tensors, io=io), {1: a, 2: b, 3: out})
    want = (a.view(dims).float() + b.view(b_dims).float()).to(TORCH[io])
    assert torch.equal(out[:math.prod(dims)].view(dims), want) and bool(torch.all(out[math.prod(dims):] == 7.0))


def test_channels_last_bias_and_first_operand_broadcast():
    n, c, h, w = 2, 24, 5, 7
    g = torch.Generator(device="cuda").manual_seed(1)
    x, bias = torch.randn(n, h, w, c, device="cuda", generator=g), torch.randn(c, device="cuda", generator=g)
    out = torch.empty_like(x)
    strides = graphs.nhwc([n, c, h, w])
    tensors = [graphs.tensor(1, "X", [n, c, h, w], "FLOAT", strides), graphs.tensor(2, "bias", [1, c, 1, 1], "FLOAT", [c, 1, c, c]), graphs.tensor(3, "O", [n, c, h, w], "FLOAT", strides)]
    execute(graphs.document("dense", [graphs.pointwise_node("sub", "SUB", 2, 3, 1)], tensors), {1: x, 2: bias, 3: out})
    assert torch.equal(out, bias - x)


FORWARD = {"EXP": torch.exp, "SIGMOID_FWD": torch.sigmoid, "TANH_FWD": torch.tanh, "SWISH_FWD": torch.nn.functional.silu, "GELU_FWD": torch.nn.functional.gelu,
           "GELU_APPROX_TANH_FWD": lambda u: torch.nn.functional.gelu(u, approximate="tanh")}


@pytest.mark.parametrize("io", ["BFLOAT16", "HALF"])
@pytest.mark.parametrize("mode", ["EXP", "SIGMOID_FWD", "TANH_FWD", "SWISH_FWD", "GELU_FWD", "GELU_APPROX_TANH_FWD", "SIGMOID_BWD", "TANH_BWD", "SWISH_BWD", "GELU_BWD", "GELU_APPROX_TANH_BWD"])
def test_sixteen_bit_activations_over_their_range(io, mode):
    # every finite 16-bit value up to 80 in magnitude, odd in number
    bits = torch.arange(65536, device="cuda", dtype=torch.int32).to(torch.uint16).view(TORCH[io])
    u = bits[torch.isfinite(bits) & (bits.abs() <= 80)].contiguous()
    u = torch.cat([u, u[:1]])[: u.numel() // 2 * 2 - 1].contiguous()
    out = torch.empty_like(u)
    backward = mode.endswith("_BWD")
    tensors = [graphs.tensor(1, "U", [u.numel()], io), graphs.tensor(3, "O", [u.numel()], io)]
    pack = {1: u, 3: out}
    if backward:
        grad = torch.full_like(u, 1.5)
        tensors.append(graphs.tensor(2, "G", [u.numel()], io))
        pack[2] = grad
        node = graphs.pointwise_node("p", mode, 2, 3, 1, swish_beta=1.0)
        leaf = u.double().requires_grad_()
        FORWARD[mode.replace("_BWD", "_FWD")](leaf).backward(grad.double())
        want = leaf.grad
    else:
        node = graphs.pointwise_node("p", mode, 1, 3, swish_beta=1.0)
        want = FORWARD[mode](u.double())
    execute(graphs.document("activation", [node], tensors, io=io), pack)
    step, top = (2.0 ** -7, 3.4e38) if io == "BFLOAT16" else (2.0 ** -10, 65504.0)
    inside = want.abs() < top * (1 - step)
    error = (out.double() - want).abs()
    # f16 results below 2^-14 are subnormal: steps of 2^-24
    bound = step * want.abs() + 3e-7 * (1 + u.double().abs()) + (2.0 ** -24 if io == "HALF" else 0.0)
    assert bool(torch.all(error[inside] <= bound[inside])), (float(u[inside][(error - bound)[inside].argmax()]), float((error / bound)[inside].max()))
    assert bool(torch.all(torch.isinf(out[want >= top * (1 + step)])))


@pytest.mark.parametrize("io", ["FLOAT", "BFLOAT16", "HALF"])
@pytest.mark.parametrize("rows,cols,blocks", [(32, 16, [1, 16]), (3, 48, [1, 16]), (64, 4112, [32, 1]), (96, 32, [1, 32]), (33, 8192, [1, 32]), (64, 48, [2, 4]), (60, 240, [3, 5]), (1, 16, [1, 1])])
@pytest.mark.parametrize("offset", [0, 4])
def test_dequantize(io, rows, cols, blocks, offset):
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    codes = torch.randint(0, 256, (rows * cols,), device="cuda", generator=g, dtype=torch.int32).to(torch.uint8)
    scale_dims = [rows // blocks[0], cols // blocks[1]]
    scales = torch.randint(100, 140, (math.prod(scale_dims) + offset,), device="cuda", generator=g, dtype=torch.int32).to(torch.uint8)[offset:]
    out = torch.empty(rows * cols, device="cuda", dtype=TORCH[io])
    tensors = [graphs.tensor(1, "Y", [rows, cols], io), graphs.tensor(2, "codes", [rows, cols], "FP8_E4M3"), graphs.tensor(3, "scale", scale_dims, "FP8_E8M0")]
    execute(graphs.document("dequantize", [graphs.dequantize_node("d", 2, 3, 1, blocks)], tensors, io=io), {1: out, 2: codes, 3: scales})
    factor = torch.pow(2.0, scales.double() - 127).view(scale_dims).repeat_interleave(blocks[0], 0).repeat_interleave(blocks[1], 1)
    want = (codes.view(torch.float8_e4m3fn).double().view(rows, cols) * factor).to(TORCH[io])
    assert torch.equal(torch.isnan(out.view(rows, cols)), torch.isnan(want))
    assert torch.equal(out.view(rows, cols).nan_to_num(0.0, 1e30, -1e30), want.nan_to_num(0.0, 1e30, -1e30))
