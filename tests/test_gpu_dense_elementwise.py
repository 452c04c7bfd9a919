"""POINTWISE on dense tensors with broadcast operands, counts and pointers that fall on no quad, axes stored in another order; the
16-bit activations over their whole range; packed dequantize at block shapes and sizes that fill no unit. Compared with torch.

Tolerances: additions and products of stored values are rounded once (exact match); 16-bit activations are within 0.52 steps of
the true value (half a step of rounding, and f32 errors of a few 2^-23 of it, 2^-17 where an exponent of up to 90 is rounded
before it is used), plus 2^-21 absolute for the derivatives that go through zero, where terms of size one cancel; dequantized
values are exact."""
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


@pytest.mark.parametrize("io", ["FLOAT", "BFLOAT16", "HALF"])
@pytest.mark.parametrize("dims,b_dims", [([700, 24], [1, 24]), ([700, 28], [1, 28]), ([700, 24], [700, 1]), ([700, 28], [700, 1]), ([512, 24], [1, 1]), ([2400, 4104], [1, 4104])])
@pytest.mark.parametrize("offsets", [(0, 0, 0), (4, 0, 0), (0, 4, 0), (0, 0, 4)])
def test_eights_fours_and_singles(io, dims, b_dims, offsets):
    """Runs of whole eights and of a four more, pointers on eight values and on four, a last tile that is not full, several tiles a CTA."""
    g = torch.Generator(device="cuda").manual_seed(dims[-1])
    a, b = (torch.randn(math.prod(d) + o, device="cuda", generator=g).to(TORCH[io])[o:] for d, o in zip((dims, b_dims), offsets))
    out = torch.full((math.prod(dims) + 8 + offsets[2],), 7.0, device="cuda").to(TORCH[io])[offsets[2]:]
    tensors = [graphs.tensor(1, "A", dims, io), graphs.tensor(2, "B", b_dims, io), graphs.tensor(3, "O", dims, io)]
    execute(graphs.document("dense", [graphs.pointwise_node("sub", "SUB", 1, 3, 2)], tensors, io=io), {1: a, 2: b, 3: out})
    want = (a.view(dims).float() - b.view(b_dims).float()).to(TORCH[io])
    assert torch.equal(out[:math.prod(dims)].view(dims), want) and bool(torch.all(out[math.prod(dims):] == 7.0))


@pytest.mark.parametrize("io", ["HALF", "BFLOAT16"])
@pytest.mark.parametrize("mode", ["SUB", "RELU_FWD"])
@pytest.mark.parametrize("over", [0, 8, 12, 4096, 4100])
def test_where_tiles_are_no_longer_walked(io, mode, over):
    """32 tiles of 4096 16-bit values per SM are walked, a tile more is not: whole eights and a four more, a last tile that is full or not."""
    count = torch.cuda.get_device_properties(0).multi_processor_count * 32 * 4096 + over
    rows = next(r for r in range(5, 0, -1) if count % (4 * r) == 0)
    dims = [rows, count // rows]
    g = torch.Generator(device="cuda").manual_seed(over)
    a, b = (torch.randn(n, device="cuda", generator=g).to(TORCH[io]) for n in (count, dims[1]))
    out = torch.full((count + 8,), 7.0, device="cuda").to(TORCH[io])
    binary = mode == "SUB"
    tensors = [graphs.tensor(1, "A", dims, io), graphs.tensor(3, "O", dims, io)] + ([graphs.tensor(2, "B", [1, dims[1]], io)] if binary else [])
    buffers = {1: a, 3: out, **({2: b} if binary else {})}
    execute(graphs.document("dense", [graphs.pointwise_node("node", mode, 1, 3, 2 if binary else None)], tensors, io=io), buffers)
    want = (a.view(dims).float() - b.view(1, -1).float()).to(TORCH[io]) if binary else torch.relu(a).view(dims)
    assert torch.equal(out[:count].view(dims), want) and bool(torch.all(out[count:] == 7.0))


def test_channels_last_bias_and_first_operand_broadcast():
    n, c, h, w = 2, 24, 5, 7
    g = torch.Generator(device="cuda").manual_seed(1)
    x, bias = torch.randn(n, h, w, c, device="cuda", generator=g), torch.randn(c, device="cuda", generator=g)
    out = torch.empty_like(x)
    strides = graphs.nhwc([n, c, h, w])
    tensors = [graphs.tensor(1, "X", [n, c, h, w], "FLOAT", strides), graphs.tensor(2, "bias", [1, c, 1, 1], "FLOAT", [c, 1, c, c]), graphs.tensor(3, "O", [n, c, h, w], "FLOAT", strides)]
    execute(graphs.document("dense", [graphs.pointwise_node("sub", "SUB", 2, 3, 1)], tensors), {1: x, 2: bias, 3: out})
    assert torch.equal(out, bias - x)


CANCELLING = ("SWISH_BWD", "GELU_BWD", "GELU_APPROX_TANH_BWD")
SIGMOID = torch.sigmoid
INNER = lambda u: math.sqrt(2 / math.pi) * (u + 0.044715 * u ** 3)
TAIL = lambda u: 0.5 * torch.special.erfc(-u * 0.5 ** 0.5)
# in f64, in forms that do not cancel in the tails
VALUE = {"EXP": torch.exp, "SIGMOID_FWD": SIGMOID, "TANH_FWD": torch.tanh, "SWISH_FWD": lambda u: u * SIGMOID(u), "GELU_FWD": lambda u: u * TAIL(u),
         "GELU_APPROX_TANH_FWD": lambda u: u * SIGMOID(2 * INNER(u)), "SIGMOID_BWD": lambda u: SIGMOID(u) * SIGMOID(-u), "TANH_BWD": lambda u: 4 * SIGMOID(2 * u) * SIGMOID(-2 * u),
         "SWISH_BWD": lambda u: SIGMOID(u) * (1 + u * SIGMOID(-u)), "GELU_BWD": lambda u: TAIL(u) + u * torch.exp(-0.5 * u * u) / math.sqrt(2 * math.pi),
         "GELU_APPROX_TANH_BWD": lambda u: SIGMOID(2 * INNER(u)) * (1 + u * 2 * math.sqrt(2 / math.pi) * (1 + 3 * 0.044715 * u * u) * SIGMOID(-2 * INNER(u)))}


@pytest.mark.parametrize("io", ["BFLOAT16", "HALF"])
@pytest.mark.parametrize("mode", list(VALUE))
def test_sixteen_bit_activations_over_their_range(io, mode):
    # every finite 16-bit value (where the tanh approximation's derivative has a finite square), odd in number
    bits = torch.arange(65536, device="cuda", dtype=torch.int32).to(torch.uint16).view(TORCH[io])
    u = bits[torch.isfinite(bits) & ((bits.double().abs() <= 1e18) if mode == "GELU_APPROX_TANH_BWD" else True)].contiguous()
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
    else:
        node = graphs.pointwise_node("p", mode, 1, 3, swish_beta=1.0)
    want = VALUE[mode](u.double()) * (1.5 if backward else 1.0)
    execute(graphs.document("activation", [node], tensors, io=io), pack)
    least, digits, top = (-126, 7, 3.38e38) if io == "BFLOAT16" else (-14, 10, 65504.0)
    step = torch.exp2(torch.floor(torch.log2(want.abs().clamp_min(1e-300))).clamp_min(least) - digits)   # of the result, subnormal ones too
    inside = want.abs() < top * (1 - 2.0 ** -digits)
    error = (out.double() - want).abs()
    bound = 0.52 * step + (2.0 ** -21 if mode in CANCELLING else 0.0)
    assert bool(torch.all(error[inside] <= bound[inside])), (float(u[inside][(error / bound)[inside].argmax()]), float((error / bound)[inside].max()))
    assert bool(torch.all(torch.isinf(out[want >= top * (1 + 2.0 ** -digits)])))


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


def test_dequantize_in_slices():
    """Blocks of rows that hold more codes than 32-bit indices reach: slices that begin inside a block, under the kernel id that takes them."""
    cols, rows = 1 << 20, 3000
    blocks = [rows, 1]
    p = dfgpu.BsdParams()
    p.x, p.scale, p.y = dfgpu.tensor(dfgpu.E4M3, [rows, cols]), dfgpu.tensor(dfgpu.E8M0, [rows // blocks[0], cols]), dfgpu.tensor(dfgpu.BF16, [rows, cols])
    p.block[0], p.block[1], p.block_count, p.kernel = blocks[0], 1, 2, dfgpu.BSD_PACKED
    assert dfgpu.query("block_scale_dequantize", p).kernel == dfgpu.BSD_PACKED
    g = torch.Generator(device="cuda").manual_seed(1)
    codes = torch.randint(0, 120, (rows, cols), device="cuda", generator=g, dtype=torch.uint8)
    scales = torch.randint(120, 131, (rows // blocks[0], cols), device="cuda", generator=g, dtype=torch.uint8)
    out = torch.empty(rows, cols, device="cuda", dtype=torch.bfloat16)
    dfgpu.block_scale_dequantize(p, codes.data_ptr(), scales.data_ptr(), out.data_ptr())
    torch.cuda.synchronize()
    for first in (0, 2040, 2047, 2048, rows - 8):   # (2047 rows of 2^20 codes are a slice)
        some = slice(first, first + 8)
        want = codes[some].view(torch.float8_e4m3fn).float() * torch.pow(2.0, scales[0].float() - 127)
        assert torch.equal(out[some], want.bfloat16())
