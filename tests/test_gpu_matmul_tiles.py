"""The tensor-core matrix kernel at extents that fill no tile: one row or column past and short of the tile edges, one K block and
remainders of it, each shape of work (two SMs per tile, one SM, clusters that share out K), both layouts of B, every operand
type, fused steps. Compared with an f64 product of the same stored values.

Tolerances: the products of stored values are exact in f32 and are added in f32, so an element is off by at most K 2^-24
sum |a b| before C is rounded once: by half a unit in the last of 8 (bf16), 11 (f16) or 24 (f32) significant bits, that is 2^-8,
2^-11 or 2^-24 relative."""
import numpy as np
import pytest

from deepforge_b200 import dfgpu, graphs, runtime
from test_matmul_shape_cpu import CODES, DIRECT, N_MAJOR_192, SIXTEEN

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TORCH = {"FLOAT": torch.float32, "BFLOAT16": torch.bfloat16, "HALF": torch.float16, "FP8_E4M3": torch.uint8, "FP8_E5M2": torch.uint8, "FP8_E8M0": torch.uint8}
ROUNDING = {"FLOAT": 2.0 ** -24, "BFLOAT16": 2.0 ** -8, "HALF": 2.0 ** -11}
# M, K, N: K and N in 16-byte rows. Single rows; edges of 128 and 256 rows; 64 / 128 / 192 / 256 columns; K of one block, less, more
EXTENTS = [(1, 16, 16), (1, 4096, 96), (7, 144, 272), (16, 4096, 4096), (64, 8192, 512), (127, 128, 112), (128, 4096, 256), (129, 272, 128), (255, 64, 192),
           (257, 1040, 400), (777, 2064, 1552), (1500, 528, 3088), (2049, 256, 2064)]


def run(doc, buffers):
    for t in doc["tensors"].values():
        if not t["is_virtual"] and t["uid"] not in buffers:
            count, dtype = int(np.prod(t["dim"])), TORCH[t["data_type"]]
            buffers[t["uid"]] = torch.full((count,), 0x5A if dtype == torch.uint8 else float("nan"), dtype=dtype, device="cuda")
    exe = runtime.compile_graph(doc)
    workspace = torch.empty(max(exe.workspace_size, 1), dtype=torch.uint8, device="cuda")
    exe.execute({uid: b.data_ptr() for uid, b in buffers.items()}, workspace.data_ptr())
    torch.cuda.synchronize()
    assert dfgpu.device_status() == 0
    return exe


def close(got, a, b, after, out_type, k):
    product, weight = a @ b, a.abs() @ b.abs()
    want = after(product)
    bound = ROUNDING[out_type] * want.abs() + k * 2.0 ** -24 * weight + 1e-30
    assert torch.all((got.double() - want).abs() <= bound), float(((got.double() - want).abs() / bound).max())


@pytest.mark.parametrize("m,n", [(1, 99), (5, 130), (5, 66), (100, 99), (128, 128), (130, 65), (12, 1001)])
@pytest.mark.parametrize("k", [520, 4096])
@pytest.mark.parametrize("first", ["bias", "addend", "f32 bias", "relu"])
def test_sums_over_a_cluster_with_their_first_operand(m, n, k, first):
    """K shared out over a cluster: CTAs without rows of their own, columns that end inside a four, a first fused operand that is fetched
    while the partial tiles meet (16 bits, per column or full, its rows on no boundary) and ones that are not."""
    io = "BFLOAT16"
    g = torch.Generator(device="cuda").manual_seed(m + n)
    full = first == "addend"
    tensors = [graphs.tensor(1, "A", [m, k], io), graphs.tensor(2, "B", [k, n], io, [1, k]), graphs.tensor(3, "X", [m, n] if full else [1, n], "FLOAT" if first == "f32 bias" else io),
               graphs.tensor(4, "C", [m, n], io), graphs.tensor(5, "p", [m, n], virtual=True), graphs.tensor(6, "q", [m, n], virtual=True)]
    add, relu = (lambda i, o: graphs.pointwise_node("add", "ADD", i, o, 3)), (lambda i, o: graphs.pointwise_node("relu", "RELU_FWD", i, o))
    nodes = [graphs.matmul_node("matmul", 1, 2, 5)] + ([relu(5, 6), add(6, 4)] if first == "relu" else [add(5, 6), relu(6, 4)])
    buffers = {uid: torch.randn(count, device="cuda", generator=g).to(torch.float32 if uid == 3 and first == "f32 bias" else TORCH[io]) for uid, count in ((1, m * k), (2, k * n), (3, m * n if full else n))}
    run(graphs.document("cluster", nodes, tensors, io=io), buffers)
    x = buffers[3].double().view(m if full else 1, n)
    close(buffers[4].view(m, n), buffers[1].view(m, k).double(), buffers[2].view(n, k).t().double(), (lambda p: torch.relu(p) + x) if first == "relu" else (lambda p: torch.relu(p + x)), io, k)


@pytest.mark.parametrize("m,k,n", [(1, 4096, 512), (7, 2048, 96), (16, 1024, 260), (100, 4096, 144), (128, 2048, 64)])
@pytest.mark.parametrize("io", ["FLOAT", "BFLOAT16"])
@pytest.mark.parametrize("b_k_major", [False, True])
@pytest.mark.parametrize("rare", ["none", "some", "all"])
def test_both_ways_to_leave_a_cluster(m, k, n, io, b_k_major, rare):
    """The CTAs that share out K part by one of two arrivals, by whether a sum is 1.5 x 2^-100: none, every second column, all. Products
    of small whole numbers and of powers of two are exact."""
    g = torch.Generator(device="cuda").manual_seed(k + n)
    a, b = (torch.randint(-2, 3, shape, device="cuda", generator=g).float() for shape in ((m, k), (n, k)))
    a[:, 0], b[:, 0] = 1.5 * 2.0 ** -50, 0.0
    columns = slice(0, 0) if rare == "none" else (slice(0, n, 2) if rare == "some" else slice(0, n))
    b[columns] = 0.0
    b[columns, 0] = 2.0 ** -50
    tensors = [graphs.tensor(1, "A", [m, k], io), graphs.tensor(2, "B", [k, n], io, [1, k] if b_k_major else [n, 1]), graphs.tensor(3, "C", [m, n], io)]
    buffers = {1: a.to(TORCH[io]), 2: (b if b_k_major else b.t().contiguous()).to(TORCH[io])}
    run(graphs.document("leave", [graphs.matmul_node("matmul", 1, 2, 3)], tensors, io=io), buffers)
    assert torch.equal(buffers[3].view(m, n), (a.double() @ b.double().t()).to(TORCH[io]))


@pytest.mark.parametrize("m,k,n", EXTENTS)
@pytest.mark.parametrize("io", ["BFLOAT16", "HALF"])
@pytest.mark.parametrize("b_k_major", [False, True])
def test_sixteen_bit_operands(m, k, n, io, b_k_major):
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n)
    tensors = [graphs.tensor(1, "A", [m, k], io), graphs.tensor(2, "B", [k, n], io, [1, k] if b_k_major else [n, 1]), graphs.tensor(3, "bias", [1, n], io),
               graphs.tensor(7, "addend", [m, n], io), graphs.tensor(4, "C", [m, n], io), graphs.tensor(5, "p", [m, n], virtual=True), graphs.tensor(6, "q", [m, n], virtual=True),
               graphs.tensor(8, "r", [m, n], virtual=True)]
    nodes = [graphs.matmul_node("matmul", 1, 2, 5), graphs.pointwise_node("bias", "ADD", 5, 6, 3), graphs.pointwise_node("relu", "RELU_FWD", 6, 8), graphs.pointwise_node("add", "ADD", 8, 4, 7)]
    buffers = {uid: torch.randn(count, device="cuda", generator=g).to(TORCH[io]) for uid, count in ((1, m * k), (2, k * n), (3, n), (7, m * n))}
    exe = run(graphs.document("tiles", nodes, tensors, io=io), buffers)
    assert exe.launch_count == 1
    a, b = buffers[1].view(m, k).double(), (buffers[2].view(n, k).t() if b_k_major else buffers[2].view(k, n)).double()
    close(buffers[4].view(m, n), a, b, lambda p: torch.relu(p + buffers[3].double()) + buffers[7].view(m, n).double(), io, k)


@pytest.mark.parametrize("m,k,n", EXTENTS)
@pytest.mark.parametrize("c_type,b_k_major", [("BFLOAT16", True), ("FLOAT", False), ("HALF", True)])
def test_fp8_codes(m, k, n, c_type, b_k_major):
    g = torch.Generator(device="cuda").manual_seed(m * 11 + n)
    codes = {uid: (torch.randn(count, device="cuda", generator=g) * 16).to(torch.float8_e4m3fn) for uid, count in ((21, m * k), (22, k * n))}
    scalars = {23: 0.5, 24: 0.25, 25: 0.125}
    buffers = {uid: c.view(torch.uint8) for uid, c in codes.items()}
    buffers.update({uid: torch.full((1,), v, device="cuda") for uid, v in scalars.items()})
    run(graphs.matmul_fp8(m, k, n, c_type, batch=(), b_k_major=b_k_major), buffers)
    a, b = codes[21].double().view(m, k), (codes[22].double().view(n, k).t() if b_k_major else codes[22].double().view(k, n))
    if c_type == "HALF":  # (values past the largest f16 become infinities on both sides)
        assert float((a @ b).abs().max()) * (0.5 * 0.25 * 0.125) < 65504
    close(buffers[26].view(m, n), a, b, lambda p: p * (0.5 * 0.25 * 0.125), c_type, k)
    top = float((a @ b).abs().max()) * 0.125
    assert abs(float(buffers[27][0]) - top) <= k * 2.0 ** -24 * float((a.abs() @ b.abs()).max())


@pytest.mark.parametrize("m,k,n", N_MAJOR_192[SIXTEEN])
@pytest.mark.parametrize("io", ["BFLOAT16", "HALF"])
def test_sixteen_bit_columns_of_one_and_a_half_boxes(m, k, n, io):
    """B [K, N] in shares of 96 columns: a box of 64 and half of the next, the other half not multiplied."""
    g = torch.Generator(device="cuda").manual_seed(n)
    doc = graphs.document("tiles", [graphs.matmul_node("matmul", 1, 2, 5), graphs.pointwise_node("bias", "ADD", 5, 4, 3)], [graphs.tensor(1, "A", [m, k], io), graphs.tensor(2, "B", [k, n], io), graphs.tensor(3, "bias", [1, n], io),
                          graphs.tensor(4, "C", [m, n], io), graphs.tensor(5, "p", [m, n], virtual=True)], io=io)
    buffers = {uid: torch.randn(count, device="cuda", generator=g).to(TORCH[io]) for uid, count in ((1, m * k), (2, k * n), (3, n))}
    assert [s["kernel"] for s in run(doc, buffers).steps()] == [dfgpu.MATMUL_UMMA_BF16]
    close(buffers[4].view(m, n), buffers[1].view(m, k).double(), buffers[2].view(k, n).double(), lambda p: p + buffers[3].double(), io, k)


@pytest.mark.parametrize("m,k,n", N_MAJOR_192[CODES])
@pytest.mark.parametrize("c_type", ["BFLOAT16", "HALF"])
def test_fp8_columns_of_three_quarters_of_a_box(m, k, n, c_type):
    g = torch.Generator(device="cuda").manual_seed(n)
    codes = {uid: (torch.randn(count, device="cuda", generator=g) * 16).to(torch.float8_e4m3fn) for uid, count in ((21, m * k), (22, k * n))}
    buffers = {uid: c.view(torch.uint8) for uid, c in codes.items()}
    buffers.update({uid: torch.full((1,), v, device="cuda") for uid, v in ((23, 0.5), (24, 0.25), (25, 0.125))})
    run(graphs.matmul_fp8(m, k, n, c_type, batch=()), buffers)
    a, b = codes[21].double().view(m, k), codes[22].double().view(k, n)
    assert float((a @ b).abs().max()) * (0.5 * 0.25 * 0.125) < 65504
    close(buffers[26].view(m, n), a, b, lambda p: p * (0.5 * 0.25 * 0.125), c_type, k)
    assert abs(float(buffers[27][0]) - float((a @ b).abs().max()) * 0.125) <= k * 2.0 ** -24 * float((a.abs() @ b.abs()).max())


@pytest.mark.parametrize("m,k,n", DIRECT[SIXTEEN] + [(4097, 64, 136)])
@pytest.mark.parametrize("io", ["BFLOAT16", "HALF"])
@pytest.mark.parametrize("pad", [1, 5])
def test_rows_of_c_off_the_boundaries(m, k, n, io, pad):
    """Stored element by element, by the owners of a cluster's rows and by single CTAs; nothing between the rows is touched."""
    g = torch.Generator(device="cuda").manual_seed(n)
    doc = graphs.document("tiles", [graphs.matmul_node("matmul", 1, 2, 5), graphs.pointwise_node("relu", "RELU_FWD", 5, 4)], [graphs.tensor(1, "A", [m, k], io), graphs.tensor(2, "B", [k, n], io, [1, k]), graphs.tensor(4, "C", [m, n], io, [n + pad, 1]),
                          graphs.tensor(5, "p", [m, n], virtual=True)], io=io)
    buffers = {uid: torch.randn(count, device="cuda", generator=g).to(TORCH[io]) for uid, count in ((1, m * k), (2, k * n))}
    buffers[4] = torch.full((m * (n + pad),), 7.0, device="cuda", dtype=TORCH[io])
    assert [s["kernel"] for s in run(doc, buffers).steps()] == [dfgpu.MATMUL_UMMA_BF16]
    c = buffers[4].view(m, n + pad)
    close(c[:, :n], buffers[1].view(m, k).double(), buffers[2].view(n, k).t().double(), torch.relu, io, k)
    assert torch.all(c[:-1, n:] == 7.0)


@pytest.mark.parametrize("m,k,n", DIRECT[CODES] + [(2050, 256, 1040)])
@pytest.mark.parametrize("c_type,code", [("FP8_E5M2", torch.float8_e5m2), ("FP8_E4M3", torch.float8_e4m3fn)])
def test_codes_as_results(m, k, n, c_type, code):
    """Whole numbers up to 2, so that sums are exact and the codes the same to the byte."""
    g = torch.Generator(device="cuda").manual_seed(n)
    codes = {uid: torch.randint(-2, 3, (count,), device="cuda", generator=g).float().to(torch.float8_e4m3fn) for uid, count in ((21, m * k), (22, k * n))}
    buffers = {uid: c.view(torch.uint8) for uid, c in codes.items()}
    buffers.update({uid: torch.full((1,), v, device="cuda") for uid, v in ((23, 0.5), (24, 0.25), (25, 0.5))})
    doc = graphs.matmul_fp8(m, k, n, c_type, batch=(), b_k_major=True)
    run(doc, buffers)
    product = codes[21].float().view(m, k).double() @ codes[22].float().view(n, k).t().double()
    assert float(product.abs().max()) / 16 < 440 and float(buffers[27][0]) == float(product.abs().max()) / 8
    assert torch.equal(buffers[26].view(m, n), (product / 16).float().to(code).view(torch.uint8))


@pytest.mark.parametrize("m,k,n", [(m, (k + 31) // 32 * 32, n) for m, k, n in EXTENTS if n > 64])
def test_block_scaled_codes(m, k, n):
    g = torch.Generator(device="cuda").manual_seed(m * 13 + n)
    buffers = {1: torch.randn(m * k, device="cuda", generator=g).to(torch.bfloat16), 2: torch.randn(k * n, device="cuda", generator=g).to(torch.bfloat16)}
    exe = run(graphs.c3_quantize_matmul(m, k, n), buffers)
    assert [s["kernel"] for s in exe.steps()][-1] == dfgpu.MATMUL_UMMA_MXF8
    scale = lambda uid: torch.pow(2.0, buffers[uid].double() - 127)
    a = buffers[3].view(torch.float8_e4m3fn).double().view(m, k) * scale(4).view(m, k // 32).repeat_interleave(32, 1)
    b = buffers[5].view(torch.float8_e4m3fn).double().view(k, n) * scale(6).view(k // 32, n).repeat_interleave(32, 0)
    close(buffers[9].view(m, n), a, b, lambda p: p, "BFLOAT16", k)


def test_operands_off_the_sixteen_byte_boundary_fall_back():
    """Extents that are no whole tiles keep the element's alignment: an operand TMA cannot read goes to the CUDA cores."""
    m, k, n = 40, 72, 88
    g = torch.Generator(device="cuda").manual_seed(5)
    doc = graphs.document("tiles", [graphs.matmul_node("matmul", 1, 2, 4)], [graphs.tensor(1, "A", [m, k], "BFLOAT16"), graphs.tensor(2, "B", [k, n], "BFLOAT16"), graphs.tensor(4, "C", [m, n], "BFLOAT16")], io="BFLOAT16")
    a, b = (torch.randn(count + 1, device="cuda", generator=g).to(torch.bfloat16)[1:] for count in (m * k, k * n))
    buffers = {1: a, 2: b}
    run(doc, buffers)
    close(buffers[4].view(m, n), a.view(m, k).double(), b.view(k, n).double(), lambda p: p, "BFLOAT16", k)


@pytest.mark.parametrize("io,c_ld", [("HALF", 128), ("BFLOAT16", 130)])
def test_whole_tiles_off_the_boundary_fall_back(io, c_ld):
    """Whole tiles in HALF, or with rows of C that are no whole 16-byte units, keep the element's alignment as well."""
    m, k, n = 128, 64, 128
    g = torch.Generator(device="cuda").manual_seed(6)
    doc = graphs.document("tiles", [graphs.matmul_node("matmul", 1, 2, 4)], [graphs.tensor(1, "A", [m, k], io), graphs.tensor(2, "B", [k, n], io), graphs.tensor(4, "C", [m, n], io, [c_ld, 1])], io=io)
    a, b = (torch.randn(count + 1, device="cuda", generator=g).to(TORCH[io])[1:] for count in (m * k, k * n))
    buffers = {1: a, 2: b, 4: torch.zeros(m * c_ld, dtype=TORCH[io], device="cuda")}
    run(doc, buffers)
    close(buffers[4].view(m, c_ld)[:, :n], a.view(m, k).double(), b.view(k, n).double(), lambda p: p, io, k)


@pytest.mark.parametrize("m,k,n,c_ld", [(1, 72, 24, 24), (77, 64, 40, 40), (77, 256, 272, 272), (129, 104, 136, 136), (130, 520, 136, 139), (300, 4112, 528, 528), (2050, 264, 1040, 1040), (2050, 8184, 1040, 1040), (4096, 1032, 4104, 4104)])
@pytest.mark.parametrize("io", ["BFLOAT16", "HALF"])
@pytest.mark.parametrize("b_k_major", [False, True])
def test_f32_results_do_not_lose_accuracy_with_depth(m, k, n, c_ld, io, b_k_major):
    """A block of 64 is off by at most four cut-off sums of four ulps (2^-21 of its value), blocks of random sign add up as their values
    do, and every addition of a block rounds the sum so far by 2^-25 in the mean."""
    g = torch.Generator(device="cuda").manual_seed(m + k)
    doc = graphs.document("tiles", [graphs.matmul_node("matmul", 1, 2, 4)], [graphs.tensor(1, "A", [m, k], io), graphs.tensor(2, "B", [k, n], io, [1, k] if b_k_major else [n, 1]), graphs.tensor(4, "C", [m, n], "FLOAT", [c_ld, 1])], io=io)
    a, b = (torch.randn(count, device="cuda", generator=g).to(TORCH[io]) for count in (m * k, k * n))
    buffers = {1: a, 2: b, 4: torch.zeros(m * c_ld, device="cuda")}
    shallow = io == "BFLOAT16" and k < 104   # (the CUDA cores' additions are the more exact)
    assert [s["kernel"] for s in run(doc, buffers).steps()] == [dfgpu.MATMUL_FFMA if shallow else dfgpu.MATMUL_UMMA_BF16]
    b = b.view(n, k).t() if b_k_major else b.view(k, n)
    want = a.view(m, k).double() @ b.double()
    error = (buffers[4].view(m, c_ld)[:, :n].double() - want).norm() / want.norm()
    assert float(error) <= 2.0 ** -21 + 2.0 ** -25 * (k / 64) ** 0.5


@pytest.mark.parametrize("m,k,n,blocks", [(128, 384, 1152, 1), (128, 640, 3840, 3), (128, 896, 3712, 4), (128, 2048, 2688, 6), (128, 3328, 1536, 7)])
@pytest.mark.parametrize("b_k_major", [False, True])
def test_f32_results_of_whole_tiles_keep_their_splits(m, k, n, blocks, b_k_major):
    """An accumulator loses 2^-24 of its value for every block of 64 it takes (sums are cut off toward zero), and adding the splits of K as
    much once more. With `blocks` of them; K in one or two accumulators is two to four times as far off."""
    g = torch.Generator(device="cuda").manual_seed(m + k)
    doc = graphs.document("tiles", [graphs.matmul_node("matmul", 1, 2, 4)], [graphs.tensor(1, "A", [m, k], "BFLOAT16"), graphs.tensor(2, "B", [k, n], "BFLOAT16", [1, k] if b_k_major else [n, 1]), graphs.tensor(4, "C", [m, n], "FLOAT")], io="BFLOAT16")
    a, b = (torch.randn(count, device="cuda", generator=g).to(torch.bfloat16) for count in (m * k, k * n))
    buffers = {1: a, 2: b}
    assert [s["kernel"] for s in run(doc, buffers).steps()] == [dfgpu.MATMUL_UMMA_BF16]
    want = a.view(m, k).double() @ (b.view(n, k).t() if b_k_major else b.view(k, n)).double()
    error = (buffers[4].view(m, n).double() - want).norm() / want.norm()
    assert float(error) <= (blocks + 1) * 2.0 ** -24


@pytest.mark.parametrize("m,k,n", [(1, 32, 80), (77, 288, 272), (300, 544, 528), (129, 4128, 144), (2050, 288, 2064), (1026, 32736, 1040)])
def test_f32_results_of_block_scaled_codes_do_not_lose_accuracy_with_depth(m, k, n):
    """As above with blocks of 128 codes, whose products hold eight significant bits: half the bound of a block."""
    g = torch.Generator(device="cuda").manual_seed(m + k)
    buffers = {1: torch.randn(m * k, device="cuda", generator=g).to(torch.bfloat16), 2: torch.randn(k * n, device="cuda", generator=g).to(torch.bfloat16)}
    exe = run(graphs.c3_quantize_matmul(m, k, n, c_type="FLOAT"), buffers)
    assert [s["kernel"] for s in exe.steps()][-1] == dfgpu.MATMUL_UMMA_MXF8
    scale = lambda uid: torch.pow(2.0, buffers[uid].double() - 127)
    a = buffers[3].view(torch.float8_e4m3fn).double().view(m, k) * scale(4).view(m, k // 32).repeat_interleave(32, 1)
    b = buffers[5].view(torch.float8_e4m3fn).double().view(k, n) * scale(6).view(k // 32, n).repeat_interleave(32, 0)
    want = a @ b
    error = (buffers[9].view(m, n).double() - want).norm() / want.norm()
    assert float(error) <= 2.0 ** -22 + 2.0 ** -25 * (k / 128) ** 0.5


@pytest.mark.parametrize("m,k,n", [(1, 16, 16), (77, 192, 272), (300, 256, 528), (130, 400, 1040), (1030, 640, 1040), (2050, 1040, 1040), (300, 4112, 528)])
@pytest.mark.parametrize("b_k_major", [False, True])
def test_f32_results_of_codes_are_as_exact_as_f32_additions(m, k, n, b_k_major):
    """Against the same values with operands one byte off, which the CUDA cores sum in f32: no further from 64 bits, with 2 % for the
    spread of two sums of squares over a few thousand elements and more."""
    g = torch.Generator(device="cuda").manual_seed(m + k)
    doc = graphs.matmul_fp8(m, k, n, "FLOAT", batch=(), b_k_major=b_k_major)
    a, b = ((torch.randn(count, device="cuda", generator=g) * 16).to(torch.float8_e4m3fn) for count in (m * k, k * n))
    want = a.view(m, k).double() @ (b.view(n, k).t() if b_k_major else b.view(k, n)).double()
    errors = []
    for shift in (0, 1):
        place = lambda x: torch.cat([torch.zeros(shift, dtype=torch.uint8, device="cuda"), x.view(torch.uint8)])[shift:]
        one = lambda: torch.ones(1, device="cuda")
        buffers = {21: place(a), 22: place(b), 23: one(), 24: one(), 25: one()}
        run(doc, buffers)
        errors.append(float((buffers[26].view(m, n).double() - want).norm() / want.norm()))
        assert float(buffers[27]) == float(buffers[26].abs().max())
    assert errors[0] <= 1.02 * errors[1] + (1e-9 if m * n < 4096 else 0.0)


@pytest.mark.parametrize("m,k,n", [(20, 4104, 136), (300, 4160, 520), (1030, 4104, 1040), (2050, 8184, 1040)])
@pytest.mark.parametrize("b_k_major", [False, True])
def test_f32_operands_beyond_the_one_launch_kernel_do_not_lose_accuracy_with_depth(m, k, n, b_k_major):
    """Products are within 2^-23, a sum of eight blocks of 64 is off by at most 32 cut-off sums of four ulps that lean one way (2^-19 at the
    worst, a quarter of that in the mean of a growing sum), and sums of random sign add up as their values do. (One accumulator: 9e-6
    at 2050 x 8184 x 1040.)"""
    g = torch.Generator(device="cuda").manual_seed(m + k)
    doc = graphs.document("tiles", [graphs.matmul_node("matmul", 1, 2, 4)], [graphs.tensor(1, "A", [m, k]), graphs.tensor(2, "B", [k, n], "FLOAT", [1, k] if b_k_major else [n, 1]), graphs.tensor(4, "C", [m, n])])
    a, b = (torch.randn(count, device="cuda", generator=g) for count in (m * k, k * n))
    buffers = {1: a, 2: b}
    exe = run(doc, buffers)
    want = a.view(m, k).double() @ (b.view(n, k).t() if b_k_major else b.view(k, n)).double()
    error = (buffers[4].view(m, n).double() - want).norm() / want.norm()
    if [s["kernel"] for s in exe.steps()] == [dfgpu.MATMUL_UMMA_F32X3]:
        assert float(error) <= 2.0 ** -21 + 2.0 ** -23
    else:
        assert m <= 300 and float(error) <= 2.0 ** -19


@pytest.mark.parametrize("m,k,n", [(77, 64, 88), (130, 192, 216), (300, 136, 600), (2049, 72, 2064)])
@pytest.mark.parametrize("first", ["bias", "full"])
@pytest.mark.parametrize("io,operand,shift", [("BFLOAT16", "BFLOAT16", 0), ("BFLOAT16", "BFLOAT16", 1), ("HALF", "HALF", 0), ("HALF", "FLOAT", 1), ("BFLOAT16", "FLOAT", 0)])
def test_fused_operands_at_the_edges(m, k, n, first, io, operand, shift):
    """Operands in 16-byte units and off them, short rows of them at the last columns, values that ReLU passes through its three ways:
    infinities (x < 0 becomes 0 (x - 0) + 0, so NaN for -inf; above the largest f32 it clips), and the ordinary ones."""
    g = torch.Generator(device="cuda").manual_seed(m + n)
    dims = [1, n] if first == "bias" else [m, n]
    tensors = [graphs.tensor(1, "A", [m, k], io), graphs.tensor(2, "B", [k, n], io), graphs.tensor(3, "x", dims, operand), graphs.tensor(4, "C", [m, n], io), graphs.tensor(5, "p", [m, n], virtual=True), graphs.tensor(6, "q", [m, n], virtual=True)]
    nodes = [graphs.matmul_node("matmul", 1, 2, 5), graphs.pointwise_node("add", "ADD", 5, 6, 3), graphs.pointwise_node("relu", "RELU_FWD", 6, 4)]
    buffers = {uid: torch.randn(count, device="cuda", generator=g).to(TORCH[io]) for uid, count in ((1, m * k), (2, k * n))}
    x = torch.randn(dims, device="cuda", generator=g).to(TORCH[operand])
    x[-1, n - 3], x[-1, 5] = -float("inf"), float("inf")
    buffers[3] = torch.zeros(x.numel() + shift, dtype=x.dtype, device="cuda")[shift:]
    buffers[3].copy_(x.reshape(-1))
    exe = run(graphs.document("tiles", nodes, tensors, io=io), buffers)
    assert exe.launch_count == 1
    a, b = buffers[1].view(m, k).double(), buffers[2].view(k, n).double()
    got, want = buffers[4].view(m, n).double(), a @ b + x.double()
    bound = ROUNDING[io] * want.abs() + k * 2.0 ** -24 * (a.abs() @ b.abs()) + 1e-30
    assert torch.equal(got.isnan(), want == -float("inf"))
    assert torch.all(got[want == float("inf")] >= torch.finfo(TORCH[io]).max)
    finite = want.isfinite()
    assert torch.all((got - torch.relu(want)).abs()[finite] <= bound[finite])


@pytest.mark.parametrize("lower,upper,negative", [(-0.0, None, -0.0), (0.0, None, 0.0), (0.0, -0.0, 0.0), (-0.0, 2.0, -0.0)])
def test_the_sign_of_a_clipped_zero(lower, upper, negative):
    """Below `lower` ReLU gives lower + 0 (x - lower): a negative zero where the clip is one, and never the other clip's sign."""
    m, k, n = 40, 64, 96
    tensors = [graphs.tensor(1, "A", [m, k], "BFLOAT16"), graphs.tensor(2, "B", [k, n], "BFLOAT16"), graphs.tensor(4, "C", [m, n], "BFLOAT16"), graphs.tensor(5, "p", [m, n], virtual=True)]
    nodes = [graphs.matmul_node("matmul", 1, 2, 5), graphs.pointwise_node("relu", "RELU_FWD", 5, 4, lower=lower, upper=upper)]
    buffers = {1: -torch.ones(m * k, device="cuda", dtype=torch.bfloat16), 2: torch.ones(k * n, device="cuda", dtype=torch.bfloat16)}
    run(graphs.document("tiles", nodes, tensors, io="BFLOAT16"), buffers)
    assert torch.all(buffers[4] == 0) and bool(torch.all(torch.signbit(buffers[4]) == (str(negative)[0] == "-")))
