"""Launches chained behind one another without a synchronisation: a kernel may be set up while the one before it still runs, and
must not read what that one writes before it has ended. Data changes with every pass; results are those of the consumer alone,
run on the finished input."""
import pytest

from deepforge_b200 import dfgpu, graphs, runtime

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TORCH = {"FLOAT": torch.float32, "BFLOAT16": torch.bfloat16, "HALF": torch.float16}
ROWS, COLS = 4096, 2048


def addition(out, dims, io):
    tensors = [graphs.tensor(1, "X", dims, io), graphs.tensor(2, "bias", [1] * (len(dims) - 1) + dims[-1:], io), graphs.tensor(out, "Y", dims, io)]
    return tensors, graphs.pointwise_node("add", "ADD", 1, out, 2)


@pytest.mark.parametrize("io", ["FLOAT", "BFLOAT16", "HALF"])
@pytest.mark.parametrize("axis", [0, 1])
def test_quantize_behind_an_addition(io, axis):
    dims = [ROWS, COLS]
    scale_dims = [size // 32 if i == axis else size for i, size in enumerate(dims)]
    tensors, node = addition(3, dims, io)
    codes = [graphs.tensor(4, "codes", dims, "FP8_E4M3"), graphs.tensor(5, "scale", scale_dims, "FP8_E8M0")]
    quantize = graphs.quantize_node("quantize", 3, 4, 5, 32, axis)
    both = runtime.compile_graph(graphs.document("both", [node, quantize], tensors + codes, io=io))
    alone = runtime.compile_graph(graphs.document("alone", [quantize], tensors[2:] + codes, io=io))
    assert len(both.steps()) == 2
    x, bias, y = torch.empty(dims, device="cuda", dtype=TORCH[io]), torch.empty(COLS, device="cuda", dtype=TORCH[io]), torch.empty(dims, device="cuda", dtype=TORCH[io])
    outs = [[torch.empty(dims, device="cuda", dtype=torch.uint8), torch.empty(scale_dims, device="cuda", dtype=torch.uint8)] for _ in range(2)]
    for i in range(6):
        x.normal_(), bias.normal_(0.0, 4.0 ** i)
        both.execute({1: x.data_ptr(), 2: bias.data_ptr(), 3: y.data_ptr(), 4: outs[0][0].data_ptr(), 5: outs[0][1].data_ptr()})
        torch.cuda.synchronize()
        alone.execute({3: y.data_ptr(), 4: outs[1][0].data_ptr(), 5: outs[1][1].data_ptr()})
        torch.cuda.synchronize()
        assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    assert dfgpu.device_status() == 0


@pytest.mark.parametrize("io,m,k,n", [("BFLOAT16", 700, 512, 1000), ("BFLOAT16", 64, 512, 4096), ("FLOAT", 300, 64, 256)])
def test_residual_written_just_before(io, m, k, n):
    dims = [m, n]
    tensors, node = addition(3, dims, io)
    product = [graphs.tensor(6, "A", [m, k], io), graphs.tensor(7, "B", [k, n], io), graphs.tensor(8, "C", dims, io), graphs.tensor(9, "P", dims, "FLOAT", virtual=True)]
    first = runtime.compile_graph(graphs.document("first", [node], tensors, io=io))
    second = runtime.compile_graph(graphs.document("second", [graphs.matmul_node("matmul", 6, 7, 9), graphs.pointwise_node("residual", "ADD", 9, 8, 3)], product + tensors[2:], io=io))
    assert len(second.steps()) == 1
    make = lambda *d: torch.empty(d, device="cuda", dtype=TORCH[io])
    x, bias, y, a, b, c = make(m, n), make(n), make(m, n), make(m, k), make(k, n), make(m, n)
    workspace = torch.empty(max(second.workspace_size, 1), device="cuda", dtype=torch.uint8)
    a.normal_(), b.normal_()
    for i in range(6):
        x.normal_(), bias.normal_(0.0, 4.0 ** i)
        pack = {6: a.data_ptr(), 7: b.data_ptr(), 8: c.data_ptr(), 3: y.data_ptr()}
        first.execute({1: x.data_ptr(), 2: bias.data_ptr(), 3: y.data_ptr()})
        second.execute(pack, workspace.data_ptr())
        torch.cuda.synchronize()
        chained = c.clone()
        second.execute(pack, workspace.data_ptr())
        torch.cuda.synchronize()
        assert torch.equal(chained, c)
    assert dfgpu.device_status() == 0
