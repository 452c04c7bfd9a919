"""Repeated execution: an Executable keeps the launches of its last few sets of pointers. Results follow the data, the pointers, the
workspace and the stream of every call, also when more sets rotate than are kept, and a pack that would be refused still is.
f32 sums of 64 products and three additions: 2^-17 of the magnitudes."""
import pytest

from deepforge_b200 import dfgpu, graphs, runtime

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
M, K, N = 40, 64, 36


def compiled():
    tensors = [graphs.tensor(1, "A", [M, K]), graphs.tensor(2, "B", [K, N]), graphs.tensor(3, "bias", [1, N]), graphs.tensor(4, "C", [M, N]),
               graphs.tensor(5, "p", [M, N], virtual=True), graphs.tensor(6, "q", [M, N], virtual=True)]
    nodes = [graphs.matmul_node("matmul", 1, 2, 5), graphs.pointwise_node("bias", "ADD", 5, 6, 3), graphs.pointwise_node("gelu", "TANH_FWD", 6, 4)]
    return runtime.compile_graph(graphs.document("recorded", nodes, tensors))


class Set:
    def __init__(self, exe):
        self.t = {1: torch.empty(M, K, device="cuda"), 2: torch.empty(K, N, device="cuda"), 3: torch.empty(1, N, device="cuda"), 4: torch.empty(M, N, device="cuda")}
        self.workspace = torch.empty(max(exe.workspace_size, 1), dtype=torch.uint8, device="cuda")

    def call(self, exe):
        for uid in (1, 2, 3):
            self.t[uid].normal_()
        self.t[4].fill_(float("nan"))
        exe.execute({uid: x.data_ptr() for uid, x in self.t.items()}, self.workspace.data_ptr())

    def check(self):
        a, b, bias = (self.t[uid].double() for uid in (1, 2, 3))
        bound = 2.0 ** -17 * (a.abs() @ b.abs() + bias.abs()) + 2.0 ** -20
        assert bool(torch.all((self.t[4].double() - torch.tanh(a @ b + bias)).abs() <= bound))


@pytest.mark.parametrize("count", [1, 4, 5, 9])
def test_rotating_pointers(count):
    exe = compiled()
    sets = [Set(exe) for _ in range(count)]
    for i in range(4 * count):
        sets[i % count].call(exe)
        sets[i % count].check()
    sets[0].workspace, old = torch.empty_like(sets[0].workspace), sets[0].workspace   # (the old one stays allocated, its contents are no longer used)
    sets[0].call(exe)
    old.fill_(0xFF)
    sets[0].check()
    assert dfgpu.device_status() == 0


def test_other_streams_and_refusals():
    exe = compiled()
    one = Set(exe)
    one.call(exe)
    for _ in range(3):
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            exe.set_stream(stream.cuda_stream)
            one.call(exe)
        stream.synchronize()
        one.check()
    exe.set_stream(None)
    one.call(exe)
    one.check()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()   # captured, not issued
    exe.set_stream(stream.cuda_stream)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        exe.execute({uid: x.data_ptr() for uid, x in one.t.items()}, one.workspace.data_ptr())
    one.t[1].normal_()
    graph.replay()
    torch.cuda.synchronize()
    one.check()
    exe.set_stream(None)
    pack = {uid: x.data_ptr() for uid, x in one.t.items()}
    for broken in ({**pack, 4: 0}, {uid: p for uid, p in pack.items() if uid != 2}, {**pack, 1: pack[1] + 1}):
        with pytest.raises(Exception):
            exe.execute(broken, one.workspace.data_ptr())
    exe.execute(pack, one.workspace.data_ptr())
    torch.cuda.synchronize()
    one.check()
