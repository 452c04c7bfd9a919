"""Repeated execution: results follow the data, the pointers, the workspace and the stream of every call, however many sets of pointers
rotate, and a pack that would be refused once it has run still is.
f32 sums of 64 products and three additions: 2^-17 of the magnitudes."""
import threading

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


class Linear:
    """bf16 A [m, k] B [k, n] chained through any number of further square matrices."""
    def __init__(self, m, k, sizes):
        g = torch.Generator(device="cuda").manual_seed(m)
        tensors, nodes, last, width = [graphs.tensor(1, "A", [m, k], "BFLOAT16")], [], 1, k
        self.pack = {1: torch.randn(m, k, device="cuda", generator=g).bfloat16()}
        self.want = self.pack[1].double()
        for i, n in enumerate(sizes):
            weight = (torch.randn(width, n, device="cuda", generator=g) * width ** -0.5).bfloat16()
            tensors += [graphs.tensor(10 + i, f"B{i}", [width, n], "BFLOAT16"), graphs.tensor(20 + i, f"C{i}", [m, n], "BFLOAT16")]
            nodes.append(graphs.matmul_node(f"matmul{i}", last, 10 + i, 20 + i))
            self.pack[10 + i], self.pack[20 + i] = weight, torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
            self.want = (self.want @ weight.double()).bfloat16().double()
            last, width = 20 + i, n
        self.exe = runtime.compile_graph(graphs.document("linear", nodes, tensors, io="BFLOAT16"))
        assert all(step["kernel"] == dfgpu.MATMUL_UMMA_BF16 for step in self.exe.steps())
        self.out = self.pack[last]

    def call(self, stream=None):
        pack = {uid: x.data_ptr() for uid, x in self.pack.items()}
        if stream is None:
            self.exe.execute(pack)
        else:
            self.exe.execute_on(stream.cuda_stream, pack)

    def check(self):
        torch.cuda.synchronize()
        # (values of about 1 rounded to bf16 after each product; a rounding that falls the other way early on moves later ones)
        assert bool(torch.all((self.out.double() - self.want).abs() <= 2.0 ** -5 * (1 + self.want.abs())))


def test_shapes_that_share_a_kernel_and_need_different_shared_memory():
    tall, single = Linear(64, 4096, [4096]), Linear(1, 4096, [4096])   # (222512 and 155952 bytes)
    for _ in range(3):
        tall.call()
    single.call()
    for one in (tall, single, tall):
        one.out.zero_()
        one.call()
        one.check()
    both = Linear(64, 4096, [4096, 192, 4096])
    for _ in range(4):
        both.out.zero_()
        both.call()
        both.check()


def test_shapes_that_share_a_kernel_on_two_threads():
    pairs = [(Linear(64, 4096, [4096]), torch.cuda.Stream()), (Linear(1, 4096, [4096]), torch.cuda.Stream())]
    torch.cuda.synchronize()
    failures = []

    def work(one, stream):
        try:
            for _ in range(300):
                one.call(stream)
        except Exception as error:
            failures.append(error)
    threads = [threading.Thread(target=work, args=pair) for pair in pairs]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert not failures
    for one, _ in pairs:
        one.check()
