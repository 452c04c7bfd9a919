"""Paged decode: a sequence's chunks meet by their maxima, and what a chunk holds reaches the result even where its weight is zero in
f32: a NaN or an infinity among keys far below the largest score is not lost. Chunks without keys count for nothing."""
import pytest

from deepforge_b200 import dfgpu, graphs, runtime

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def decode(batch, spoil):
    hkv, block, length = 2, 64, 4096
    pages = batch * length // block
    exe = runtime.compile_graph(graphs.c5_paged_decode(batch, 8, hkv, 128, pages, block, length))
    assert exe.steps()[0]["kernel"] == dfgpu.SDPA_PAGED_DECODE_UMMA
    q = torch.full((batch, 8, 1, 128), 4.0, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.zeros(pages, hkv, block, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    v += 1.0
    table = torch.arange(pages, device="cuda", dtype=torch.int32)
    k[:: length // block, :, 5] = 4.0   # one key of each sequence scores 181, the others 0
    spoil(k, v, length // block)
    lengths = torch.tensor([length - 700 * (i % 2) for i in range(batch)], device="cuda", dtype=torch.int32)   # (the last chunks of every second sequence are empty)
    o = torch.zeros_like(q)
    ones = torch.ones(batch, device="cuda", dtype=torch.int32)
    workspace = torch.full((exe.workspace_size,), 255, device="cuda", dtype=torch.uint8)
    exe.execute({uid: x.data_ptr() for uid, x in ((1, q), (2, k), (3, v), (4, o), (5, ones), (6, lengths), (7, table), (8, table))}, workspace.data_ptr())
    torch.cuda.synchronize()
    assert dfgpu.device_status() == 0
    return o


@pytest.mark.parametrize("batch", [1, 64])
def test_far_below_the_maximum(batch):
    def nan_key(k, v, pages):
        k[pages // 2 :: pages, 0, 9, 3] = float("nan")

    def infinite_value(k, v, pages):
        v[pages // 2 :: pages, 0, 9] = float("inf")
    assert torch.equal(decode(batch, lambda *_: None), torch.ones(batch, 8, 1, 128, device="cuda", dtype=torch.bfloat16))
    for spoil in (nan_key, infinite_value):
        o = decode(batch, spoil)   # heads 0-3 read KV head 0
        assert not bool(torch.isfinite(o[:, :4]).any()) and bool(torch.all(o[:, 4:] == 1.0))


@pytest.mark.parametrize("tiles", [1, 2, 7, 8, 9, 31, 32, 33, 65, 128, 129, 200])
def test_any_number_of_chunks(tiles):
    """Chunks of one key tile: the most that are merged eight at once and one more; groups of 32 that are full, one over and one short, and more than the first four. A probability is within
    2^-8 of its value and O is rounded once by 2^-9, with as much again for the exponentials and sums."""
    hq, block, length = 8, 64, 128 * tiles
    pages = length // block
    exe = runtime.compile_graph(graphs.c5_paged_decode(2, hq, 1, 128, 2 * pages, block, length))
    assert exe.steps()[0]["kernel"] == dfgpu.SDPA_PAGED_DECODE_UMMA
    g = torch.Generator(device="cuda").manual_seed(tiles)
    q, k, v = (torch.randn(shape, device="cuda", generator=g).to(torch.bfloat16) for shape in ((2, hq, 1, 128), (2 * pages, 1, block, 128), (2 * pages, 1, block, 128)))
    lengths = torch.tensor([length, max(1, length - 200)], device="cuda", dtype=torch.int32)
    ones, table, o = torch.ones(2, device="cuda", dtype=torch.int32), torch.arange(2 * pages, device="cuda", dtype=torch.int32), torch.zeros_like(q)
    workspace = torch.full((exe.workspace_size,), 255, device="cuda", dtype=torch.uint8)
    exe.execute({uid: x.data_ptr() for uid, x in ((1, q), (2, k), (3, v), (4, o), (5, ones), (6, lengths), (7, table), (8, table))}, workspace.data_ptr())
    torch.cuda.synchronize()
    assert dfgpu.device_status() == 0
    for i, n in enumerate(lengths.tolist()):
        keys, values = (x.view(2, length, 128)[i, :n].double() for x in (k, v))
        p = torch.softmax(q[i, :, 0].double() @ keys.t() * 128 ** -0.5, -1)
        assert bool(torch.all((o[i, :, 0].double() - p @ values).abs() <= 2.0 ** -7 * (p @ values.abs())))
