"""SDPA on the tensor cores at lengths that fill no tile: one row past and short of the 128-row tiles, single rows, more and fewer
keys than queries, grouped heads, padding masks with short and empty sequences (NaN in the padding must not leak), causal or
not, both 16-bit types and head dimensions, strided layouts, a negative scale. Compared with an f64 softmax of the stored values.

Tolerances of check(): a probability within u of its value (u = 2^-8 for bf16, 2^-11 for f16, relative) and exponentials within
2^-13, so O is off by at most (u + 2^-12) sum p |v| before it is rounded once by u; subnormal f16 probabilities (up to 2^-24 of
the largest) add 2^-24 sum |v|. Stats carry the exponentials' error and f32 scores. `fine` is what forms that are not whole bf16
tiles of 128 channels promise: probabilities of 16 bits or more (2^-17), exponentials within 2^-22 and scores whose f32 sums over 128
channels are off by at most 2^-20 sum |q k| (below 2^-16 here), 2^-14 sum p |v| in all, and Stats within 2^-16 (both times `amplify`, the
factor by which Q and so the scores' errors are larger)."""
import pytest

from deepforge_b200 import dfgpu, graphs, runtime

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TORCH = {"BFLOAT16": torch.bfloat16, "HALF": torch.float16}
ROUNDING = {"BFLOAT16": 2.0 ** -8, "HALF": 2.0 ** -11}


def attention(q, k, v, scale, causal, len_q=None, len_kv=None):
    b, h, sq, _ = q.shape
    group, skv = h // k.shape[1], k.shape[2]
    k, v = k.double().repeat_interleave(group, 1), v.double().repeat_interleave(group, 1)
    keys, rows = torch.arange(skv, device="cuda"), torch.arange(sq, device="cuda")
    valid = torch.ones(b, 1, sq, skv, dtype=torch.bool, device="cuda")
    if causal:
        valid = valid & (keys[None, :] <= rows[:, None])
    if len_q is not None:
        valid = valid & (keys[None, None, None, :] < len_kv[:, None, None, None]) & (rows[None, None, :, None] < len_q[:, None, None, None])
        v = torch.where(keys[None, None, :, None] < len_kv[:, None, None, None], v, 0.0)
        k = torch.where(keys[None, None, :, None] < len_kv[:, None, None, None], k, 0.0)
        q = torch.where(rows[None, None, :, None] < len_q[:, None, None, None], q, 0.0)
    s = (q.double() @ k.transpose(-1, -2) * scale).masked_fill(~valid, -float("inf"))
    stats = torch.logsumexp(s, -1)
    p = torch.where(valid, torch.exp(s - torch.where(torch.isinf(stats), 0.0, stats)[..., None]), 0.0)
    return p @ v, p @ v.abs(), v.abs().sum(-2, keepdim=True), stats


def check(b, h, hkv, sq, skv, d, io, causal, padding=None, scale=None, strided=False, seed=3, fine=False, amplify=1.0, cold=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    scale = d ** -0.5 if scale is None else scale
    def operand(heads, length):
        x = torch.randn(b, length, heads, d, device="cuda", generator=g).to(TORCH[io])   # [B, S, H, D]
        return x.transpose(1, 2) if strided else x.transpose(1, 2).contiguous()
    q, k, v = operand(h, sq), operand(hkv, skv), operand(hkv, skv)
    q = q * amplify
    o = torch.full_like(q, float("nan"))
    stats = torch.full((b, h, sq), float("nan"), device="cuda")
    tensors = [graphs.tensor(uid, name, list(x.shape), io, list(x.stride())) for uid, name, x in ((1, "Q", q), (2, "K", k), (3, "V", v), (4, "O", o))]
    tensors.append(graphs.tensor(5, "Stats", [b, h, sq, 1], "FLOAT"))
    inputs, pack, len_q, len_kv = {"Q": 1, "K": 2, "V": 3}, {1: q, 2: k, 3: v, 4: o, 5: stats}, None, None
    if padding is not None:
        len_q, len_kv = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in padding)
        for i in range(b):
            q[i, :, len_q[i]:], k[i, :, len_kv[i]:], v[i, :, len_kv[i]:] = float("nan"), float("nan"), float("inf")
        tensors += [graphs.tensor(6, "SEQ_LEN_Q", [b, 1, 1, 1], "INT32"), graphs.tensor(7, "SEQ_LEN_KV", [b, 1, 1, 1], "INT32")]
        inputs.update(SEQ_LEN_Q=6, SEQ_LEN_KV=7)
        pack.update({6: len_q, 7: len_kv})
    node = graphs.sdpa_node("sdpa", inputs, {"O": 4, "Stats": 5}, scale, padding is not None, True, right_bound=0 if causal else None)
    exe = runtime.compile_graph(graphs.document("ragged", [node], tensors, io=io))
    assert exe.steps()[0]["kernel"] == dfgpu.SDPA_UMMA and exe.workspace_size == 0
    exe.execute({uid: x.data_ptr() for uid, x in pack.items()})
    torch.cuda.synchronize()
    assert dfgpu.device_status() == 0
    first, first_stats = o.clone(), stats.clone()
    for i in range(cold):   # (operands out of HBM, at another pace than out of the L2 cache: the same bits)
        torch.full((1 << 26,), float(i), device="cuda")
        o.fill_(float("nan")), stats.fill_(float("nan"))
        exe.execute({uid: x.data_ptr() for uid, x in pack.items()})
        torch.cuda.synchronize()
        assert dfgpu.device_status() == 0 and torch.equal(o, first) and torch.equal(stats, first_stats)
    want, weight, every, want_stats = attention(q, k, v, scale, causal, len_q, len_kv)
    u = ROUNDING[io]
    bound = (amplify * 2.0 ** -14 if fine else u + 2.0 ** -12) * weight + u * want.abs() + (2.0 ** -24 * every if io == "HALF" else 0.0) + 1e-30
    error = (o.double() - want).abs()
    assert bool(torch.all(error <= bound)), float((error / bound).nan_to_num(1e9).max())
    dead = torch.isinf(want_stats)
    assert bool(torch.all(torch.isneginf(stats[dead]))) and bool(torch.all((stats.double() - want_stats)[~dead].abs() <= (amplify * 2.0 ** -16 if fine else 1e-3)))


@pytest.mark.parametrize("io,d", [("BFLOAT16", 128), ("HALF", 128), ("BFLOAT16", 64), ("HALF", 64)])
@pytest.mark.parametrize("b,h,hkv,sq,skv,causal", [(1, 2, 1, 1, 1, False), (2, 4, 2, 19, 301, False), (1, 4, 4, 127, 127, True), (1, 2, 2, 128, 129, False), (2, 2, 1, 129, 129, True),
                                                   (3, 8, 2, 257, 64, False), (1, 3, 1, 300, 1000, True), (2, 40, 8, 641, 641, True), (1, 2, 2, 1000, 130, True)])
def test_any_lengths(io, d, b, h, hkv, sq, skv, causal):
    check(b, h, hkv, sq, skv, d, io, causal)


@pytest.mark.parametrize("io,d", [("BFLOAT16", 128), ("HALF", 64)])
@pytest.mark.parametrize("causal", [False, True])
def test_padded_lengths(io, d, causal):
    check(5, 4, 2, 300, 300, d, io, causal, padding=([300, 130, 1, 0, 257], [300, 130, 1, 200, 0]))
    check(3, 40, 8, 513, 400, d, io, causal, padding=([513, 400, 128], [128, 129, 400]))


def test_strides_scale_and_misalignment():
    check(2, 4, 2, 200, 200, 128, "BFLOAT16", True, strided=True)
    check(1, 2, 2, 200, 300, 64, "HALF", False, scale=-0.2)
    check(1, 2, 1, 150, 260, 128, "BFLOAT16", False, scale=0.0)
    check(1, 2, 2, 384, 384, 128, "BFLOAT16", True, scale=1.5)   # (the running maximum jumps: O is rescaled)


@pytest.mark.parametrize("io", ["BFLOAT16", "HALF"])
@pytest.mark.parametrize("b,h,hkv,sq,skv,causal,scale", [(1, 37, 37, 1000, 1000, True, None), (1, 40, 8, 700, 700, True, 1.5), (2, 60, 12, 256, 1500, False, 1.5), (1, 148, 4, 200, 129, False, None),
                                                         (1, 16, 8, 2171, 2171, True, None), (2, 96, 96, 300, 300, True, 1.5)])
def test_several_items_per_place(io, b, h, hkv, sq, skv, causal, scale):
    """More work items than SMs, which walk them one after another, with maxima that jump."""
    check(b, h, hkv, sq, skv, 128, io, causal, scale=scale)


@pytest.mark.parametrize("io,d", [("BFLOAT16", 128), ("HALF", 128), ("BFLOAT16", 64)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("s,lengths", [(520, [257, 520, 272, 513, 258, 400]), (300, [16, 300, 1, 299, 129, 256]), (1100, [1100, 260, 5, 1025, 641, 130])])
def test_few_keys_in_a_last_tile_out_of_memory(io, d, causal, s, lengths):
    """V rows behind a batch's length (infinities) are cleared when they have come, however late the tiles before them do: a head's keys are
    nobody else's, lists of several query tiles, tiles with one to sixteen keys whose softmax is short."""
    check(6, 30, 30, s, s, d, io, causal, padding=(lengths, lengths), cold=6)


@pytest.mark.parametrize("io,d", [("BFLOAT16", 128), ("HALF", 128), ("BFLOAT16", 64)])
@pytest.mark.parametrize("b,h,sq,skv,causal", [(1, 140, 128, 256, False), (3, 60, 5, 200, False), (2, 148, 128, 128, True), (1, 74, 256, 256, True), (1, 40, 129, 700, False)])
def test_first_key_tiles_out_of_memory(io, d, b, h, sq, skv, causal):
    """The first and second key tile of every CTA, in the ring's slots that held nothing and a K tile before: whole tiles and others, items of one key tile."""
    check(b, h, h, sq, skv, d, io, causal, cold=6)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("h,sq,skv", [(6, 390, 400), (24, 23, 23), (12, 130, 260)])
def test_several_padded_items_per_place(causal, h, sq, skv):
    lengths = [(i * 97) % (skv + 1) for i in range(12)]
    check(12, h, 2, sq, skv, 128, "BFLOAT16", causal, padding=([min(sq, n + 30) for n in lengths], lengths))


@pytest.mark.parametrize("io,d", [("BFLOAT16", 128), ("HALF", 64)])
@pytest.mark.parametrize("b,h,sq,causal", [(128, 2, 300, True), (129, 2, 300, True), (40, 5, 513, False)])
def test_padded_items_by_their_lengths(io, d, b, h, sq, causal):
    """Items walked by falling length: the most (batch, pair)s that are put in order, one too many, and a list that ends inside a reversed
    round; equal lengths, empty ones and all in between."""
    lengths = [sq if i % 3 == 0 else (i * 97) % (sq + 1) for i in range(b)]
    check(b, h, 1, sq, sq, d, io, causal, padding=(lengths[::-1], lengths), fine=True)


@pytest.mark.parametrize("io,d", [("BFLOAT16", 128), ("HALF", 64)])
@pytest.mark.parametrize("b,h,sq,skv", [(7, 24, 256, 128), (5, 40, 513, 200), (3, 80, 300, 100), (2, 9, 1300, 130)])
def test_padded_queries_in_more_tiles_than_the_keys(io, d, b, h, sq, skv):
    """Query tiles without keys among the others, several an SM: behind a batch's queries, of batches without keys, and rows of a tile that is not."""
    len_q = [(sq, skv, 1, sq - 1, 128, 129, 0)[i % 7] for i in range(b)]
    len_kv = [(skv, 1, skv - 1, 0, 128, 100, 50)[i % 7] for i in range(b)]
    check(b, h, h, sq, skv, d, io, False, padding=(len_q, len_kv), fine=True)


@pytest.mark.parametrize("b,sq,causal", [(256, 500, True), (257, 500, True), (256, 500, False), (255, 512, True)])
def test_padded_items_as_many_as_are_listed(b, sq, causal):
    """1024 (batch, query tile)s are put in order by their lengths, 1028 are not, and 1020 are."""
    lengths = [sq if i % 3 == 0 else (i * 97) % (sq + 1) for i in range(b)]
    check(b, 1, 1, sq, sq, 64, "BFLOAT16", causal, padding=(lengths[::-1], lengths), fine=True)


@pytest.mark.parametrize("b,h,s,padded", [(1, 230, 900, False), (10, 20, 1100, False), (1, 220, 1024, False), (10, 20, 1100, True), (10, 23, 900, True)])
def test_more_keys_than_the_cache_holds(b, h, s, padded):
    """Causal lists that stay with one head at a time, a heavy query tile and then a light one: even and odd numbers of tiles, whole tiles, lengths."""
    lengths = ([s - 200 * (i % 4) for i in range(b)], [s - 130 * (i % 3) for i in range(b)]) if padded else None
    check(b, h, h, s, s, 128, "BFLOAT16", True, padding=lengths, fine=s % 128 != 0)


@pytest.mark.parametrize("io,d", [("BFLOAT16", 128), ("HALF", 128), ("BFLOAT16", 64), ("HALF", 64)])
@pytest.mark.parametrize("b,h,hkv,sq,skv,causal", [(3, 1, 1, 17, 17, True), (5, 4, 1, 75, 89, False), (1, 37, 37, 1000, 1000, True), (2, 96, 96, 300, 300, True), (2, 60, 12, 256, 1500, False)])
def test_probabilities_as_accurate_as_f32_ones(io, d, b, h, hkv, sq, skv, causal):
    """Short lists and long."""
    check(b, h, hkv, sq, skv, d, io, causal, fine=True)


def test_padded_and_strided_probabilities_as_accurate_as_f32_ones():
    check(5, 4, 2, 300, 300, 128, "BFLOAT16", True, padding=([300, 130, 1, 0, 257], [300, 130, 1, 200, 0]), fine=True)
    check(2, 4, 2, 256, 256, 128, "BFLOAT16", True, strided=True, fine=True)      # (whole tiles, rows that are not packed)
    check(2, 4, 2, 128, 384, 128, "BFLOAT16", True, fine=True)                    # (whole tiles, more keys than queries under a causal mask)
    check(2, 4, 2, 256, 256, 128, "HALF", False, fine=True)


@pytest.mark.parametrize("io,d", [("BFLOAT16", 128), ("HALF", 128), ("BFLOAT16", 64), ("HALF", 64)])
@pytest.mark.parametrize("b,h,sq,skv,causal", [(3, 1, 17, 17, True), (1, 37, 500, 500, True), (2, 96, 300, 300, False)])
@pytest.mark.parametrize("amplify", [700.0, 9000.0])
def test_large_scores(io, d, b, h, sq, skv, causal, amplify):
    """Scores of thousands, as the row maximum: probabilities are formed against the maximum itself, not a rounded one."""
    check(b, h, h, sq, skv, d, io, causal, fine=True, amplify=amplify)


@pytest.mark.parametrize("h", [1, 90])
def test_scores_that_are_all_minus_infinity(h):
    b, s, d = 2, 200, 128
    q, k, v = (torch.full((b, h, s, d), x, device="cuda", dtype=torch.bfloat16) for x in (1e30, -1e30, 1.0))
    q[:, :, 1::2] = 0.0   # every other row: scores of zero
    o = torch.empty_like(q)
    outs = [torch.empty(b, h, s, 1, device="cuda") for _ in range(3)]
    tensors = [graphs.tensor(uid, name, [b, h, s, d], "BFLOAT16") for uid, name in ((1, "Q"), (2, "K"), (3, "V"), (4, "O"))]
    tensors += [graphs.tensor(uid, name, [b, h, s, 1], "FLOAT") for uid, name in ((5, "Stats"), (6, "Max"), (7, "Sum_exp"))]
    node = graphs.sdpa_node("sdpa", {"Q": 1, "K": 2, "V": 3}, {"O": 4, "Stats": 5, "Max": 6, "Sum_exp": 7}, 0.5, False, True)
    exe = runtime.compile_graph(graphs.document("infinite", [node], tensors, io="BFLOAT16"))
    assert exe.steps()[0]["kernel"] == dfgpu.SDPA_UMMA
    exe.execute({uid: x.data_ptr() for uid, x in enumerate([q, k, v, o] + outs, 1)})
    torch.cuda.synchronize()
    assert dfgpu.device_status() == 0
    stats, largest, total = (x[:, :, 0::2] for x in outs)
    assert bool(torch.all(o[:, :, 0::2] == 0)) and bool(torch.all(torch.isneginf(stats))) and bool(torch.all(torch.isneginf(largest))) and bool(torch.all(total == 0))
    assert bool(torch.all(o[:, :, 1::2] == 1)) and bool(torch.all((outs[2][:, :, 1::2] - s).abs() <= 1e-3))


@pytest.mark.parametrize("io,d,strided", [("HALF", 128, False), ("BFLOAT16", 128, True)])
def test_whole_tiles_off_the_boundary_fall_back(io, d, strided):
    """Whole tiles in HALF or in a layout other than packed B, H, S, D accept pointers on the element's boundary."""
    g = torch.Generator(device="cuda").manual_seed(8)
    shape = (1, 256, 2, d) if strided else (1, 2, 256, d)
    q, k, v, o = (torch.randn(2 * 256 * d + 1, device="cuda", generator=g).to(TORCH[io])[1:].view(shape) for _ in range(4))
    if strided:
        q, k, v, o = (x.transpose(1, 2) for x in (q, k, v, o))
    tensors = [graphs.tensor(uid, name, list(x.shape), io, list(x.stride())) for uid, name, x in ((1, "Q", q), (2, "K", k), (3, "V", v), (4, "O", o))]
    exe = runtime.compile_graph(graphs.document("units", [graphs.sdpa_node("sdpa", {"Q": 1, "K": 2, "V": 3}, {"O": 4}, d ** -0.5, False, False)], tensors, io=io))
    exe.execute({1: q.data_ptr(), 2: k.data_ptr(), 3: v.data_ptr(), 4: o.data_ptr()})
    torch.cuda.synchronize()
    want, weight, _, _ = attention(q, k, v, d ** -0.5, False)
    u = ROUNDING[io]
    assert bool(torch.all((o.double() - want).abs() <= 2.0 ** -14 * weight + u * want.abs() + 1e-30))   # (the general kernel: f32 throughout)
