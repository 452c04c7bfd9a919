"""Cases on which the speed of this framework is measured: graphs compiled once with runtime.compile_graph and run
with Executable.execute, the way a host program drives the library, over the sizes such programs meet.

A case is a dict of plain values whose "kind" names the graph:

  conv             one f32 CONV_FPROP node, channels-last: the graph the reference was built around
  bottleneck       the ResNet-50 bottleneck DAG in bf16 (three convolutions, biases, ReLUs, residual)
  quantize_matmul  two BLOCK_SCALE_QUANTIZE nodes (MXFP8) feeding a MATMUL
  matmul_fp8       one MATMUL_FP8 node with per-tensor scales and Amax_C
  matmul           MATMUL + bias + ReLU, a linear layer
  sdpa             attention over whole prompts (prefill), causal or not, with or without padding
  decode           one new token per sequence over a paged KV cache
  pointwise        one POINTWISE node: activations and their backward forms, bias and residual additions
  quantize         one BLOCK_SCALE_QUANTIZE node
  dequantize       one BLOCK_SCALE_DEQUANTIZE node
"""
import torch

from deepforge_b200 import graphs, runtime

TORCH = {"FLOAT": torch.float32, "BFLOAT16": torch.bfloat16, "HALF": torch.float16, "INT32": torch.int32, "FP8_E4M3": torch.uint8, "FP8_E8M0": torch.uint8}
WIDTH = {name: torch.empty(0, dtype=dtype).element_size() for name, dtype in TORCH.items()}


def listed():
    return [
        # one image through one 3x3 convolution: the reference's own benchmark shape, bound by launch latency
        {"name": "conv_one_image", "kind": "conv", "n": 1, "c": 64, "k": 64, "h": 56, "w": 56, "r": 3},
        # a batch of images through a ResNet-50 bottleneck: the framework's headline workload
        {"name": "bottleneck_batch_32", "kind": "bottleneck", "n": 32, "h": 56, "w": 56},
        # a large linear layer whose weights and activations are quantized to MXFP8 on the way
        {"name": "mxfp8_4096", "kind": "quantize_matmul", "m": 4096, "k": 4096, "n": 4096},
        # an FP8 linear layer over the tokens of a few prompts: a row count that is no multiple of anything
        {"name": "fp8_ragged_tokens", "kind": "matmul_fp8", "m": 777, "k": 4096, "n": 3072, "c_type": "BFLOAT16", "b_k_major": True},
        # a bf16 linear layer with bias and activation in training or prefill
        {"name": "linear_bf16", "kind": "matmul", "m": 2048, "k": 4096, "n": 4096, "io": "BFLOAT16", "b_k_major": False},
        # attention over a batch of full prompts
        {"name": "prefill_2048", "kind": "sdpa", "b": 8, "h": 32, "hkv": 32, "s": 2048, "skv": 2048, "d": 128, "io": "BFLOAT16", "causal": True, "padding": False},
        # attention over a few prompts of different lengths, padded to the longest; grouped heads
        {"name": "prefill_padded", "kind": "sdpa", "b": 4, "h": 16, "hkv": 4, "s": 1000, "skv": 1000, "d": 128, "io": "BFLOAT16", "causal": True, "padding": True},
        # a full decode batch over a 16384-page cache
        {"name": "decode_batch_64", "kind": "decode", "batch": 64, "hq": 32, "hkv": 8, "block": 64, "pages": 16384, "min_len": 512, "max_len": 8192},
        # one or two interactive users: latency counts, few blocks in flight
        {"name": "decode_batch_2", "kind": "decode", "batch": 2, "hq": 32, "hkv": 8, "block": 64, "pages": 320, "min_len": 512, "max_len": 8192},
        # bias addition: one vector of channels broadcast over the rows
        {"name": "bias_add", "kind": "pointwise", "mode": "ADD", "io": "BFLOAT16", "rows": 4096, "cols": 3072, "broadcast": True},
        # the backward pass of an activation
        {"name": "gelu_backward", "kind": "pointwise", "mode": "GELU_BWD", "io": "BFLOAT16", "rows": 4096, "cols": 8192, "broadcast": False},
        # MXFP8 weights back to bf16
        {"name": "dequantize_weights", "kind": "dequantize", "rows": 4096, "cols": 4096, "axis": 1, "io": "BFLOAT16"},
    ]


KINDS = ("conv", "bottleneck", "quantize_matmul", "matmul_fp8", "matmul", "sdpa", "decode", "pointwise", "quantize", "dequantize")
MAX_FLOPS = 2.7e11
UNARY = ("RELU_FWD", "GELU_FWD", "GELU_APPROX_TANH_FWD", "SWISH_FWD", "SIGMOID_FWD", "TANH_FWD", "EXP")
BINARY = ("ADD", "MUL", "SUB", "RELU_BWD", "GELU_BWD", "SWISH_BWD", "SIGMOID_BWD", "TANH_BWD")
FLOATS = ("BFLOAT16", "BFLOAT16", "FLOAT", "HALF")  # bf16 is what most graphs carry


def draw(rng):
    def spread(low, high, step=1):
        """A multiple of step in [low, high], spread over the logarithm."""
        value = low * (high / low) ** rng.random()
        return max(low, min(high, int(value / step + 0.5) * step))

    while True:
        kind = rng.choice(KINDS)
        if kind == "conv":
            case = {"n": spread(1, 4), "c": spread(8, 128, 4), "k": spread(8, 128, 4), "h": spread(8, 64), "w": spread(8, 64), "r": rng.choice((1, 3, 3, 5))}
        elif kind == "bottleneck":
            side = spread(7, 56)
            case = {"n": spread(1, 64), "h": side, "w": side}
        elif kind == "quantize_matmul":
            case = {"m": spread(1, 8192), "k": spread(256, 8192, 32), "n": spread(256, 8192, 16)}
        elif kind == "matmul_fp8":
            case = {"m": spread(1, 4096), "k": spread(256, 8192, 16), "n": spread(256, 8192, 16), "c_type": rng.choice(("BFLOAT16", "BFLOAT16", "FLOAT")), "b_k_major": rng.random() < 0.6}
        elif kind == "matmul":
            io = rng.choice(FLOATS)
            case = {"m": spread(1, 8192), "k": spread(64, 8192, 8), "n": spread(64, 8192, 8), "io": io, "b_k_major": rng.random() < 0.5}
        elif kind == "sdpa":
            hkv = rng.choice((1, 2, 4, 8, 16))
            causal = rng.random() < 0.6
            s = spread(16, 4096)
            case = {"b": spread(1, 16), "h": min(32, hkv * rng.choice((1, 2, 4, 8))), "hkv": hkv, "s": s, "skv": s if causal or rng.random() < 0.5 else spread(16, 4096),
                    "d": rng.choice((64, 128, 128)), "io": rng.choice(("BFLOAT16", "BFLOAT16", "HALF")), "causal": causal, "padding": rng.random() < 0.4}
        elif kind == "decode":
            hkv, block = rng.choice((2, 4, 8, 8)), rng.choice((16, 32, 64, 128))
            batch, max_len = spread(1, 128), spread(256, 32768, 128)
            case = {"batch": batch, "hq": hkv * rng.choice((1, 2, 4, 4, 8)), "hkv": hkv, "block": block, "pages": batch * (max_len // block) * 5 // 4 + 1,
                    "min_len": rng.choice((1, max_len // 4, max_len // 2)), "max_len": max_len}
        elif kind == "pointwise":
            mode = rng.choice(UNARY + BINARY)
            case = {"mode": mode, "io": rng.choice(FLOATS), "rows": spread(1, 16384), "cols": spread(64, 8192), "broadcast": mode in ("ADD", "MUL") and rng.random() < 0.5}
        elif kind == "quantize":
            case = {"rows": spread(32, 8192, 32), "cols": spread(64, 8192, 32), "axis": rng.choice((0, 1)), "io": rng.choice(FLOATS)}
        else:
            case = {"rows": spread(32, 8192, 32), "cols": spread(64, 8192, 32), "axis": rng.choice((0, 1)), "io": rng.choice(FLOATS)}
        case["kind"] = kind
        cost = work(case)
        cache = 0 if kind != "decode" else case["pages"] * case["hkv"] * case["block"] * 128 * 4
        if cost["flops"] <= MAX_FLOPS and cost["bytes"] <= 1.3e9 and cache <= 4.4e9:
            return case


def document(case):
    kind = case["kind"]
    if kind == "conv":
        return graphs.c1_conv("nhwc", case["n"], case["c"], case["h"], case["w"], case["k"], case["r"], case["r"] // 2)
    if kind == "bottleneck":
        return graphs.c2_bottleneck(case["n"], case["h"], case["w"])
    if kind == "quantize_matmul":
        return graphs.c3_quantize_matmul(case["m"], case["k"], case["n"])
    if kind == "matmul_fp8":
        return graphs.matmul_fp8(case["m"], case["k"], case["n"], case["c_type"], batch=(), b_k_major=case["b_k_major"])
    if kind == "matmul":
        m, k, n, io = case["m"], case["k"], case["n"], case["io"]
        tensors = [graphs.tensor(1, "A", [m, k], io), graphs.tensor(2, "B", [k, n], io, [1, k] if case["b_k_major"] else [n, 1]), graphs.tensor(3, "bias", [1, n], io),
                   graphs.tensor(4, "C", [m, n], io), graphs.tensor(5, "product", [m, n], "FLOAT", virtual=True), graphs.tensor(6, "biased", [m, n], "FLOAT", virtual=True)]
        nodes = [graphs.matmul_node("matmul", 1, 2, 5), graphs.pointwise_node("bias_add", "ADD", 5, 6, 3), graphs.pointwise_node("relu", "RELU_FWD", 6, 4)]
        return graphs.document("linear", nodes, tensors, io=io)
    if kind == "sdpa":
        b, h, hkv, s, skv, d, io = (case[key] for key in ("b", "h", "hkv", "s", "skv", "d", "io"))
        tensors = [graphs.tensor(1, "Q", [b, h, s, d], io), graphs.tensor(2, "K", [b, hkv, skv, d], io), graphs.tensor(3, "V", [b, hkv, skv, d], io),
                   graphs.tensor(4, "O", [b, h, s, d], io), graphs.tensor(5, "Stats", [b, h, s, 1], "FLOAT")]
        inputs = {"Q": 1, "K": 2, "V": 3}
        if case["padding"]:
            tensors += [graphs.tensor(6, "SEQ_LEN_Q", [b, 1, 1, 1], "INT32"), graphs.tensor(7, "SEQ_LEN_KV", [b, 1, 1, 1], "INT32")]
            inputs.update(SEQ_LEN_Q=6, SEQ_LEN_KV=7)
        node = graphs.sdpa_node("sdpa", inputs, {"O": 4, "Stats": 5}, d ** -0.5, case["padding"], True, right_bound=0 if case["causal"] else None)
        return graphs.document("prefill", [node], tensors, io=io)
    if kind == "decode":
        return graphs.c5_paged_decode(case["batch"], case["hq"], case["hkv"], 128, case["pages"], case["block"], case["max_len"])
    if kind == "pointwise":
        dims, io = [case["rows"], case["cols"]], case["io"]
        tensors = [graphs.tensor(1, "IN_0", dims, io), graphs.tensor(3, "OUT_0", dims, io)]
        if case["mode"] in BINARY:
            tensors.append(graphs.tensor(2, "IN_1", [1, case["cols"]] if case["broadcast"] else dims, io))
        return graphs.document("pointwise", [graphs.pointwise_node("pointwise", case["mode"], 1, 3, 2 if case["mode"] in BINARY else None)], tensors, io=io)
    dims, io, axis = [case["rows"], case["cols"]], case["io"], case["axis"]
    scale_dims = [size // 32 if i == axis else size for i, size in enumerate(dims)]
    codes, scales = graphs.tensor(2, "codes", dims, "FP8_E4M3"), graphs.tensor(3, "scale", scale_dims, "FP8_E8M0")
    if kind == "quantize":
        return graphs.document("quantize", [graphs.quantize_node("quantize", 1, 2, 3, 32, axis)], [graphs.tensor(1, "X", dims, io), codes, scales], io=io)
    return graphs.document("dequantize", [graphs.dequantize_node("dequantize", 2, 3, 1, [32, 1] if axis == 0 else [1, 32])], [graphs.tensor(1, "Y", dims, io), codes, scales], io=io)


def prepare(case, seed):
    kind, doc = case["kind"], document(case)
    generator = torch.Generator(device="cuda").manual_seed(seed)
    buffers = {}

    def buffer(uid):
        """Uninitialised storage of an argument, one element per storage slot (every tensor here is dense)."""
        t = doc["tensors"][str(uid)]
        count = 1
        for extent in t["dim"]:
            count *= extent
        buffers[uid] = torch.empty(count, dtype=TORCH[t["data_type"]], device="cuda")
        return buffers[uid]

    def normal(uid, std=1.0):
        return buffer(uid).normal_(0.0, std, generator=generator)

    def uniform(uid, low, high):
        return buffer(uid).uniform_(low, high, generator=generator)

    def integers(uid, low, high):
        return buffer(uid).random_(low, high + 1, generator=generator)

    def outliers(uid):
        """Activations and weights as quantization meets them: one value in a hundred is 64 times larger."""
        x = normal(uid)
        return x.mul_(1 + 63 * (torch.rand(x.numel(), device="cuda", generator=generator) < 0.01).to(x.dtype))

    def codes(uid):
        x = torch.randn(buffer(uid).numel(), device="cuda", generator=generator) * 16
        buffers[uid].copy_(x.to(torch.float8_e4m3fn).view(torch.uint8))

    if kind == "conv":
        uniform(1, -1.0, 1.0), uniform(2, -1.0, 1.0)
        outputs = (3,)
    elif kind == "bottleneck":
        normal(1)
        for uid, fan_in in ((2, 256), (4, 9 * 64), (6, 64)):
            normal(uid, (2.0 / fan_in) ** 0.5)
        uniform(3, -0.1, 0.1), uniform(5, -0.1, 0.1)
        outputs = (7,)
    elif kind == "quantize_matmul":
        outliers(1), outliers(2)
        outputs = (3, 4, 5, 6, 9)
    elif kind == "matmul_fp8":
        codes(21), codes(22)
        for uid, value in ((23, 1 / 16), (24, 1 / 16), (25, 0.125)):
            buffer(uid).fill_(value)
        outputs = (26, 27)
    elif kind == "matmul":
        normal(1), normal(2, case["k"] ** -0.5), uniform(3, -0.1, 0.1)
        outputs = (4,)
    elif kind == "sdpa":
        normal(1), normal(2), normal(3)
        if case["padding"]:  # prompts between half the padded length and all of it
            longest = min(case["s"], case["skv"])
            buffers[7] = integers(6, max(1, longest // 2), longest).clone()
        outputs = (4, 5)
    elif kind == "decode":
        normal(1), normal(2), normal(3)
        buffer(5).fill_(1), integers(6, case["min_len"], case["max_len"])
        for uid in (7, 8):  # pages in the order in which a busy cache hands them out
            slots = buffer(uid)
            slots.copy_(torch.randperm(case["pages"], device="cuda", generator=generator)[: slots.numel()])
        outputs = (4,)
    elif kind == "pointwise":
        normal(1)
        if case["mode"] in BINARY:
            normal(2)
        outputs = (3,)
    elif kind == "quantize":
        outliers(1)
        outputs = (2, 3)
    else:
        codes(2), integers(3, 120, 131)
        outputs = (1,)
    for t in doc["tensors"].values():
        if not t["is_virtual"] and t["uid"] not in buffers:
            buffer(t["uid"])
    executable = runtime.compile_graph(doc)
    workspace = torch.empty(max(executable.workspace_size, 1), dtype=torch.uint8, device="cuda")
    return {"executable": executable, "pack": {uid: tensor.data_ptr() for uid, tensor in buffers.items()}, "workspace": workspace, "buffers": buffers, "outputs": outputs}


def run(state):
    state["executable"].execute(state["pack"], state["workspace"].data_ptr())
    return [state["buffers"][uid] for uid in state["outputs"]]


def work(case):
    kind = case["kind"]
    if kind == "conv":
        n, c, k, h, w, r = (case[key] for key in ("n", "c", "k", "h", "w", "r"))
        h_out, w_out = h + 2 * (r // 2) - r + 1, w + 2 * (r // 2) - r + 1
        return {"bytes": 4 * (n * c * h * w + k * c * r * r + n * k * h_out * w_out), "flops": 2 * n * h_out * w_out * k * c * r * r}
    if kind == "bottleneck":
        pixels, weights = case["n"] * case["h"] * case["w"], 256 * 64 + 9 * 64 * 64 + 64 * 256
        return {"bytes": 2 * (2 * pixels * 256 + weights + 2 * 64), "flops": 2 * pixels * weights}
    if kind == "quantize_matmul":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": (m * k + k * n) * (2 + 1 + 1 / 32) + 2 * m * n, "flops": 2 * m * k * n}
    if kind == "matmul_fp8":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": m * k + k * n + m * n * WIDTH[case["c_type"]], "flops": 2 * m * k * n}
    if kind == "matmul":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": WIDTH[case["io"]] * (m * k + k * n + n + m * n), "flops": 2 * m * k * n}
    if kind == "sdpa":
        b, h, hkv, s, skv, d = (case[key] for key in ("b", "h", "hkv", "s", "skv", "d"))
        fill = 0.75 if case["padding"] else 1.0  # mean share of the padded length
        pairs = (s * (s + 1) / 2 if case["causal"] else s * skv) * fill * fill
        return {"bytes": fill * 2 * d * (b * h * s + 2 * b * hkv * skv) + 2 * d * b * h * s + 4 * b * h * s, "flops": 4 * b * h * d * pairs}
    if kind == "decode":
        tokens = case["batch"] * (case["min_len"] + case["max_len"]) / 2
        return {"bytes": tokens * case["hkv"] * 128 * 4 + 4 * case["batch"] * case["hq"] * 128, "flops": 4 * tokens * case["hq"] * 128}
    elements = case["rows"] * case["cols"]
    if kind == "pointwise":
        operands = 2 + (case["mode"] in BINARY and not case["broadcast"])
        return {"bytes": WIDTH[case["io"]] * (elements * operands + (case["cols"] if case["broadcast"] else 0)), "flops": elements}
    return {"bytes": elements * (WIDTH[case["io"]] + 1 + 1 / 32), "flops": elements}


def tolerance(case):
    kind = case["kind"]
    if kind in ("quantize", "dequantize"):
        return "exact"  # codes and scales, and products of a code and a power of two
    if kind == "conv":
        return {"rel": 1e-5}
    if kind == "quantize_matmul":
        return {"rel": 1e-2, "differ": 0.0}  # codes and scales stay as they are
    if kind == "matmul_fp8":
        return {"rel": 1e-2 if case["c_type"] == "BFLOAT16" else 1e-4}
    if kind in ("matmul", "pointwise"):
        return {"rel": {"FLOAT": 1e-5, "HALF": 2e-3, "BFLOAT16": 1e-2}[case["io"]]}
    return {"rel": 1e-2}
