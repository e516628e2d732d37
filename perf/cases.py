"""The workloads this framework's speed is judged on, through its public entry points.

A case is a dict of plain values; `kind` says which part of an int4-AWQ language model's path it is:

  qkv          RMSNorm, one int4 GEMV over Wq|Wk|Wv and RoPE of the Q and K columns: the front of a decode layer
  gemv         one int4 decode GEMV (a projection with or without the residual add), 1 to 64 token rows
  dequant      an AWQ weight to bf16 (loading a layer for a bf16 consumer)
  stack        a stack of resident decode FFN layers (RMSNorm, gate/up, SwiGLU, down, residual), 1 to 64 token rows, called
               the three ways a program calls it: `step` (eager, device tensors), `replay` (captured graph, device tensors)
               and `host` (captured graph, host arrays in and out)
  gemm         one int4 prefill GEMM
  ffn_prefill  the prefill FFN on int4 weights: gate/up GEMM with SwiGLU, down GEMM with the residual add
  ffn_bf16     the FFN on un-quantised bf16 weights: gate, up, silu * up, down

Weights and inputs have the distributions of the benchmark: nibbles and zero points uniform, scales U(0.001, 0.02),
group 128, activations N(0, 1).
"""
import math

import numpy as np
import torch

from mlir_air_b200 import ops
from mlir_air_b200.ffn import DecodeFFNStack, random_layer

GROUP = 128


def listed():
    return [
        # The reference's own model (llama32_1b_int4: hidden 2048, 32 heads of 64, 8 KV heads): the front of one decode
        # layer for one token, four small launches in a row.  The smallest calls, where latency counts.
        dict(name="qkv_1b_b1", kind="qkv", batch=1, hidden=2048, n_heads=32, n_kv_heads=8, head_dim=64),
        # One AWQ weight of the dequant example's size.
        dict(name="dequant_2048", kind="dequant", K=2048, N=2048),
        # One decode projection at Llama-2-7B dimensions, one token.
        dict(name="gemv_7b_b1", kind="gemv", batch=1, K=4096, N=11008, residual=False),
        # The reference's model, all 16 layers, one token, called eagerly layer stack by layer stack: interactive decoding.
        dict(name="stack_1b_b1", kind="stack", batch=1, hidden=2048, intermediate=8192, layers=16, call="step"),
        # Llama-2-7B dimensions, 16 concurrent requests: the host-side call of a small serving loop.
        dict(name="stack_7b_b16", kind="stack", batch=16, hidden=4096, intermediate=11008, layers=8, call="host"),
        # Llama-3-70B dimensions, the headline batch of 8, captured graph.
        dict(name="stack_70b_b8", kind="stack", batch=8, hidden=8192, intermediate=28672, layers=8, call="replay"),
        # The same with 32 requests per step.
        dict(name="stack_70b_b32", kind="stack", batch=32, hidden=8192, intermediate=28672, layers=4, call="replay"),
        # The same with 64 requests per step, from and to host arrays.
        dict(name="stack_70b_b64", kind="stack", batch=64, hidden=8192, intermediate=28672, layers=4, call="host"),
        # Prefill of 2048 tokens through Llama-3-8B's up projection.
        dict(name="gemm_8b_2048", kind="gemm", M=2048, K=4096, N=14336),
        # A prompt of ragged length through a Llama-3-8B FFN.
        dict(name="ffn_prefill_8b_777", kind="ffn_prefill", M=777, hidden=4096, intermediate=14336),
        # A long prompt through a Llama-3-70B FFN: the largest case.
        dict(name="ffn_prefill_70b_4096", kind="ffn_prefill", M=4096, hidden=8192, intermediate=28672),
        # The un-quantised sibling path of the reference's prefill FFN example at its 1B model's dimensions.
        dict(name="ffn_bf16_1b_512", kind="ffn_bf16", M=512, hidden=2048, intermediate=8192),
    ]


def _log_int(rng, lo, hi, step=1):
    """An integer multiple of `step` in [lo, hi], spread over its logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(max(int(round(v / step)) * step, -(-lo // step) * step), hi // step * step)


def _dims(rng, weights_max):
    """hidden and intermediate of an FFN: multiples of the group, intermediate 2 to 4 times hidden."""
    while True:
        hidden = _log_int(rng, 512, 8192, GROUP)
        inter = int(hidden * rng.uniform(2.0, 4.0)) // GROUP * GROUP
        if 3 * hidden * inter <= weights_max:
            return hidden, inter


def draw(rng):
    kind = rng.choice(["qkv", "dequant", "gemv", "gemv", "stack", "stack", "stack", "gemm", "ffn_prefill", "ffn_prefill",
                       "ffn_bf16"])
    if kind == "qkv":
        head_dim = rng.choice([64, 128])
        n_kv = rng.choice([4, 8])
        n_heads = n_kv * rng.choice([1, 2, 4, 8])
        return dict(kind=kind, batch=_log_int(rng, 1, 64), hidden=n_heads * head_dim, n_heads=n_heads, n_kv_heads=n_kv,
                    head_dim=head_dim)
    if kind == "dequant":
        return dict(kind=kind, K=_log_int(rng, 512, 16384, GROUP), N=_log_int(rng, 512, 16384, 32))
    if kind == "gemv":
        return dict(kind=kind, batch=_log_int(rng, 1, 64), K=_log_int(rng, 512, 28672, GROUP),
                    N=_log_int(rng, 512, 28672, 32), residual=rng.random() < 0.5)
    if kind == "stack":
        hidden, inter = _dims(rng, 710e6)
        layers = max(1, min(_log_int(rng, 2, 16), int(5.6e9 / (3 * hidden * inter))))
        return dict(kind=kind, batch=_log_int(rng, 1, 64), hidden=hidden, intermediate=inter, layers=layers,
                    call=rng.choice(["step", "replay", "host"]))
    if kind == "gemm":
        return dict(kind=kind, M=_log_int(rng, 65, 4096), K=_log_int(rng, 512, 8192, GROUP),
                    N=_log_int(rng, 512, 28672, 32))
    if kind == "ffn_prefill":
        hidden, inter = _dims(rng, 710e6)
        return dict(kind=kind, M=_log_int(rng, 65, 4096), hidden=hidden, intermediate=inter)
    hidden = _log_int(rng, 512, 4096, 8)
    return dict(kind=kind, M=_log_int(rng, 1, 2048), hidden=hidden, intermediate=int(hidden * rng.uniform(2.0, 4.0)) // 8 * 8)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _weight(K, N, gen):
    qw = torch.randint(-2 ** 31, 2 ** 31 - 1, (K, N // 8), dtype=torch.int32, device="cuda", generator=gen)
    qz = torch.randint(-2 ** 31, 2 ** 31 - 1, (K // GROUP, N // 8), dtype=torch.int32, device="cuda", generator=gen)
    s = (torch.rand((K // GROUP, N), device="cuda", generator=gen) * 0.019 + 0.001).to(torch.bfloat16)
    return ops.AwqWeight(qw, qz, s, GROUP)


def _randn(shape, gen, scale=1.0):
    return (torch.randn(shape, device="cuda", generator=gen) * scale).to(torch.bfloat16)


def prepare(case, seed):
    kind = case["kind"]
    gen = _gen(1000003 * seed + 17)
    st = dict(case=case)
    if kind == "qkv":
        B, H, hd = case["batch"], case["hidden"], case["head_dim"]
        N = (case["n_heads"] + 2 * case["n_kv_heads"]) * hd
        st["w"], st["ws"] = _weight(H, N, gen), ops.Workspace(H, N)
        st["x"] = _randn((B, H), gen)
        st["gamma"] = (torch.randn(H, device="cuda", generator=gen) * 0.1 + 1.0).to(torch.bfloat16)
        # a table row [cos | sin] per token, at the positions of requests of different lengths
        pos = torch.randint(0, 4096, (B, 1), device="cuda", generator=gen).float()
        inv = 500000.0 ** (-torch.arange(0, hd, 2, device="cuda").float() / hd)
        st["lut"] = torch.cat([torch.cos(pos * inv), torch.sin(pos * inv)], 1).to(torch.bfloat16)
    elif kind == "dequant":
        st["w"] = _weight(case["K"], case["N"], gen)
    elif kind == "gemv":
        K, N, B = case["K"], case["N"], case["batch"]
        st["w"], st["ws"] = _weight(K, N, gen), ops.Workspace(K, N)
        st["x"] = _randn((B, K), gen)
        st["residual"] = _randn((B, N), gen) if case["residual"] else None
    elif kind == "stack":
        H, I, B = case["hidden"], case["intermediate"], case["batch"]
        layers = [random_layer(H, I, seed=1009 * seed + i) for i in range(case["layers"])]
        st["stack"] = DecodeFFNStack(layers, H)
        st["x"] = _randn((B, H), gen)
        if case["call"] == "host":
            from ml_dtypes import bfloat16
            st["x"] = st["x"].cpu().view(torch.int16).numpy().view(bfloat16)
        if case["call"] != "step":
            st["stack"].capture(B)  # a serving program captures its batch sizes when it starts
    elif kind == "gemm":
        st["w"] = _weight(case["K"], case["N"], gen)
        st["x"] = _randn((case["M"], case["K"]), gen)
    elif kind == "ffn_prefill":
        layer = random_layer(case["hidden"], case["intermediate"], seed=1009 * seed, with_gamma=False)
        st["gateup"], st["down"] = layer.gateup, layer.down
        st["x"] = _randn((case["M"], case["hidden"]), gen)
        st["h"] = _randn((case["M"], case["hidden"]), gen)
    elif kind == "ffn_bf16":
        M, H, I = case["M"], case["hidden"], case["intermediate"]
        st["x"] = _randn((M, H), gen)
        st["wg"], st["wu"] = _randn((I, H), gen, H ** -0.5), _randn((I, H), gen, H ** -0.5)
        st["wd"] = _randn((H, I), gen, I ** -0.5)
    else:
        raise ValueError(kind)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "qkv":
        q, kv, hd = case["n_heads"] * case["head_dim"], case["n_kv_heads"] * case["head_dim"], case["head_dim"]
        normed = ops.rmsnorm(st["x"], st["gamma"])
        qkv = ops.gemv(normed, st["w"], st["ws"])
        ops.rope_halfsplit(qkv[:, :q], st["lut"], case["n_heads"], hd)
        ops.rope_halfsplit(qkv[:, q:q + kv], st["lut"], case["n_kv_heads"], hd)
        return qkv
    if kind == "dequant":
        return ops.dequant(st["w"])
    if kind == "gemv":
        return ops.gemv(st["x"], st["w"], st["ws"], residual=st["residual"])
    if kind == "stack":
        stack, B = st["stack"], case["batch"]
        if case["call"] == "step":
            return stack.step(st["x"])
        if case["call"] == "replay":
            stack.load_input(st["x"])
            return stack.replay(B)
        out = stack.forward_host(st["x"])
        return torch.from_numpy(out.view(np.int16)).view(torch.bfloat16)
    if kind == "gemm":
        return ops.gemm(st["x"], st["w"])
    if kind == "ffn_prefill":
        inter = ops.gemm(st["x"], st["gateup"], swiglu=True)
        return ops.gemm(inter, st["down"], residual=st["h"])
    gate = ops.linear_bf16(st["x"], st["wg"])
    up = ops.linear_bf16(st["x"], st["wu"])
    return ops.linear_bf16(ops.silu_mul(gate, up), st["wd"])


def _weight_bytes(K, N):
    return K * N // 2 + K // GROUP * N // 2 + K // GROUP * N * 2


def work(case):
    kind = case["kind"]
    if kind == "qkv":
        H, B = case["hidden"], case["batch"]
        N = (case["n_heads"] + 2 * case["n_kv_heads"]) * case["head_dim"]
        return dict(bytes=_weight_bytes(H, N) + 2 * H + 2 * B * (H + N + case["head_dim"]), flops=2 * B * H * N)
    if kind == "dequant":
        return dict(bytes=_weight_bytes(case["K"], case["N"]) + 2 * case["K"] * case["N"], flops=2 * case["K"] * case["N"])
    if kind == "gemv":
        B, K, N = case["batch"], case["K"], case["N"]
        return dict(bytes=_weight_bytes(K, N) + 2 * B * (K + N * (2 if case["residual"] else 1)), flops=2 * B * K * N)
    if kind == "gemm":
        M, K, N = case["M"], case["K"], case["N"]
        return dict(bytes=_weight_bytes(K, N) + 2 * M * (K + N), flops=2 * M * K * N)
    H, I = case["hidden"], case["intermediate"]
    if kind == "stack":
        B, L = case["batch"], case["layers"]
        return dict(bytes=L * (_weight_bytes(H, 2 * I) + _weight_bytes(I, H) + 2 * H) + 2 * B * 2 * H, flops=L * 6 * B * H * I)
    M = case["M"]
    if kind == "ffn_prefill":
        return dict(bytes=_weight_bytes(H, 2 * I) + _weight_bytes(I, H) + 2 * M * 3 * H, flops=6 * M * H * I)
    return dict(bytes=2 * 3 * H * I + 2 * M * 2 * H, flops=6 * M * H * I)


def tolerance(case):
    # Each is about four times the largest relative error seen on these cases and on drawn ones, against the same chain in
    # 64-bit arithmetic with the path's own bf16 rounding points (normalised rows, gate and up sums, SwiGLU outputs, hidden
    # states, results).  A dequantised weight is one exact product rounded once.
    kind = case["kind"]
    if kind == "dequant":
        return "exact"
    if kind in ("gemv", "qkv"):
        return {"rel": 1e-3}  # seen: 2.4e-4 (results that fall on the other side of a bf16 rounding boundary)
    if kind == "gemm":
        return {"rel": 1e-2}  # seen: 2.5e-3 (weights rounded to bf16 for the tensor core)
    if kind == "ffn_prefill":
        return {"rel": 1.9e-2}  # seen: 4.7e-3 (two such products in a row)
    if kind == "ffn_bf16":
        return {"rel": 3e-3}  # seen: 6.9e-4
    # A rounding that falls differently in one layer moves the next layer's inputs: seen 2.1e-3 after 2 layers, 7.4e-3 after
    # 4, 1.2e-2 after 6 and 8, 2.0e-2 after 14 and 16.
    return {"rel": min(8e-3 * max(case["layers"], 2), 8e-2)}
