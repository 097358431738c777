"""The work that users of nanoquant_b200 have it do, as cases to measure.

A case is a dict of plain values.  ``kind`` says which public entry points it goes through:

* ``linear``  one prepared ``NanoQuantLinear`` called as a module (what a class-swapped ``nn.Linear`` of a model is),
              any size, with or without bias: ``N`` in, rank ``R``, ``M`` out.  ``kernel`` is what it was prepared
              for; either takes any number of tokens.
* ``layer``   the seven quantised linears of ``layers`` decoder layers (q/k/v/o with ``hidden`` and ``kv`` columns,
              gate/up/down with ``inter``) at ``bpw`` bits per weight, ``tokens`` tokens.  ``mode``:
              ``modules``  every linear called on its own, eagerly (the reference's way of running a model);
              ``groups``   ``LinearGroup``: q/k/v and gate/up as one launch group each, eagerly;
              ``graph``    the same groups captured once in a CUDA graph that is replayed for every decode step.
* ``head``    the un-quantised ``lm_head`` of a decode step, ``ops.dense_gemv_forward``.
* ``pack``    the weight formats: ``form`` ``rows`` packs a dense +-1 matrix into checkpoint words, turns the words
              into the kernels' tile layout and unpacks them again (save, load and inspect a checkpoint);
              ``marlin`` packs it into the Marlin layout with its permuted scales.

Weights are random signs, scales (U[0,1) + 0.5) * 0.01, activations N(0, 1): the distributions of the repository's
benchmark.
"""
from __future__ import annotations

import math

import torch

from nanoquant_b200 import ops
from nanoquant_b200.kernel import utils as ku
from nanoquant_b200.modules.group import LinearGroup
from nanoquant_b200.modules.linear import NanoQuantLinear

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def listed():
    return [
        # the smallest projection of a small model (Llama-3.2-1B k_proj), one token: call overhead and launch latency
        dict(name="linear-2048x512-t1", kind="linear", N=2048, R=384, M=512, tokens=1, dtype="fp16", kernel="gemv",
             bias=False),
        # a linear whose sizes divide by nothing, three sequences, with a bias
        dict(name="linear-odd-bias-t3", kind="linear", N=1003, R=333, M=777, tokens=3, dtype="bf16", kernel="gemv",
             bias=True),
        # one decoded token through the seven linears of a Qwen3-8B layer, the way a class-swapped model calls them
        dict(name="qwen3-8b-modules-t1", kind="layer", mode="modules", hidden=4096, inter=12288, kv=1024, bpw=0.8,
             layers=1, tokens=1, dtype="bf16", kernel="gemv"),
        # two sequences through launch groups without a graph (Llama-3.2-1B shapes)
        dict(name="llama-1b-groups-t2", kind="layer", mode="groups", hidden=2048, inter=8192, kv=512, bpw=1.0,
             layers=4, tokens=2, dtype="fp16", kernel="gemv"),
        # the decode step of a serving loop: launch groups in a replayed CUDA graph, packed factors larger than L2
        dict(name="qwen3-8b-graph-t1", kind="layer", mode="graph", hidden=4096, inter=12288, kv=1024, bpw=0.8,
             layers=8, tokens=1, dtype="bf16", kernel="gemv"),
        # the same for four and for sixteen sequences
        dict(name="qwen3-8b-graph-t4", kind="layer", mode="graph", hidden=4096, inter=12288, kv=1024, bpw=0.8,
             layers=8, tokens=4, dtype="fp16", kernel="gemv"),
        dict(name="qwen3-8b-graph-t16", kind="layer", mode="graph", hidden=4096, inter=12288, kv=1024, bpw=0.8,
             layers=8, tokens=16, dtype="bf16", kernel="gemv"),
        # a 128-token prompt (the reference's benchmark condition) through one Llama-2-7B layer, module by module
        dict(name="llama-7b-modules-t128", kind="layer", mode="modules", hidden=4096, inter=11008, kv=4096, bpw=1.0,
             layers=1, tokens=128, dtype="fp16", kernel="gemm"),
        # a prompt of no particular length
        dict(name="qwen3-8b-groups-t517", kind="layer", mode="groups", hidden=4096, inter=12288, kv=1024, bpw=0.8,
             layers=1, tokens=517, dtype="bf16", kernel="gemv"),
        # a long prompt: tensor-core bound
        dict(name="llama-7b-groups-t2048", kind="layer", mode="groups", hidden=4096, inter=11008, kv=4096, bpw=1.0,
             layers=1, tokens=2048, dtype="bf16", kernel="gemv"),
        # the bf16 head of a decode step (Qwen3-8B vocabulary)
        dict(name="head-151936x4096-t1", kind="head", V=151936, N=4096, tokens=1, dtype="bf16"),
        # one factor of a Qwen3-8B projection through the checkpoint formats
        dict(name="pack-rows-12288x2432", kind="pack", form="rows", rows=12288, cols=2432),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _up(v, m):
    return max(m, (v + m - 1) // m * m)


def draw(rng):
    most = work(next(c for c in listed() if c["name"] == "llama-7b-groups-t2048"))
    while True:
        c = _draw(rng)
        w = work(c)
        if w["flops"] <= most["flops"] and w["bytes"] <= 1.3e9:
            return c


def _draw(rng):
    dtype = rng.choice(["fp16", "bf16"])
    kind = rng.choice(["linear", "linear", "linear", "layer", "layer", "layer", "layer", "layer", "head", "pack"])
    if kind == "linear":
        # one in four divides by nothing; the others by 32 (or 64) as model widths do.  Odd sizes decode only: the
        # tensor-core path takes multiples of 8.
        odd = rng.random() < 0.25
        N, M = _log(rng, 512, 14336), _log(rng, 256, 14336)
        if not odd:
            N, M = _up(N, 64), _up(M, 64)
        R = rank_for_bits(N, M, rng.uniform(0.5, 1.5)) + (rng.randrange(32) if odd else 0)
        T = rng.randint(1, 4) if odd or rng.random() < 0.4 else _log(rng, 1, 2048)
        return dict(kind="linear", N=N, R=R, M=M, tokens=T, dtype=dtype,
                    kernel="gemv" if odd else rng.choice(["gemv", "gemm"]), bias=rng.random() < 0.3)
    if kind == "layer":
        mode = rng.choice(["modules", "groups", "graph"])
        hidden = _up(_log(rng, 1024, 8192), 128)
        inter = _up(int(hidden * rng.uniform(2.5, 4.0)), 64)
        kv = hidden // rng.choice([1, 2, 4, 8])
        if mode == "graph":   # decode steps
            T, layers = rng.choice([1, 1, 2, 3, 4, _log(rng, 5, 64)]), rng.randint(2, 8)
        else:
            T, layers = rng.choice([1, _log(rng, 1, 64), _log(rng, 64, 2048)]), rng.randint(1, 2)
        return dict(kind="layer", mode=mode, hidden=hidden, inter=inter, kv=kv, bpw=round(rng.uniform(0.5, 1.5), 2),
                    layers=layers, tokens=T, dtype=dtype,
                    kernel=rng.choice(["gemv", "gemm"]) if mode == "modules" else "gemv")
    if kind == "head":
        return dict(kind="head", V=_log(rng, 8000, 152000), N=_up(_log(rng, 1024, 8192), 64),
                    tokens=_log(rng, 1, 16), dtype=dtype)
    if rng.random() < 0.5:
        return dict(kind="pack", form="rows", rows=_log(rng, 256, 28672), cols=_log(rng, 256, 12288))
    return dict(kind="pack", form="marlin", rows=_up(_log(rng, 256, 28672), 64), cols=_up(_log(rng, 256, 12288), 16))


def rank_for_bits(in_f, out_f, bits):
    """Rank of a layer at a bit budget (the two-scale formula of the model family: multiples of 32)."""
    r = int(in_f * out_f * bits / (in_f + out_f) - 16) // 32 * 32
    return max(32, min(r, in_f, out_f))


def _layer_linears(c):
    """(name, input buffer, N, R, M) of a decoder layer."""
    h, i, kv = c["hidden"], c["inter"], c["kv"]
    spec = [("q", "h", h, h), ("k", "h", h, kv), ("v", "h", h, kv), ("o", "a", h, h), ("gate", "m", h, i),
            ("up", "m", h, i), ("down", "i", i, h)]
    return [(n, src, N, rank_for_bits(N, M, c["bpw"]), M) for (n, src, N, M) in spec]


_GROUPS = (("q", "k", "v"), ("o",), ("gate", "up"), ("down",))


def _packed(gen, rows, cols):
    """Random sign bits as checkpoint words; the padding columns of the last word are +1 (bit 0)."""
    w = torch.randint(-2 ** 31, 2 ** 31 - 1, (rows, (cols + 31) // 32), generator=gen, device="cuda",
                      dtype=torch.int32)
    if cols % 32:
        w[:, -1] &= (1 << (cols % 32)) - 1
    return w


def _module(gen, N, R, M, dtype, kernel, bias=False):
    m = NanoQuantLinear(N, M, R)
    if bias:
        m.bias = torch.nn.Parameter((torch.randn(M, generator=gen, device="cuda") * 0.01).to(dtype),
                                    requires_grad=False)
    scale = lambda n: ((torch.rand(n, generator=gen, device="cuda") + 0.5) * 0.01).to(dtype)
    m.load_packed(_packed(gen, R, N), (R, N), _packed(gen, M, R), (M, R), scale(N), scale(M), scale(R), dtype=dtype,
                  kernel_type=kernel)
    return m


def _activations(gen, T, N, dtype):
    """Decode: one token of each of T sequences; more than 64 tokens: one sequence."""
    shape = (T, 1, N) if T <= 64 else (1, T, N)
    return torch.randn(shape, generator=gen, device="cuda").to(dtype)


@torch.no_grad()
def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "pack":
        rows, cols = case["rows"], case["cols"]
        w = torch.randint(0, 2, (rows, cols), generator=gen, device="cuda", dtype=torch.int8).mul_(2).sub_(1)
        s = [((torch.rand(n, generator=gen, device="cuda") + 0.5) * 0.01).to(torch.bfloat16) for n in (cols, rows // 32 * 32)]
        return dict(kind="pack-" + case["form"], w=w, shape=(rows, cols), scales=s)
    dtype = DTYPES[case["dtype"]]
    if kind == "head":
        w = (torch.randn((case["V"], case["N"]), generator=gen, device="cuda") * 0.02).to(dtype)
        return dict(kind="head", w=w, x=_activations(gen, case["tokens"], case["N"], dtype))
    if kind == "linear":
        m = _module(gen, case["N"], case["R"], case["M"], dtype, case["kernel"], case["bias"])
        return dict(kind="linear", m=m, x=_activations(gen, case["tokens"], case["N"], dtype))
    state = dict(kind=case["mode"], calls=[])
    for _ in range(case["layers"]):
        mods, xs = {}, {}
        for name, src, N, R, M in _layer_linears(case):
            mods[name] = (_module(gen, N, R, M, dtype, case["kernel"]), src)
            if src not in xs:
                xs[src] = _activations(gen, case["tokens"], N, dtype)
        if case["mode"] == "modules":
            state["calls"] += [(m, xs[src]) for m, src in mods.values()]
        else:
            state["calls"] += [(LinearGroup([mods[n][0] for n in names]), xs[mods[names[0]][1]]) for names in _GROUPS]
    if case["mode"] == "graph":
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            _groups(state)   # warm-up outside the capture
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                state["outputs"] = _groups(state)
        torch.cuda.current_stream().wait_stream(stream)
        state["graph"] = graph
    return state


def _groups(state):
    return [y for group, x in state["calls"] for y in group(x)]


@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["m"](state["x"])
    if kind == "modules":
        return [m(x) for m, x in state["calls"]]
    if kind == "groups":
        return _groups(state)
    if kind == "graph":
        state["graph"].replay()
        return state["outputs"]
    if kind == "head":
        return ops.dense_gemv_forward(state["x"], state["w"])
    if kind == "pack-rows":
        words = ku.pack_binary_gemv(state["w"], method="lsb_first")
        tiles = ku.pack_tiles(words, state["shape"], "lsb_first")
        return words, tiles, ku.unpack_binary_gemv(words, state["shape"], method="lsb_first")
    return ku.pack_binary_marlin(state["w"], *state["scales"])[:3]


def work(case):
    """Every packed factor, scale, input and output once; two operations per weight of the factors and token."""
    kind = case["kind"]
    if kind == "pack":
        rows, cols = case["rows"], case["cols"]
        if case["form"] == "marlin":   # dense in, words out, both scales in and out
            return dict(bytes=rows * cols + rows * cols // 8 + 4 * (rows + cols), flops=0)
        words, tiles = 4 * rows * ((cols + 31) // 32), 512 * ((rows + 15) // 16) * ((cols + 255) // 256)
        return dict(bytes=rows * cols + words + tiles + rows * cols, flops=0)
    T = case["tokens"]
    if kind == "head":
        V, N = case["V"], case["N"]
        return dict(bytes=2 * V * N + 2 * T * (V + N), flops=2 * T * V * N)
    if kind == "linear":
        N, R, M = case["N"], case["R"], case["M"]
        return dict(bytes=R * (N + M) // 8 + 2 * (N + R + M) + 2 * T * (N + M) + (2 * M if case["bias"] else 0),
                    flops=2 * T * R * (N + M))
    nbytes = flops = 0
    inputs = {}
    for _, src, N, R, M in _layer_linears(case):
        inputs[src] = 2 * T * N
        nbytes += R * (N + M) // 8 + 2 * (N + R + M) + 2 * T * M
        flops += 2 * T * R * (N + M)
    return dict(bytes=case["layers"] * (nbytes + sum(inputs.values())), flops=case["layers"] * flops)


def tolerance(case):
    """Packed words and bytes are exact.  Outputs are rounded to the I/O type, and the tensor-core path keeps the
    rank-R intermediate in that type as well: 2^-9 (bf16) or 2^-12 (fp16) per rounding."""
    if case["kind"] == "pack":
        return "exact"
    return {"rel": 1e-2, "max": 0.1} if case["dtype"] == "bf16" else {"rel": 1.5e-3, "max": 0.015}
