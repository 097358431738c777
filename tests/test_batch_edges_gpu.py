"""Batch kernel (5 tokens up to its limit) at the edges of its tiles: column groups of 8 tokens, row groups of 16,
chunks of 256 columns, more row groups per CTA than a pass takes, with bias and residual, in a launch group."""
import numpy as np
import pytest
import torch

from tests.util import exact_np, make_group, tiles_on_gpu

pytestmark = pytest.mark.gpu


def bound(L, y, want, dtype):
    """What rounding the intermediate t and the output to `dtype` and summing in fp32 may cost, element by element.

    Every t_r is rounded once, by at most half a unit in its last place d_r, uniform and independent, so the sum over r stays
    within six standard deviations of d_r / sqrt(3) each, and never exceeds the sum of the d_r.  fp32 sums: 2^-24 a step in a random walk over up to 4104 steps, 2^-18 of the norm of the terms.  The output
    is rounded once: half a unit in its last place.  (2e-3 of the largest output, the bar of the other tests, is not a bound
    for a handful of outputs: the largest of five may be small beside the norm of its terms.)"""
    half = dtype == torch.float16
    xs = exact_np(L["x"]) * exact_np(L["s_pre"])
    mid = exact_np(L["s_mid"]) if L["s_mid"] is not None else np.ones(L["R"])
    t = (xs @ L["V"].T.astype(np.float64)) * mid
    half_ulp = lambda v: 2.0 ** (np.floor(np.log2(np.maximum(np.abs(v), 2.0 ** (-14 if half else -126)))) - (11 if half else 8))
    d = half_ulp(t)
    rounding_t = np.minimum(d.sum(axis=1), 6 / np.sqrt(3) * np.sqrt((d * d).sum(axis=1)))
    fp32 = 2.0 ** -18 * np.sqrt(L["R"]) * np.abs(mid).max() * np.sqrt((xs * xs).sum(axis=1))
    return np.outer(rounding_t + fp32, np.abs(exact_np(L["s_post"]))) + half_ulp(np.maximum(np.abs(y), np.abs(want)))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T", [5, 8, 9, 16, 17, 25, 32, 33])
@pytest.mark.parametrize("shapes", [
    [(8, 8, 1)], [(264, 24, 17), (264, 256, 400)], [(4104, 264, 1000)], [(512, 1032, 30000)],
    [(1024, 96, 500), (1024, 200, 64), (1024, 40, 64), (1024, 8, 8)],
])
def test_batch_tile_edges(shapes, T, dtype):
    from nanoquant_b200 import ops
    layers = make_group(shapes, T, dtype, seed=T + shapes[0][0], no_mid=(1,))
    n = len(layers)
    tens = [(L["s_pre"], tiles_on_gpu(L["V"]), L["s_mid"], tiles_on_gpu(L["U"]), L["s_post"], L["R"]) for L in layers]
    g = torch.Generator(device="cuda").manual_seed(T)
    scale = [float(abs(L["y64"]).max()) for L in layers]
    biases = [None if i % 2 else (torch.randn(L["M"], generator=g, device="cuda") * scale[i]).to(dtype) for i, L in enumerate(layers)]
    resid = [None if i % 2 == 0 else (torch.randn(T, L["M"], generator=g, device="cuda") * scale[i]).to(dtype) for i, L in enumerate(layers)]
    ys = ops.group_forward([L["x"] for L in layers], tens, T, dtype, torch.device("cuda", 0), biases, resid)
    torch.cuda.synchronize()
    for i in range(n):
        want = layers[i]["y64"].copy()
        if biases[i] is not None:
            want += exact_np(biases[i])
        if resid[i] is not None:
            want += exact_np(resid[i])
        y = exact_np(ys[i])
        worst = float((np.abs(y - want) - bound(layers[i], y, want, dtype)).max())
        assert worst <= 0, f"linear {i} of {shapes}, {T} tokens: {worst:.3e} beyond the bound"


@pytest.mark.parametrize("shape,T", [
    ((264, 5016, 9999), 5), ((264, 5016, 9999), 16),      # blocks of up to and beyond 512 outputs, an odd last row, rows at odd addresses
    ((264, 5016, 10000), 16),                             # pairs of outputs as one store
    ((8, 8, 700000), 5),                                  # more rows of a CTA than it keeps scales of
    ((28680, 2376, 48), 8),                               # one staged step per warp
])
@pytest.mark.parametrize("shifted", [False, True])        # scales of both stages and bias at an address that a bulk copy does not take
def test_batch_blocks_of_outputs(shape, T, shifted):
    from nanoquant_b200 import ops
    dtype = torch.bfloat16
    L = make_group([shape], T, dtype, seed=T)[0]
    scale = float(abs(L["y64"]).max())
    g = torch.Generator(device="cuda").manual_seed(T)
    bias = (torch.randn(L["M"], generator=g, device="cuda") * scale).to(dtype)
    resid = (torch.randn(T, L["M"], generator=g, device="cuda") * scale).to(dtype)
    move = lambda v: torch.cat([v[:1], v])[1:] if shifted else v
    tens = (L["s_pre"], tiles_on_gpu(L["V"]), move(L["s_mid"]), tiles_on_gpu(L["U"]), move(L["s_post"]), L["R"])
    y = exact_np(ops.group_forward([L["x"]], [tens], T, dtype, torch.device("cuda", 0), [move(bias)], [resid])[0])
    want = L["y64"] + exact_np(bias) + exact_np(resid)
    assert float((np.abs(y - want) - bound(L, y, want, dtype)).max()) <= 0


@pytest.mark.parametrize("T,single", [(4, False), (8, False), (16, False), (16, True)])
def test_output_scales_written_by_the_kernel_before(T, single):
    """The output scales of a first stage are the result of the linear directly before it on the stream, which lets its successor in early."""
    from nanoquant_b200 import _lib, ops
    dtype, dev = torch.bfloat16, torch.device("cuda", 0)
    # few CTAs, a long chunk loop; four tokens of more than 3328 columns take the batch kernel
    A, B = make_group([(8192, 64, 1032), (4104, 1032, 264)], T, dtype, seed=T)
    tiles = {id(L): (tiles_on_gpu(L["V"]), tiles_on_gpu(L["U"])) for L in (A, B)}
    tens = lambda L, mid: (L["s_pre"], tiles[id(L)][0], mid, tiles[id(L)][1], L["s_post"], L["R"])
    ops.reserve_scratch(dev, max(ops.group_scratch_bytes([(L["N"], L["R"], L["M"])], T) for L in (A, B)))
    x = A["x"][:1].clone()
    out, status = torch.empty(T, B["R"], dtype=dtype, device=dev), torch.zeros(64, dtype=torch.int32, device=dev)

    def use(scales):
        if not single:
            return ops.group_forward([B["x"]], [tens(B, scales)], T, dtype, dev)[0]
        _lib.check(_lib.lib().nq_onebit_gemm_fwd(B["x"].data_ptr(), tiles[id(B)][0].data_ptr(), B["s_pre"].data_ptr(), scales.data_ptr(), out.data_ptr(),
                                                 status.data_ptr(), T, B["N"], B["R"], _lib.NQ_BF16, torch.cuda.current_stream().cuda_stream), "nq_onebit_gemm_fwd")
        return out

    def both():
        scales = ops.group_forward([x], [tens(A, A["s_mid"])], 1, dtype, dev)[0].view(-1)
        return scales, use(scales)

    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        both()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            scales, y = both()
    torch.cuda.current_stream().wait_stream(stream)
    for i in range(8):
        x.copy_(torch.randn_like(x))          # other scales in the same place
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        got, now = y.clone(), scales.clone()
        assert torch.equal(got, use(now)), f"replay {i}"


def with_epilogue(layers, T, dtype, seed):
    """Biases and residuals of the size of the outputs, and what is expected with them."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    draw = lambda shape, L: (torch.randn(shape, generator=g, device="cuda") * float(abs(L["y64"]).max())).to(dtype)
    biases, resid = [draw((L["M"],), L) for L in layers], [draw((T, L["M"]), L) for L in layers]
    return biases, resid, [L["y64"] + exact_np(b) + exact_np(r) for L, b, r in zip(layers, biases, resid)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shapes,T", [(2 * [(8192, 5056, 264)], 7), (2 * [(8192, 5056, 264)], 8), (4 * [(2048, 5056, 64)], 5), (4 * [(2048, 5056, 64)], 8)])
def test_first_stage_of_more_than_512_outputs_per_block(shapes, T, dtype):
    """Rows two apart of the fragment order are stored together, one column group.  gate/up of 8192 columns: five row groups per CTA and a token per thread;
    the others nine and up to two, the second of which does not exist for all threads at five tokens."""
    from nanoquant_b200 import ops
    layers = make_group(shapes, T, dtype, seed=T)
    tens = [(L["s_pre"], tiles_on_gpu(L["V"]), L["s_mid"], tiles_on_gpu(L["U"]), L["s_post"], L["R"]) for L in layers]
    biases, resid, wants = with_epilogue(layers, T, dtype, T)
    ys = ops.group_forward([L["x"] for L in layers], tens, T, dtype, torch.device("cuda", 0), biases, resid)
    for L, y, want in zip(layers, ys, wants):
        y = exact_np(y)
        assert float((np.abs(y - want) - bound(L, y, want, dtype)).max()) <= 0


@pytest.mark.parametrize("T", [9, 16])
def test_precise_intermediate_in_large_blocks(T):
    """Powers of two per token taken out of more than 512 outputs per block, with a residual that is the output itself."""
    from nanoquant_b200 import ops
    dtype = torch.bfloat16
    L = make_group([(1032, 1000, 10001)], T, dtype, seed=T)[0]
    tens = (L["s_pre"], tiles_on_gpu(L["V"]), L["s_mid"], tiles_on_gpu(L["U"]), L["s_post"], L["R"])
    x = L["x"].clone()
    x[1] *= 2.0 ** 20          # powers of two that differ between the tokens
    x[T - 1] *= 2.0 ** -20
    token = np.ones((T, 1))
    token[1], token[T - 1] = 2.0 ** 20, 2.0 ** -20
    g = torch.Generator(device="cuda").manual_seed(T)
    bias = (torch.randn(L["M"], generator=g, device="cuda") * float(abs(L["y64"]).max())).to(dtype)
    resid = (torch.randn(T, L["M"], generator=g, device="cuda") * torch.from_numpy(token * np.abs(L["y64"]).max()).float().cuda()).to(dtype)
    want = L["y64"] * token + exact_np(bias) + exact_np(resid)
    old = ops.set_precise_intermediate(True)
    try:
        y = exact_np(ops.group_forward([x], [tens], T, dtype, x.device, [bias], [resid], out=resid)[0])
    finally:
        ops.set_precise_intermediate(old)
    # 1e-3 of a token's largest product, the bar of this mode, and half a unit of the output
    half_ulp = 2.0 ** (np.floor(np.log2(np.maximum(np.maximum(np.abs(y), np.abs(want)), 2.0 ** -126))) - 8)
    assert (np.abs(y - want) <= 1e-3 * token * np.abs(L["y64"]).max(axis=1, keepdims=True) + half_ulp).all()
