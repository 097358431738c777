"""Batch kernel (5 tokens up to its limit) at the edges of its tiles: column groups of 8 tokens, row groups of 16,
chunks of 256 columns, more row groups per CTA than a pass takes, with bias and residual, in a launch group."""
import pytest
import torch

from oracle import nanoquant_oracle as oc
from tests.util import assert_parity, exact_np, make_group, tiles_on_gpu

pytestmark = pytest.mark.gpu


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
        if dtype == torch.float16 and scale[i] < 1e-3:      # outputs near fp16's subnormals: only the magnitude is checked
            assert oc.rel_err(exact_np(ys[i]), want) < 0.05
        else:
            assert_parity(exact_np(ys[i]), want, dtype, rel=2.5e-3, what=f"linear {i} of {shapes}, {T} tokens")
