"""Four tokens through the decode dispatch: groups large enough for the two launches with a split intermediate, at ragged
rows, ranks and chunks, against the oracle within what the decode GEMV reaches, and beside the same linears alone."""
import pytest
import torch

from tests.util import assert_parity, exact_np, make_group, tiles_on_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shapes", [
    [(4104, 1032, 20001)], [(12296, 2440, 4100)], [(1024, 2056, 9000), (1024, 136, 64), (1024, 1000, 5000)],
    [(1032, 6000, 4096), (1032, 8, 16)],       # a rank whose fragments do not fit: stays with the GEMV
])
def test_four_tokens_large_groups(shapes, dtype):
    from nanoquant_b200 import ops
    T = 4
    layers = make_group(shapes, T, dtype, seed=shapes[0][0], no_mid=(1,))
    tens = [(L["s_pre"], tiles_on_gpu(L["V"]), L["s_mid"], tiles_on_gpu(L["U"]), L["s_post"], L["R"]) for L in layers]
    g = torch.Generator(device="cuda").manual_seed(T)
    scale = [float(abs(L["y64"]).max()) for L in layers]
    biases = [None if i % 2 else (torch.randn(L["M"], generator=g, device="cuda") * scale[i]).to(dtype) for i, L in enumerate(layers)]
    resid = [None if i % 2 == 0 else (torch.randn(T, L["M"], generator=g, device="cuda") * scale[i]).to(dtype) for i, L in enumerate(layers)]
    ys = ops.group_forward([L["x"] for L in layers], tens, T, dtype, torch.device("cuda", 0), biases, resid)
    again = ops.group_forward([L["x"] for L in layers], tens, T, dtype, torch.device("cuda", 0), biases, resid)
    for i, L in enumerate(layers):
        want = L["y64"].copy()
        if biases[i] is not None:
            want += exact_np(biases[i])
        if resid[i] is not None:
            want += exact_np(resid[i])
        assert_parity(exact_np(ys[i]), want, dtype, rel=1e-4, what=f"linear {i} of {shapes}")
        assert torch.equal(ys[i], again[i])
