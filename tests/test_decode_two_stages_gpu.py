"""Four tokens through the decode dispatch: linears wide enough for the two launches with a split intermediate, at ragged
rows, ranks and chunks, against the oracle within what the decode GEMV reaches, and beside the same linears alone."""
import ctypes

import pytest
import torch

from tests.util import assert_parity, exact_np, make_group, tiles_on_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shapes", [
    [(4104, 1032, 20001)], [(12296, 2440, 4100)], [(3592, 2056, 9000), (3592, 136, 64), (3592, 1000, 5000)],
    [(4104, 6000, 4096), (4104, 8, 16)],       # a rank whose fragments do not fit: that linear stays with the GEMV
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


def call(layers, tiles, T, dtype):
    """One nq_decode_group_fwd of the first T tokens."""
    from nanoquant_b200 import _lib
    Lb = _lib.lib()
    st = torch.cuda.current_stream().cuda_stream
    ys = [torch.empty(T, L["M"], dtype=dtype, device="cuda") for L in layers]
    d = (_lib.LinearDesc * len(layers))(*[
        _lib.LinearDesc(L["x"].data_ptr(), L["s_pre"].data_ptr(), v.data_ptr(), L["s_mid"].data_ptr(), u.data_ptr(),
                        L["s_post"].data_ptr(), y.data_ptr(), L["N"], L["R"], L["M"], L["N"], L["M"])
        for L, (v, u), y in zip(layers, tiles, ys)])
    nb = Lb.nq_gemv_group_scratch_bytes(d, len(layers), T)
    scratch = torch.zeros(nb, dtype=torch.uint8, device="cuda")
    _lib.check(Lb.nq_decode_group_fwd(d, len(layers), T, _lib.NQ_BF16 if dtype == torch.bfloat16 else _lib.NQ_F16,
                                      scratch.data_ptr(), ctypes.c_size_t(nb), st), "nq_decode_group_fwd")
    assert Lb.nq_scratch_status(scratch.data_ptr(), st) == 0
    return ys


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shapes", [
    [(4096, 1600, 4096), (4096, 608, 1024), (4096, 608, 1024)],          # q/k/v: k alone is a quarter of a megabyte
    [(3328, 264, 512), (3329 + 7, 264, 512)],                            # on both sides of the line
    [(4096, 1600, 1000), (4096, 64, 500), (4096, 1001, 40), (1003, 333, 77)],   # a rank below 128, ragged ranks and widths
    [(12288, 2432, 4096), (2048, 384, 512)],
])
def test_group_equals_linears_alone(shapes, dtype):
    T = 7
    layers = make_group(shapes, T, dtype, seed=11)
    tiles = [(tiles_on_gpu(L["V"]), tiles_on_gpu(L["U"])) for L in layers]
    group = {n: call(layers, tiles, n, dtype) for n in (1, 2, 3, 4, 7)}
    for i, L in enumerate(layers):
        for n in (3, 4, 7):
            assert torch.equal(group[n][i], call([L], tiles[i:i + 1], n, dtype)[0]), f"linear {i} of {shapes}, {n} tokens"
        assert_parity(exact_np(group[7][i]), L["y64"], dtype, what=f"linear {i} of {shapes}")
        assert torch.equal(group[7][i][:4], group[4][i])         # four tokens at a time, the rest by the decode kernel
        # up to three tokens: the same bits however many ride along
        assert torch.equal(group[1][i], group[3][i][:1]) and torch.equal(group[2][i], group[3][i][:2])


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_group_equals_linears_alone_in_larger_blocks(dtype):
    """A CTA has 2 and 6 row groups of these linears alone, 7 of either in the group: outputs dealt one by one and by pairs of rows."""
    layers = make_group([(4096, 264, 4736), (4096, 264, 12288)], 4, dtype, seed=5)
    tiles = [(tiles_on_gpu(L["V"]), tiles_on_gpu(L["U"])) for L in layers]
    group = call(layers, tiles, 4, dtype)
    for i, L in enumerate(layers):
        assert torch.equal(group[i], call([L], tiles[i:i + 1], 4, dtype)[0])
        assert_parity(exact_np(group[i]), L["y64"], dtype, rel=1e-4, what=f"linear {i}")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_group_equals_linears_alone_in_larger_blocks_of_the_first_stage(dtype):
    """A CTA has three row groups of the first stage of these linears alone and nine in the group: value and remainder stored one by one and by pairs."""
    layers = make_group(4 * [(4096, 5000, 64)], 4, dtype, seed=7)
    tiles = [(tiles_on_gpu(L["V"]), tiles_on_gpu(L["U"])) for L in layers]
    group = call(layers, tiles, 4, dtype)
    for i, L in enumerate(layers):
        assert torch.equal(group[i], call([L], tiles[i:i + 1], 4, dtype)[0])
        assert_parity(exact_np(group[i]), L["y64"], dtype, rel=1e-4, what=f"linear {i}")
