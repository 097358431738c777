"""Activations that are not finite, and activations far below one: a token with a NaN or an infinity has NaN in every
output and leaves the other tokens' bits alone; a token scaled by a power of two gives the scaled result."""
import pytest
import torch

from tests.util import assert_parity, exact_np, make_layer, tiles_on_gpu

pytestmark = pytest.mark.gpu

SHAPES = [(520, 136, 96), (4104, 264, 1000), (1003, 333, 77)]


def gemv(L, x):
    """The decode kernel through the C ABI."""
    from nanoquant_b200 import _lib
    Lb = _lib.lib()
    (T, N), R, M = x.shape, L["R"], L["M"]
    st = torch.cuda.current_stream().cuda_stream
    nb = Lb.nq_gemv_scratch_bytes(T, N, R, M)
    scratch = torch.zeros(nb, dtype=torch.uint8, device="cuda")
    y = torch.empty((T, M), dtype=x.dtype, device="cuda")
    vt, ut = tiles_on_gpu(L["V"]), tiles_on_gpu(L["U"])
    _lib.check(Lb.nq_gemv_fwd(x.data_ptr(), L["s_pre"].data_ptr(), vt.data_ptr(), L["s_mid"].data_ptr(), ut.data_ptr(),
                              L["s_post"].data_ptr(), y.data_ptr(), scratch.data_ptr(), nb, T, N, R, M,
                              _lib.NQ_BF16 if x.dtype == torch.bfloat16 else _lib.NQ_F16, st), "nq_gemv_fwd")
    assert Lb.nq_scratch_status(scratch.data_ptr(), st) == 0
    return y


def spoil(x, tok, value):
    """`value` in two columns of token `tok`, in different chunks of 256 columns."""
    x = x.clone()
    x[tok, 7] = value
    x[tok, x.size(1) - 2] = value
    return x


@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("T,dtype", [(1, torch.bfloat16), (2, torch.float16), (3, torch.bfloat16), (4, torch.float16)])
@pytest.mark.parametrize("N,R,M", SHAPES)
def test_decode_kernel_not_finite(N, R, M, T, dtype, value):
    L = make_layer(N, R, M, T, dtype, seed=N + T)
    clean = gemv(L, L["x"])
    y = gemv(L, spoil(L["x"], T - 1, value))
    assert torch.isnan(y[T - 1]).all()
    assert torch.equal(y[:T - 1], clean[:T - 1])


@pytest.mark.parametrize("exponent", [-40, -96, -100, -104])
@pytest.mark.parametrize("T", [1, 4])
def test_decode_kernel_small_activations(T, exponent):
    # products s_in * x from 1e-14 down to 1e-33, whose fixed-point scale has no fp32 reciprocal; the unit of a chunk is
    # then a subnormal of 18 bits or more, and outputs (1e-34 and above) are normal in bf16
    N, R, M = 1032, 136, 520
    L = make_layer(N, R, M, T, torch.bfloat16, seed=5)
    L["s_mid"] = torch.ones_like(L["s_mid"])
    from oracle import nanoquant_oracle as oc
    want = oc.forward_fp64(exact_np(L["x"]), L["V"], L["U"], exact_np(L["s_pre"]), None, exact_np(L["s_post"]))
    y = gemv(L, L["x"] * 2.0 ** exponent)
    assert_parity(exact_np(y) * 2.0 ** -exponent, want, torch.bfloat16, rel=1e-4, what=f"2^{exponent}")


@pytest.mark.parametrize("exponent", [60, 119, 121, 122, 123])
@pytest.mark.parametrize("T", [1, 2, 3, 4])
def test_decode_kernel_large_activations(T, exponent):
    # maxima on both sides of 1e37, from where on their approximate reciprocal would be subnormal
    N, R, M = 40, 136, 520
    L = make_layer(N, R, M, T, torch.bfloat16, seed=5)
    L["s_pre"] = torch.ones_like(L["s_pre"])
    L["s_mid"] = torch.full_like(L["s_mid"], 2.0 ** -100)
    from oracle import nanoquant_oracle as oc
    x = L["x"] * 2.0 ** exponent
    assert torch.isfinite(x).all() and (exponent < 123 or x.abs().max() > 1e37)
    want = oc.forward_fp64(exact_np(x), L["V"], L["U"], exact_np(L["s_pre"]), exact_np(L["s_mid"]), exact_np(L["s_post"]))
    assert_parity(exact_np(gemv(L, x)), want, torch.bfloat16, rel=1e-4, what=f"2^{exponent}")


@pytest.mark.parametrize("largest", [8.4e37, 8.6e37, 1.5e38, 2.5e38])
@pytest.mark.parametrize("T", [1, 2, 3, 4])
def test_decode_kernel_reciprocal_below_normal_numbers(T, largest):
    # Above 2^126 = 8.5e37 the reciprocal of a maximum is subnormal (flushed, all integers would be zero).  Three columns of a token, whose sum
    # stays finite: each is at most half an integer, 1.5e-5 of the maximum, off, the intermediate the same again, which averages over the rank.
    N, R, M = 40, 136, 520
    L = make_layer(N, R, M, T, torch.bfloat16, seed=5)
    L["s_pre"] = torch.ones_like(L["s_pre"])
    L["s_mid"] = torch.full_like(L["s_mid"], 2.0 ** -100)
    x = torch.zeros_like(L["x"])
    for t in range(T):
        for k, part in enumerate((1.0, -0.25, 0.0625)):
            x[t, (7 * t + 11 * k) % N] = largest * part
    assert torch.isfinite(x).all() and ((x.abs().amax(dim=1) > 2.0 ** 126) == (largest > 8.5e37)).all()
    from oracle import nanoquant_oracle as oc
    want = oc.forward_fp64(exact_np(x), L["V"], L["U"], exact_np(L["s_pre"]), exact_np(L["s_mid"]), exact_np(L["s_post"]))
    assert_parity(exact_np(gemv(L, x)), want, torch.bfloat16, rel=1e-4, what=f"{largest}")


def dispatched(L, x, resid=None, precise=False):
    """A launch group of one, as the module calls it."""
    from nanoquant_b200 import ops
    tens = [(L["s_pre"], tiles_on_gpu(L["V"]), L["s_mid"], tiles_on_gpu(L["U"]), L["s_post"], L["R"])]
    old = ops.set_precise_intermediate(precise)
    try:
        return ops.group_forward([x], tens, x.size(0), x.dtype, x.device, [None], None if resid is None else [resid])[0]
    finally:
        ops.set_precise_intermediate(old)


# four tokens of a linear large enough for the pair of bf16 words; batch kernel at one and three column groups; GEMM with
# the K split over a cluster and without
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,N,R,M", [(1, 520, 136, 96), (4, 4104, 1032, 8000), (8, 520, 136, 96), (20, 1032, 264, 1000),
                                     (40, 520, 136, 96), (300, 1032, 264, 8200)])
def test_dispatch_not_finite(T, N, R, M, dtype, value):
    L = make_layer(N, R, M, T, dtype, seed=N + T)
    bad = spoil(L["x"], T - 1, value)
    for precise in ((False, True) if T > 4 and dtype == torch.bfloat16 else (False,)):
        clean = dispatched(L, L["x"], precise=precise)
        y = dispatched(L, bad, precise=precise)
        assert torch.isnan(y[T - 1]).all()
        assert torch.equal(y[:T - 1], clean[:T - 1]) and torch.isfinite(clean).all()
    # a residual that is not finite belongs to its element
    resid = torch.zeros(T, M, dtype=dtype, device="cuda")
    resid[0, 1] = value
    y = dispatched(L, L["x"], resid)
    bound = 64512.0 if dtype == torch.float16 else torch.finfo(dtype).max      # 64504 as fp16
    assert torch.isnan(y[0, 1]) if value != value else y[0, 1].item() == bound
    y[0, 1] = 0
    clean = dispatched(L, L["x"], torch.zeros_like(resid))
    clean[0, 1] = 0
    assert torch.equal(y, clean)
