"""Decode kernel at the edges of its tiles: row groups of 16, chunks of 256 columns, row blocks that do not fit shared
memory at once, one to four tokens; and a CTA that computes the rows it has polled for in vain."""
import pytest
import torch

from tests.util import assert_parity, exact_np, make_layer, tiles_on_gpu

pytestmark = pytest.mark.gpu


def _run(L, T, N, R, M, dtype, offset=0):
    from nanoquant_b200 import _lib
    Lb = _lib.lib()
    st = torch.cuda.current_stream().cuda_stream
    nb = Lb.nq_gemv_scratch_bytes(T, N, R, M)
    room = torch.zeros(nb + offset + 64, dtype=torch.uint8, device="cuda")
    scratch = room[offset:offset + nb]
    y = torch.full((T, M), float("nan"), dtype=dtype, device="cuda")
    vt, ut = tiles_on_gpu(L["V"]), tiles_on_gpu(L["U"])
    args = (L["x"].data_ptr(), L["s_pre"].data_ptr(), vt.data_ptr(), L["s_mid"].data_ptr(), ut.data_ptr(),
            L["s_post"].data_ptr(), y.data_ptr(), scratch.data_ptr(), nb, T, N, R, M,
            _lib.NQ_BF16 if dtype == torch.bfloat16 else _lib.NQ_F16, st)
    _lib.check(Lb.nq_gemv_fwd(*args), "nq_gemv_fwd")
    first = y.clone()
    for _ in range(3):
        _lib.check(Lb.nq_gemv_fwd(*args), "nq_gemv_fwd")
    torch.cuda.synchronize()
    assert Lb.nq_scratch_status(scratch.data_ptr(), st) == 0
    assert torch.equal(first, y)
    assert not room[:offset].any() and not room[offset + nb:].any()
    return y, scratch.view(torch.int32)[3].item()       # result, number of CTAs that computed others' rows


@pytest.mark.parametrize("T", [1, 2, 3, 4])
@pytest.mark.parametrize("N,R,M", [
    (8, 1, 1), (255, 15, 17), (256, 16, 16), (257, 17, 15), (264, 33, 500), (2056, 520, 96),
    (4104, 264, 4100),          # 17 chunks of input, more of them than warps
    (16640, 40, 24),            # 65 chunks
    (512, 4112, 40000),         # many row groups per CTA: several row blocks
])
def test_tile_edges(N, R, M, T):
    dtype = torch.bfloat16 if T % 2 or N < 200 else torch.float16     # (eight columns: outputs below fp16's normal range)
    L = make_layer(N, R, M, T, dtype, seed=N + R + M)
    y, _ = _run(L, T, N, R, M, dtype)
    assert_parity(exact_np(y), L["y64"], dtype, what=f"N={N} R={R} M={M} T={T}")


@pytest.mark.parametrize("T", [1, 2, 3, 4])
@pytest.mark.parametrize("N,R,M", [(256, 16, 16), (1003, 333, 777)])
def test_scratch_between_two_multiples_of_32(N, R, M, T):
    # 16 bytes are what the scratch has to be aligned to; the intermediate is loaded in 32
    L = make_layer(N, R, M, T, torch.bfloat16, seed=3)
    want, _ = _run(L, T, N, R, M, torch.bfloat16)
    y, _ = _run(L, T, N, R, M, torch.bfloat16, offset=16)
    assert torch.equal(y, want)


@pytest.mark.parametrize("T", [1, 4])
@pytest.mark.parametrize("N,R,M", [(1003, 333, 777), (4096, 608, 1024), (32768, 64, 4096)])
def test_rows_polled_for_in_vain_are_computed(N, R, M, T):
    # a short wait limit makes a CTA compute the other CTAs' rows soon after its first failed poll: same bits
    from nanoquant_b200 import _lib
    Lb = _lib.lib()
    L = make_layer(N, R, M, T, torch.float16, seed=7)
    want, _ = _run(L, T, N, R, M, torch.float16)
    # help comes after 1/16 of the limit: after the second poll in vain
    old = Lb.nq_gemv_set_wait_limit(31)
    try:
        helpers = 0
        for _ in range(4):
            y, h = _run(L, T, N, R, M, torch.float16)
            assert torch.equal(y, want)
            helpers += h
        # four row groups of 128 chunks: most CTAs have no row of the intermediate and poll while four compute it
        assert helpers > 0 or N != 32768
    finally:
        Lb.nq_gemv_set_wait_limit(old)
