"""The tag that marks the decode kernel's intermediate as this launch's: NaNs that a GEMM stage leaves in the shared scratch
(0x7FFF as bf16 and fp16) must not look like one, whatever the launch count."""
import pytest
import torch

from tests.util import assert_parity, exact_np, make_layer, tiles_on_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [0, 0xF7FFF, 0xFFFFF, 0x7FFFF])
def test_stored_nans_are_not_tags(count):
    from nanoquant_b200 import _lib
    Lb = _lib.lib()
    T, N, R, M = 1, 4096, 608, 1024
    L = make_layer(N, R, M, T, torch.bfloat16, seed=2)
    vt, ut = tiles_on_gpu(L["V"]), tiles_on_gpu(L["U"])
    st = torch.cuda.current_stream().cuda_stream
    nb = Lb.nq_gemv_scratch_bytes(T, N, R, M)
    scratch = torch.zeros(nb, dtype=torch.uint8, device="cuda")
    scratch.view(torch.int32)[64:] = 0x7FFF7FFF         # the intermediate of a GEMM whose token had a NaN
    scratch.view(torch.int64)[0] = count * 1024         # launches so far: an earlier form of the tag made 0xF7FFF that word
    y = torch.empty(T, M, dtype=torch.bfloat16, device="cuda")
    for _ in range(2):
        _lib.check(Lb.nq_gemv_fwd(L["x"].data_ptr(), L["s_pre"].data_ptr(), vt.data_ptr(), L["s_mid"].data_ptr(), ut.data_ptr(),
                                  L["s_post"].data_ptr(), y.data_ptr(), scratch.data_ptr(), nb, T, N, R, M, _lib.NQ_BF16, st),
                   "nq_gemv_fwd")
        assert Lb.nq_scratch_status(scratch.data_ptr(), st) == 0
        assert_parity(exact_np(y), L["y64"], torch.bfloat16, what=f"launch count {count:#x}")
    assert scratch.view(torch.int64)[0].item() == (count + 2) * 1024
