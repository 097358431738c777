"""Bounded device-side waits, made to run out without faulting or hanging anything: a wait that nothing will
ever satisfy returns after its (shortened) limit, the host reads NQ_ERR_TIMEOUT from the status word, and the
next call after re-zeroing works."""
import pytest
import torch

from tests.util import assert_parity, exact_np, gemm_kernels, make_group, make_layer, tiles_on_gpu

pytestmark = pytest.mark.gpu


def test_gemv_wait_for_a_stale_intermediate_expires():
    # The launch tag of a scratch is its launch count.  A header whose counter says "launch 5" while the buffer
    # holds no element with that tag is what a consumer sees when a producer never writes: here the producers DO
    # write, so to make a wait run out the status word is pre-set instead, which turns every wait of the launch
    # into a single poll (sticky expiry); the status stays set, and re-zeroing restores normal operation.
    from nanoquant_b200 import _lib
    Lb = _lib.lib()
    T, N, R, M = 1, 1024, 256, 512
    L = make_layer(N, R, M, T, torch.float16, seed=1)
    vt, ut = tiles_on_gpu(L["V"]), tiles_on_gpu(L["U"])
    st = torch.cuda.current_stream().cuda_stream
    nb = Lb.nq_gemv_scratch_bytes(T, N, R, M)
    scratch = torch.zeros(nb, dtype=torch.uint8, device="cuda")
    y = torch.empty(T, M, dtype=torch.float16, device="cuda")
    args = (L["x"].data_ptr(), L["s_pre"].data_ptr(), vt.data_ptr(), L["s_mid"].data_ptr(), ut.data_ptr(),
            L["s_post"].data_ptr(), y.data_ptr(), scratch.data_ptr(), nb, T, N, R, M, _lib.NQ_F16, st)
    old = Lb.nq_gemv_set_wait_limit(64)          # a few dozen polls instead of four million
    try:
        scratch.view(torch.int32)[2] = 7         # an earlier expiry left its mark: this launch must not spin
        _lib.check(Lb.nq_gemv_fwd(*args), "nq_gemv_fwd")
        torch.cuda.synchronize()
        assert Lb.nq_scratch_status(scratch.data_ptr(), st) != 0
        scratch.zero_()
        _lib.check(Lb.nq_gemv_fwd(*args), "nq_gemv_fwd")
        assert Lb.nq_scratch_status(scratch.data_ptr(), st) == 0
        assert_parity(exact_np(y), L["y64"], torch.float16, what="after re-zeroing")
    finally:
        assert Lb.nq_gemv_set_wait_limit(old) == 64


def test_gemv_wait_that_runs_out():
    # Four row groups of 128 chunks each: four CTAs produce the intermediate while the others poll for it from the start.
    # With a limit of one poll in vain, too small for a CTA to help, their wait runs out long before the rows are there.
    from nanoquant_b200 import _lib
    Lb = _lib.lib()
    T, N, R, M = 1, 32768, 64, 4096
    L = make_layer(N, R, M, T, torch.float16, seed=3)
    vt, ut = tiles_on_gpu(L["V"]), tiles_on_gpu(L["U"])
    st = torch.cuda.current_stream().cuda_stream
    nb = Lb.nq_gemv_scratch_bytes(T, N, R, M)
    scratch = torch.zeros(nb, dtype=torch.uint8, device="cuda")
    y = torch.empty(T, M, dtype=torch.float16, device="cuda")
    args = (L["x"].data_ptr(), L["s_pre"].data_ptr(), vt.data_ptr(), L["s_mid"].data_ptr(), ut.data_ptr(),
            L["s_post"].data_ptr(), y.data_ptr(), scratch.data_ptr(), nb, T, N, R, M, _lib.NQ_F16, st)
    old = Lb.nq_gemv_set_wait_limit(1)
    try:
        _lib.check(Lb.nq_gemv_fwd(*args), "nq_gemv_fwd")
        assert Lb.nq_scratch_status(scratch.data_ptr(), st) == _lib.NQ_ERR_TIMEOUT
        assert scratch.view(torch.int32)[3].item() == 0                 # nobody helped
    finally:
        Lb.nq_gemv_set_wait_limit(old)
    _lib.check(Lb.nq_gemv_fwd(*args), "nq_gemv_fwd")
    assert Lb.nq_scratch_status(scratch.data_ptr(), st) == _lib.NQ_ERR_TIMEOUT     # stays until the scratch is zeroed
    scratch.zero_()
    _lib.check(Lb.nq_gemv_fwd(*args), "nq_gemv_fwd")
    assert Lb.nq_scratch_status(scratch.data_ptr(), st) == 0
    assert_parity(exact_np(y), L["y64"], torch.float16, what="after re-zeroing")


def test_allgather_wait_for_an_absent_peer_expires():
    # world = 2 on one GPU, both "ranks" pointing at this process's buffer; slot 1's flag is never written, so the
    # wait for rank 1 runs out: the kernel returns, the status says so, and after re-zeroing a world of 1 works.
    from nanoquant_b200 import _lib
    import ctypes
    Lb = _lib.lib()
    if not hasattr(Lb, "nq_allgather_set_wait_limit"):
        pytest.skip("library without a run-time limit for the all-gather wait")
    st = torch.cuda.current_stream().cuda_stream
    shard = torch.arange(64, dtype=torch.float16, device="cuda")
    buf = torch.zeros(4096, dtype=torch.uint8, device="cuda")
    state = torch.zeros(Lb.nq_allgather_state_bytes(), dtype=torch.uint8, device="cuda")
    bases = (ctypes.c_void_p * 2)(buf.data_ptr(), buf.data_ptr())
    old = Lb.nq_allgather_set_wait_limit(2000)
    try:
        rc = Lb.nq_allgather_push(shard.data_ptr(), shard.numel() * 2, bases, 0, 1024, state.data_ptr(), 2, 0, st)
        _lib.check(rc, "nq_allgather_push")
        torch.cuda.synchronize()
        assert Lb.nq_allgather_status(state.data_ptr(), st) == _lib.NQ_ERR_TIMEOUT
        buf.zero_(); state.zero_()
        bases1 = (ctypes.c_void_p * 1)(buf.data_ptr())
        _lib.check(Lb.nq_allgather_push(shard.data_ptr(), shard.numel() * 2, bases1, 0, 1024, state.data_ptr(), 1, 0, st), "push")
        assert Lb.nq_allgather_status(state.data_ptr(), st) == 0
        assert torch.equal(buf[1024:1024 + 128].view(torch.float16), shard)
    finally:
        Lb.nq_allgather_set_wait_limit(old)


@pytest.mark.parametrize("kernel,stage,T,shapes", [
    # a first stage of 98304 columns, 45 us: the second stage's CTAs, resident from the start, wait for it
    ("wgemm_kernel", 1, 128, [(98304, 256, 4096)]),
    # K split over two CTAs in the second stage: the second CTA of the linear of rank 256 has no columns, and owns the tokens from 16 on,
    # for which it waits in vain (the first one gave up behind the first stage)
    ("wgemm_kernel", 1, 32, [(98304, 512, 128), (98304, 256, 128)]),
    # the epilogue of a pair waits for a tile's main loop, 17 us
    ("pgemm_kernel", 0, 2048, [(4096, 2048, 256)]),
])
def test_gemm_wait_that_runs_out(kernel, stage, T, shapes):
    # With a limit of one attempt after the first (10 us in all), these waits run out; with 8 (4 for the last) they always did, too.
    # The launch ends all the same, drains what is in flight, gives its tensor memory back and reports; the next one on a zeroed scratch is right.
    from nanoquant_b200 import _lib
    Lb = _lib.lib()
    dtype = torch.float16
    layers = make_group(shapes, T, dtype, seed=T)
    keep, descs, ys = [], [], []
    for L in layers:
        vt, ut = tiles_on_gpu(L["V"]), tiles_on_gpu(L["U"])
        keep += [vt, ut]
        ys.append(torch.empty(T, L["M"], dtype=dtype, device="cuda"))
        descs.append(_lib.LinearDesc(L["x"].data_ptr(), L["s_pre"].data_ptr(), vt.data_ptr(), L["s_mid"].data_ptr(), ut.data_ptr(),
                                     L["s_post"].data_ptr(), ys[-1].data_ptr(), L["N"], L["R"], L["M"], L["N"], L["M"]))
    arr = (_lib.LinearDesc * len(descs))(*descs)
    st = torch.cuda.current_stream().cuda_stream
    scratch = torch.zeros(Lb.nq_gemm_group_scratch_bytes(arr, len(arr), T), dtype=torch.uint8, device="cuda")
    run = lambda: _lib.check(Lb.nq_gemm_group_fwd(arr, len(arr), T, _lib.NQ_F16, scratch.data_ptr(), scratch.numel(), st), "nq_gemm_group_fwd")
    status = lambda: Lb.nq_scratch_status(scratch.data_ptr(), st)
    assert gemm_kernels(shapes, T)[stage] == kernel
    run()
    assert status() == 0
    old = Lb.nq_gemm_set_wait_limit(1)
    try:
        ys[-1].fill_(7)
        run()
        assert status() == _lib.NQ_ERR_TIMEOUT
        if len(ys) > 1:                               # no CTA of this linear had all it needs: none stored anything
            assert (ys[-1] == 7).all()
    finally:
        assert Lb.nq_gemm_set_wait_limit(old) == 1
    run()
    assert status() == _lib.NQ_ERR_TIMEOUT            # stays until the scratch is zeroed
    scratch.zero_()
    run()
    assert status() == 0
    for L, y in zip(layers, ys):
        assert_parity(exact_np(y), L["y64"], dtype, what=f"{L['N']} columns")
