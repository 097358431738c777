"""The native host path of the modules against the general route, which serves every call it does not take."""
import sys

import pytest
import torch

from oracle import nanoquant_oracle as oc
from tests.util import exact_np

pytestmark = pytest.mark.gpu


def _module(N, R, M, dtype, kernel, bias, seed):
    from nanoquant_b200.modules.linear import NanoQuantLinear
    d = oc.synth_linear(N, R, M, 1, seed=seed)
    t = lambda a: torch.from_numpy(a)
    m = NanoQuantLinear(N, M, R)
    if bias:
        m.bias = torch.nn.Parameter(torch.linspace(-1, 1, M).to(dtype).cuda(), requires_grad=False)
    s = lambda k: t(d[k]).float().to(dtype)
    m.load_packed(t(oc.pack_rows(d["V"], "lsb_first")), (R, N), t(oc.pack_rows(d["U"], "lsb_first")), (M, R), s("s_pre"),
                  s("s_post"), s("s_mid"), dtype=dtype, kernel_type=kernel)
    return m, d


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kernel,bias", [("gemv", False), ("gemv", True), ("gemm", False), ("gemm", True)])
@pytest.mark.parametrize("lead", [(1,), (3, 1), (2, 17)])
def test_module_call_equals_the_general_route(dtype, kernel, bias, lead):
    from nanoquant_b200 import _lib, ops
    m, d = _module(256, 96, 200, dtype, kernel, bias, seed=5)
    x = torch.randn(*lead, 256, device="cuda").to(dtype)
    ops_of = m.launch_operands()
    assert _lib.ext().linear_forward(x, *ops_of) is not None          # the native path takes this call
    want = ops.linear_forward(x.reshape(-1, 256), *ops_of[:6], bias=ops_of[6]).view(*lead, 200)
    assert torch.equal(m(x), want)
    # calls it leaves alone: other dtype, a strided input, a residual of another type
    assert _lib.ext().linear_forward(x.float(), *ops_of) is None
    assert torch.equal(m(x.float()).to(dtype), want)
    wide = torch.zeros(*lead, 512, device="cuda", dtype=dtype)
    wide[..., ::2] = x
    assert torch.equal(m(wide[..., ::2]), want)
    y64 = oc.forward_fp64(exact_np(x.reshape(-1, 256)), d["V"], d["U"], *[exact_np(t) for t in (ops_of[0], ops_of[2], ops_of[4])],
                          **({"bias": exact_np(ops_of[6])} if bias else {}))
    assert oc.rel_err(exact_np(want.reshape(-1, 200)), y64) <= 2e-3 + 2.0 ** -8


@pytest.mark.parametrize("T", [1, 4, 5, 33])
def test_group_call_equals_the_general_route(T):
    from nanoquant_b200 import ops
    from nanoquant_b200.modules.group import LinearGroup
    mods = [_module(256, 96, M, torch.bfloat16, "gemv", M == 64, seed=M)[0] for M in (200, 64)]
    x = torch.randn(T, 256, device="cuda").to(torch.bfloat16)
    res = [torch.randn(T, 200, device="cuda").to(torch.bfloat16), None]
    lay = [m.launch_operands() for m in mods]
    for r in (None, res):
        want = ops.group_forward([x, x], [a[:6] for a in lay], T, torch.bfloat16, x.device, [a[6] for a in lay], r)
        got = LinearGroup(mods)(x.view(T, 1, 256), residuals=r)
        assert [tuple(y.shape) for y in got] == [(T, 1, 200), (T, 1, 64)]
        assert all(torch.equal(a.reshape(T, -1), b) for a, b in zip(got, want))


def test_call_keeps_hooks_and_overrides():
    # the module's own __call__ passes a call on unless nothing could notice: hooks of every kind, a replaced forward, a subclass's forward
    from torch.nn.modules.module import register_module_forward_hook
    from nanoquant_b200.modules.linear import NanoQuantLinear
    m, _ = _module(256, 96, 200, torch.bfloat16, "gemv", False, seed=5)
    x = torch.randn(3, 256, device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        want = m.forward(x)
        assert torch.equal(m(x), want) and torch.equal(m(x=x), want)
        seen = []
        for register in (m.register_forward_hook, m.register_forward_pre_hook, register_module_forward_hook):
            handle = register(lambda *a: seen.append(register.__name__))
            m(x)
            handle.remove()
        assert len(seen) == 3
        handle = m.register_forward_hook(lambda mod, args, y: y + 1)
        assert torch.equal(m(x), want + 1)
        handle.remove()
        m.forward = lambda x: "replaced"
        assert m(x) == "replaced"
        del m.forward
        with pytest.MonkeyPatch.context() as patch:
            patch.setattr(NanoQuantLinear, "forward", lambda self, x: "patched")
            assert m(x) == "patched"
        assert torch.equal(m(x), want)
        m.__class__ = type("Sub", (NanoQuantLinear,), {"forward": lambda self, x: "subclass"})
        assert m(x) == "subclass"


@pytest.mark.parametrize("kernel,bias", [("gemv", True), ("gemm", False)])
def test_call_holds_its_operands(kernel, bias):
    # A module's operands may be replaced by another thread while a call is under way without the GIL.  Python code that the call itself
    # runs (growing the scratch) stands in for the thread here: it counts the references, and replaces the operands where they are held.
    from nanoquant_b200 import _lib, ops
    m, _ = _module(256, 96, 200, torch.bfloat16, kernel, bias, seed=5)
    x = torch.randn(3, 256, device="cuda").to(torch.bfloat16)
    ext, buf = _lib.ext(), ops.reserve_scratch(x.device, 256)
    places = [(m._parameters, n) for n in ("scale_pre", "scale_mid", "scale_post", "s1", "s2", "s3", "bias")] + [(m.__dict__, "V_int8"), (m.__dict__, "U_int8")]
    places = [(d, n) for d, n in places if d.get(n) is not None]
    count = lambda: [sys.getrefcount(d[n]) for d, n in places]
    before, during = count(), []
    want = m(x)
    assert count() == before                                         # and gives them back

    def grow(idx, nbytes):
        during.extend(count())
        if all(b > a for a, b in zip(before, during)):
            for d, n in places:
                d[n] = torch.zeros_like(d[n])
        ext.set_scratch(idx, buf.data_ptr(), buf.numel())

    ext.set_callbacks(_lib.check, grow, ops._nanoquant_dyn_forward_cuda, ops._marlin_nanoquant_forward_cuda)
    try:
        ext.set_scratch(x.device.index or 0, buf.data_ptr(), 0)      # too small: the call asks for more
        y = m(x)
    finally:
        ops.connect_host_path(ext)
    assert len(places) == 5 + bias and len(during) == len(places)
    assert all(b > a for a, b in zip(before, during)), (before, during)
    assert torch.equal(y, want)
    assert not torch.equal(m(x), want)                               # the operands are the replaced ones from the next call on


@pytest.mark.parametrize("kernel,bias", [("gemv", False), ("gemm", False), ("gemv", True)])
def test_tensors_with_more_than_a_memory(kernel, bias):
    # wrappers of transforms, lazily negated tensors and calls that autograd records go to the operator (or are resolved first)
    from nanoquant_b200.modules.group import LinearGroup
    m, _ = _module(256, 96, 200, torch.bfloat16, kernel, bias, seed=5)
    x = torch.randn(3, 2, 256, device="cuda").to(torch.bfloat16)
    want = torch.stack([m(a) for a in x])
    neg = torch.stack([m(-a) for a in x])
    for a, y in zip(x, neg):
        assert torch.equal(m(torch._neg_view(a)), y)
        assert torch.equal(m.forward(torch._neg_view(a)), y)
        assert torch.equal(LinearGroup([m])(torch._neg_view(a))[0], y)
    if bias:
        return                                     # (behind a bias there is no operator)
    if kernel == "gemv":                           # (the other operator may write its workspace, which transforms refuse)
        assert torch.equal(torch.vmap(m)(x), want)
        assert torch.equal(torch.func.functionalize(m)(x[0]), want[0])
        assert not torch.func.grad(lambda a: m(a).float().sum())(x[0]).any()      # (no derivative; the value is computed)
    xg = x[0].clone().requires_grad_()
    assert m(xg).requires_grad and torch.equal(m(xg), want[0])
    with torch.no_grad():
        assert not m(xg).requires_grad


def test_lazily_negated_operands_elsewhere():
    from nanoquant_b200 import ops
    from nanoquant_b200.kernel import utils as ku
    x, w = torch.randn(3, 256, device="cuda").half(), torch.randn(40, 256, device="cuda").half()
    for a, b in ((torch._neg_view(x), w), (x, torch._neg_view(w))):
        assert torch.equal(ops.dense_gemv_forward(a, b), ops.dense_gemv_forward(-x, w))
    s = (torch.randint(0, 2, (64, 96), device="cuda") * 2 - 1).to(torch.int8)
    assert torch.equal(ku.pack_binary_gemv(torch._neg_view(s)), ku.pack_binary_gemv(-s))
    for got, want in zip(ku.pack_binary_marlin(torch._neg_view(s), torch._neg_view(x[0, :96]), x[0, :64]),
                         ku.pack_binary_marlin(-s, -x[0, :96], x[0, :64])):
        assert torch.equal(got, want) if torch.is_tensor(want) else got == want


def test_call_is_seen_by_whoever_watches_module_calls(tmp_path):
    from nanoquant_b200.modules import linear
    from nanoquant_b200.modules.linear import NanoQuantLinear
    m, _ = _module(256, 96, 200, torch.bfloat16, "gemv", False, seed=5)
    x = torch.randn(3, 256, device="cuda").to(torch.bfloat16)
    want, seen = m(x), []
    assert linear.module_class()[3:5] == (torch.nn.Module.__call__, torch.nn.Module._call_impl)      # (unwatched: the short way)

    def watched(f):
        def call(self, *args, **kwargs):
            seen.append(type(self))
            return f(self, *args, **kwargs)
        return call

    for cls, name in ((torch.nn.Module, "__call__"), (torch.nn.Module, "_call_impl"), (NanoQuantLinear, "_call_impl")):
        with pytest.MonkeyPatch.context() as patch:
            patch.setattr(cls, name, watched(getattr(cls, name)))
            assert torch.equal(m(x), want)
    m._call_impl = lambda *args: (seen.append(NanoQuantLinear), NanoQuantLinear._call_impl(m, *args))[1]
    assert torch.equal(m(x), want)
    del m._call_impl
    assert seen == 4 * [NanoQuantLinear] and torch.equal(m(x), want) and len(seen) == 4
    # torch.profiler's module tree
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CPU], with_stack=True) as prof:
        assert torch.equal(m(x), want)
    prof.export_chrome_trace(str(tmp_path / "trace.json"))
    assert "nn.Module: NanoQuantLinear" in (tmp_path / "trace.json").read_text()
