"""What the operators' native host path takes as it is, and what it leaves to the general path."""
from types import SimpleNamespace

import pytest
import torch

from deltanet_b200 import _lib
from deltanet_b200.gdn2 import _require_cuda


@pytest.fixture(scope="module")
def host():
    return _lib.host()


# ---- tensors of one call are on one device
def test_plain_asks_for_one_device(host):
    q = torch.zeros(4, 8)
    assert host.plain(torch.zeros(2, 2), q) and host.plain(torch.zeros(3, dtype=torch.int32), q)
    assert not host.plain(torch.zeros(4, 8, device="meta"), q)
    assert not host.plain(q, torch.zeros(4, 8, device="meta"))
    assert not host.plain(torch.zeros(8, 4).t(), q)


def test_general_path_refuses_other_devices():
    on = lambda d: SimpleNamespace(is_cuda=d.startswith("cuda"), device=torch.device(d))
    _require_cuda(on("cuda:1"), None, on("cuda:1"))
    with pytest.raises(RuntimeError, match="must be on one device, got cuda:0 and cuda:1"):
        _require_cuda(on("cuda:0"), on("cuda:0"), on("cuda:1"))
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        _require_cuda(on("cuda:0"), on("cpu"))


@pytest.mark.gpu
@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_ids_of_another_gpu_are_moved():
    import deltanet_b200 as dn
    gen = torch.Generator().manual_seed(3)
    t = [torch.randn(1, 96, 2, 64, generator=gen).cuda() for _ in range(3)] + [-torch.rand(1, 96, 2, generator=gen).cuda() for _ in range(3)]
    seg = (torch.arange(96) > 40).int()[None]
    cu = torch.tensor([0, 41, 96], dtype=torch.int32)
    ref = dn.chunk_gdn2(*t, segment_ids=seg.cuda())
    assert torch.equal(dn.chunk_gdn2(*t, segment_ids=seg.to("cuda:1")), ref)
    assert torch.equal(dn.chunk_gdn2(*t, cu_seqlens=cu.to("cuda:1")), ref)
    with pytest.raises(RuntimeError, match="one device"):
        dn.chunk_gdn2(*t[:5], t[5].to("cuda:1"))


# ---- what follows a call: autograd's other modes, transforms, tracing, dispatch modes
def test_wrapped_tensors_are_not_plain(host):
    q = torch.randn(2, 3)
    assert not host.plain(torch._neg_view(q), q)
    seen = []
    torch.vmap(lambda t: (seen.append(host.plain(t, q)), t)[1])(q[None])
    torch.func.grad(lambda t: (seen.append(host.plain(t, q)), t.sum())[1])(q)
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode() as m:
        seen.append(host.plain(m.from_tensor(q), q))
    assert seen == [False] * 3


def test_bare_calls(host):
    import torch.autograd.forward_ad as fwd
    t, p = torch.randn(3), torch.randn(3, requires_grad=True)
    assert host.bare(t, None, t) and not host.bare(t, p)
    with torch.no_grad():
        assert host.bare(t, p)
    with fwd.dual_level():
        assert not host.bare(fwd.make_dual(t, t))
    from torch.utils._python_dispatch import TorchDispatchMode

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, f, types, args=(), kwargs=None):
            return f(*args, **(kwargs or {}))
    with Mode():
        assert not host.bare(t)
    seen = []
    torch.jit.trace(lambda x: (seen.append(host.bare(x)), x * 2)[1], (t,), check_trace=False)
    assert seen == [False]


def _inputs(seed, grad=False):
    gen = torch.Generator().manual_seed(seed)
    t = [torch.randn(1, 96, 2, 64, generator=gen) for _ in range(3)]
    t += [-torch.rand(1, 96, 2, 64, generator=gen), torch.rand(1, 96, 2, 64, generator=gen), torch.rand(1, 96, 2, 64, generator=gen)]
    return [x.cuda().requires_grad_(grad) for x in t]


@pytest.fixture(scope="module")
def fn():
    import deltanet_b200 as dn
    return lambda *t: dn.chunk_gdn2(*t, precision="fp32", qk_l2norm=True)


@pytest.mark.gpu
@pytest.mark.parametrize("grad", [False, True])
def test_tangents_are_refused(fn, grad):
    import torch.autograd.forward_ad as fwd
    t = _inputs(1, grad)
    with fwd.dual_level(), pytest.raises(NotImplementedError, match="jvp"):
        fn(fwd.make_dual(t[0], torch.randn_like(t[0])), *t[1:])


@pytest.mark.gpu
def test_transforms_and_fakes_are_refused(fn):
    t = _inputs(2)
    for f in (lambda: torch.func.grad(lambda q: fn(q, *t[1:]).sum())(t[0]), lambda: torch.func.jvp(lambda q: fn(q, *t[1:]), (t[0],), (t[0],)),
              lambda: torch.vmap(lambda q: fn(q, *t[1:]))(torch.stack([t[0]] * 2))):
        with pytest.raises(RuntimeError, match="functorch transforms"):
            f()
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode() as m, pytest.raises(RuntimeError, match="no memory of its own"):
        fn(*[m.from_tensor(x) for x in t])


@pytest.mark.gpu
def test_trace_follows_its_inputs(fn):
    t, u = _inputs(3), _inputs(4)
    f = torch.jit.trace(lambda *x: fn(*x) * 2, tuple(t), check_trace=False)
    assert torch.equal(f(*u), fn(*u) * 2)


@pytest.mark.gpu
def test_saved_tensor_hooks_see_the_inputs_only(fn):
    t = _inputs(5, True)
    ref = torch.autograd.grad(fn(*t).sum(), t)
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda x: (seen.append(x.dtype), x)[1], lambda x: x):
        out = fn(*t)
    got = torch.autograd.grad(out.sum(), t, retain_graph=True)
    again = torch.autograd.grad(out.sum(), t)
    assert seen == [torch.float32] * 6
    assert all(torch.equal(x, y) and torch.equal(x, z) for x, y, z in zip(ref, got, again))


@pytest.mark.gpu
def test_sign_views(fn):
    t = _inputs(6)
    assert torch.equal(fn(torch._neg_view(t[0]), *t[1:]), fn(-t[0], *t[1:]))


# ---- addresses: rows are moved 16 bytes at a time
def test_odd_offsets_are_copied(host):
    flat = torch.arange(33, dtype=torch.float32)
    even, odd = flat[:32].view(4, 8), flat[1:].view(4, 8)
    assert host.aligned(even) is even and host.plain(odd, even)
    got = host.aligned(odd)
    assert got.data_ptr() % 16 == 0 and torch.equal(got, odd)


@pytest.mark.parametrize("K,V", [(64, 64), (128, 128)])
def test_misaligned_buffers_get_a_status(K, V):
    """No address here is ever read: the status comes before anything is enqueued."""
    lib, at = _lib.lib(), 1 << 20
    s = _lib.Shape(B=1, L=64, Hk=1, Hv=1, K=K, V=V, chunk=128, g_heads=1, g_cols=K, b_heads=1, b_cols=K, w_heads=1, w_cols=V,
                   qkv_dtype=_lib.DN_BF16, gate_dtype=_lib.DN_F32, precision=_lib.DN_PREC_BF16, flags=0, scale=1.0)
    res = _lib.Residuals()
    for odd in range(8):
        a = [at + (2 if i == odd else 0) for i in range(8)]
        assert lib.dn_chunk_fwd(s, *a[:6], None, None, a[6], None, None, a[7], 1 << 30, None) == 9
    assert lib.dn_residual_carve(s, at + 8, res) == 0
    assert lib.dn_prepass_fwd(s, *[at] * 6, None, res, at, 1 << 30, None) == 9
    assert lib.dn_prepass_fwd_static(s, *[at] * 6, None, res, None) == 9
    assert lib.dn_state_bwd(s, res, None, at, None, at, at, None, None) == 9
    for odd in range(14):
        a = [at + (2 if i == odd else 0) for i in range(14)]
        assert lib.dn_chunk_bwd(s, *a[:6], None, None, None, a[6], None, *a[7:13], None, a[13], 1 << 30, None) == 9
    d = _lib.DecodeShape(B=1, Hk=1, Hv=1, K=K, V=V, g_heads=1, g_cols=1, b_heads=1, b_cols=1, w_heads=1, w_cols=1, qkv_dtype=_lib.DN_F32,
                         gate_dtype=_lib.DN_F32, state_in_dtype=_lib.DN_F32, state_out_dtype=_lib.DN_F32, flags=0, scale=1.0, stability_tau=1.0)
    for i, o in ((at + 4, at), (at, at + 8)):
        assert lib.dn_decode_step(d, *[at] * 6, i, None, at, o, None) == 9


def _offset(t):
    return torch.cat([t.new_zeros(1), t.detach().reshape(-1)])[1:].view(t.shape)


@pytest.mark.gpu
@pytest.mark.parametrize("K,V,dtype,precision", [(64, 64, torch.bfloat16, "bf16"), (128, 128, torch.bfloat16, "bf16"), (64, 64, torch.float32, "fp32")])
def test_offset_views_give_the_same(K, V, dtype, precision):
    import deltanet_b200 as dn
    gen = torch.Generator().manual_seed(9)
    r = lambda *s: torch.rand(*s, generator=gen)
    t = [(r(1, 200, 2, n) - 0.5).to(dtype).cuda() for n in (K, K, V)] + [-r(1, 200, 2, K).cuda(), r(1, 200, 2, K).cuda(), r(1, 200, 2, V).cuda()]
    cot = (r(1, 200, 2, V) - 0.5).to(dtype).cuda()
    res = []
    for leaves, d in ((t, cot), ([_offset(x) for x in t], _offset(cot))):
        leaves = [x.detach().requires_grad_() for x in leaves]
        out = dn.chunk_gdn2(*leaves, precision=precision, qk_l2norm=True)
        res.append((out,) + torch.autograd.grad(out, leaves, d))
    assert all(torch.equal(x, y) for x, y in zip(*res))
    tok, state = [x[:, 0].contiguous() for x in t], r(1, 2, K, V).cuda()
    one = dn.gdn2_decode_step(*tok, state)
    two = dn.gdn2_decode_step(*tok, _offset(state))
    assert all(torch.equal(x, y) for x, y in zip(one, two))
    two = dn.gdn2_decode_step(*[_offset(x) for x in tok], state)          # the other decode kernel: sums of K in another order
    for x, y in zip(one, two):                                            # (fp32, or one rounding of the outputs to bf16)
        assert float((x.float() - y.float()).norm() / x.float().norm()) < (1e-2 if x.dtype == torch.bfloat16 else K * 2.0 ** -24)
    with pytest.raises(ValueError, match="multiple of 16 bytes"):
        dn.gdn2_decode_step(*tok, state, out_state=_offset(state))


@pytest.mark.gpu
def test_offset_views_of_the_layer_steps():
    import deltanet_b200 as dn
    gen = torch.Generator().manual_seed(10)
    x, w = torch.randn(1, 50, 256, generator=gen).cuda(), torch.randn(256, 4, generator=gen).cuda()
    o, z, n = torch.randn(1, 50, 2, 64, generator=gen).cuda(), torch.randn(1, 50, 2, 64, generator=gen).cuda(), torch.ones(64).cuda()
    kw = dict(num_k_heads=1, num_v_heads=2, head_k_dim=64, head_v_dim=64)
    assert all(torch.equal(a, b) for a, b in zip(dn.gdn_qkv_producer(x, w, **kw), dn.gdn_qkv_producer(_offset(x), w, **kw)))
    assert torch.equal(dn.gated_rmsnorm(o, z, n), dn.gated_rmsnorm(_offset(o), _offset(z), n))


# ---- other Python threads run while a call is enqueued
@pytest.mark.gpu
def test_calls_are_enqueued_without_the_interpreter_lock(host, fn):
    """PyGILState_Check, 1 where the calling thread holds the lock, stands in for the entry points: its answer is their status."""
    import ctypes as C
    import deltanet_b200 as dn
    lib, held = _lib.lib(), C.cast(C.pythonapi.PyGILState_Check, C.c_void_p).value
    real = {n: C.cast(getattr(lib, n), C.c_void_p).value for n in _lib._HOST_USES}
    t, token = _inputs(11, True), [x[:, 0].contiguous() for x in _inputs(12)]
    host.bind(dict(real, dn_decode_step=held, dn_chunk_fwd=held, dn_chunk_bwd=held))
    try:
        dn.gdn2_decode_step(*token, torch.zeros(1, 2, 64, 64, device="cuda"))
        torch.autograd.grad(fn(*t).sum(), t)
        wide = [torch.stack([x, x], -1)[..., 0] for x in t]                 # the general path
        torch.autograd.grad(fn(*wide).sum(), t)
    finally:
        host.bind(real)
