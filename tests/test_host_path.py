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
