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
