"""When the differentiable projection keeps its path integrals: small ones without
asking the driver for the free memory, others by it, an explicit limit as is."""
from types import SimpleNamespace

import torch

from virtualcbct_b200 import autograd


def test_keep_asks_for_free_memory_only_above_the_small_share(monkeypatch):
    total, asked = 180 << 30, []
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d: SimpleNamespace(total_memory=total))
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda: asked.append(1) or (4 << 30, total))
    assert autograd._keep(total // autograd.SMALL_SHARE, None) and not asked
    assert autograd._keep(1 << 30, None) and len(asked) == 1
    assert not autograd._keep((1 << 30) + 1, None) and len(asked) == 2
    assert not autograd._keep(1, 0) and autograd._keep(1, 1) and len(asked) == 2


def test_keep_on_a_nearly_full_device(monkeypatch):
    """Small path integrals are not held where a quarter of the free memory is
    less, unless torch holds the step's memory already."""
    total, asked, held = 180 << 30, [], {}
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d: SimpleNamespace(total_memory=total))
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda: asked.append(1) or (16 << 20, total))
    monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", lambda: held)
    n = 100 << 20
    assert not autograd._keep(n, None) and len(asked) == 1  # nothing held: the allocator has not run
    held.update(reserved_bytes={"all": {"current": 10 * n}}, allocated_bytes={"all": {"current": 7 * n}})
    assert autograd._keep(n, None, 2 * n) and len(asked) == 1
    assert not autograd._keep(n, None, 2 * n + 1) and len(asked) == 2
