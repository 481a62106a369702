"""Which slot maps the quad conversion hands to its kernel; every other one goes
through torch's own index arithmetic.  No GPU: stand-ins for the map."""
from types import SimpleNamespace

import pytest
import torch


def _map(device=0, n=8 * 16 * 3, dtype=torch.int32, shape=1, contiguous=True, address=1 << 20, cuda=True):
    return SimpleNamespace(is_cuda=cuda, device=SimpleNamespace(index=device), dtype=dtype, dim=lambda: shape,
                           is_contiguous=lambda: contiguous, numel=lambda: n, data_ptr=lambda: address)


@pytest.mark.parametrize("current", [0, 1])
def test_only_maps_on_the_current_device(monkeypatch, current):
    from att_gb300 import gat_ops
    monkeypatch.setattr(torch.cuda, "current_device", lambda: current)
    assert gat_ops._quad_kernel_takes(_map(current), 8, 16)
    assert not gat_ops._quad_kernel_takes(_map(1 - current), 8, 16)


def test_other_forms_take_the_general_path(monkeypatch):
    from att_gb300 import gat_ops
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    assert gat_ops._quad_kernel_takes(_map(), 8, 8)
    for kw in (dict(cuda=False), dict(dtype=torch.int64), dict(shape=2), dict(contiguous=False),
               dict(address=(1 << 20) + 4), dict(n=8 * 16 * 3 + 4)):
        assert not gat_ops._quad_kernel_takes(_map(**kw), 8, 16), kw
    assert not gat_ops._quad_kernel_takes(_map(n=8 * 6 * 4), 8, 6)  # not whole quads


@pytest.mark.parametrize("wide", [6, 8, 16])
def test_the_general_path(wide):
    """A map on the CPU: every slot (row, column) is found again in the quad layout."""
    from att_gb300 import gat_ops
    W, cols = 8, 48
    m = torch.randperm(cols * W).int()
    q = gat_ops.map_to_quad(m, W, wide)
    g, r = torch.meshgrid(torch.arange(cols), torch.arange(W), indexing="ij")
    assert torch.equal(q[(g - g % 4) * W + r * 4 + g % 4], m[(g - g % wide) * W + r * wide + g % wide])
