"""Dense block values through the quad map: every type code that is not 16-bit
means fp32, in the layout that was asked for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("code", ["F32", "I32", "NONE"])
@pytest.mark.parametrize("out_wide", [4, 8, 16])
def test_other_type_codes_are_fp32(cuda, code, out_wide):
    from att_gb300 import _lib, ops
    W, cols = 8, 32
    g = torch.Generator().manual_seed(out_wide)
    qmap = (torch.randperm(cols * W, generator=g) - cols * W // 4).clamp_min(-1).int()  # a quarter of the slots empty
    vals = torch.rand(2, cols * W, generator=g)
    out = torch.full((2, cols * W), float("nan"), device="cuda")
    q, v = qmap.cuda(), vals.cuda()
    _lib.call("att_gather_slot_values", ops._p(q), cols * W, W, 4, out_wide, ops._p(v), _lib.F32, cols * W, 1, 2,
              ops._p(out), getattr(_lib, code), cols * W, ops._stream())
    c, r = torch.meshgrid(torch.arange(cols), torch.arange(W), indexing="ij")
    e = qmap[(c - c % 4) * W + r * 4 + c % 4].long()
    want = torch.where(e >= 0, vals[:, e.clamp_min(0)], torch.zeros(()))
    assert torch.equal(out.cpu()[:, (c - c % out_wide) * W + r * out_wide + c % out_wide], want)
