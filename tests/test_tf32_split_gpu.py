"""The tf32 operands of the fp32 kernels: the tensor core reads an fp32 register
without its low 13 bits, so x and x - trunc(x) stand for the truncated pair."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F", [32, 100])
def test_operands_are_truncated(cuda, F):
    """Rows of one edge with a value of 1: the output is trunc(x) + trunc(x -
    trunc(x)), whose at most 24 significant bits are exact in fp32, for random
    bit patterns of every exponent, subnormals among them."""
    from att_gb300 import ops
    n = 2048
    rowptr, col = torch.arange(n + 1, dtype=torch.int32), torch.arange(n, dtype=torch.int32)
    f = ops.block_convert(rowptr, col, torch.ones(n, dtype=torch.float32), wide=4)
    g = torch.Generator().manual_seed(F)
    bits = torch.randint(0, 1 << 31, (n, F), generator=g) % (254 << 23) + (1 << 31) * torch.randint(0, 2, (n, F), generator=g)
    X = (bits - (bits >= 1 << 31) * (1 << 32)).int().view(torch.float32)
    assert torch.isfinite(X).all()

    def trunc(v):
        return (v.view(torch.int32) & -8192).view(torch.float32)
    hi = trunc(X)
    want = hi.double() + trunc(X - hi).double()
    got = ops.spmm(f.rowptr, f.col, f.val, f.window_of_part, f.atomic, X.cuda(), n, wide=4).cpu()
    assert torch.equal(want.float().double(), want) and torch.equal(got.double(), want)
