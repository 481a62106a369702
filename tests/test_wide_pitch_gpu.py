"""Feature matrices whose row pitch or extent passes 2^31: the 64-bit forms of
the kernels give the same bits as the 32-bit ones on the same rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _strided(x, ld):
    """The rows of x at a pitch of ld elements."""
    n, F = x.shape
    big = torch.zeros((n - 1) * ld + F, dtype=torch.uint8 if x.element_size() == 1 else x.dtype, device="cuda")
    v = big.view(x.dtype).as_strided((n, F), (ld, 1))
    for r in range(n):
        v[r].copy_(x[r])
    return v


@pytest.mark.parametrize("dt,ld,wide", [(torch.float16, 1 << 30, 8), (torch.float32, 1 << 29, 4),
                                        (torch.float8_e4m3fn, 1 << 31, 8)])
@pytest.mark.parametrize("F", [32, 144])
def test_spmm(cuda, dt, ld, wide, F):
    from att_gb300 import ops
    n, n_x = 64, 3
    rowptr = torch.cumsum(torch.tensor([0] + [1 + r % 3 for r in range(n)]), 0).int()
    col = torch.cat([torch.arange(1 + r % 3) for r in range(n)]).int()
    deg = torch.full((n,), 0.5, dtype=torch.float32 if wide == 4 else torch.float16)
    f = ops.block_convert(rowptr, col, deg, wide=wide, n_cols=n_x)
    x = torch.randint(-8, 9, (n_x, F), generator=torch.Generator().manual_seed(F)).float().to(dt).cuda()
    scale = torch.ones(n_x, device="cuda") if dt == torch.float8_e4m3fn else None
    args = (f.rowptr, f.col, f.val, f.window_of_part, f.atomic)
    near = ops.spmm(*args, x, n, wide=wide, x_scale=scale)
    far = ops.spmm(*args, _strided(x, ld), n, wide=wide, x_scale=scale)
    rows = torch.repeat_interleave(torch.arange(n), rowptr[1:] - rowptr[:-1])
    ref = torch.zeros(n, F).index_add_(0, rows, 0.25 * x.float().cpu()[col.long()])
    assert torch.equal(near.cpu(), ref) and torch.equal(far.cpu(), ref)
    del far
    torch.cuda.empty_cache()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("stats", [False, True])
def test_fused_gat_forward(cuda, mode, stats):
    from att_gb300 import gat
    n, F = 16, 32
    G = gat.GATGraph(torch.arange(0, n * n + 1, n, dtype=torch.int32), torch.arange(n, dtype=torch.int32).repeat(n))
    x = (torch.rand(n, F, generator=torch.Generator().manual_seed(1)) * 2 - 1).half().cuda()
    s0, s1 = torch.rand(2, 1, n, device="cuda")
    got = [G.attention(v, mode=mode, s0=s0, s1=s1, stats=stats) for v in (x, _strided(x, 1 << 27))]
    for a, b in zip(*got):
        assert (a is None) == (b is None) and (a is None or torch.equal(a, b))
    torch.cuda.empty_cache()
