"""Parts that do not start and end on a block boundary (a malformed format): the
fused GAT forward flags them and leaves out those parts alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide", [8, 16])
@pytest.mark.parametrize("per_run", [1, 4, 40])
@pytest.mark.parametrize("bad", [[0], [1, 2], [3], [5, 9], [38], [0, 38], list(range(39))])
@pytest.mark.parametrize("dt", [torch.float16, torch.float32])
def test_only_the_misaligned_parts_are_left_out(cuda, wide, per_run, bad, dt):
    from att_gb300 import _lib, gat, ops
    parts, n, F = 40, 40 * wide + 16, 32
    g = torch.Generator().manual_seed(wide)
    adj = torch.rand(n, n, generator=g) < 0.4
    adj[0, :parts * wide] = True          # window 0 has every one of its columns
    adj[:8, parts * wide:] = False        # and whole blocks of them
    adj[8:, ] &= torch.rand(n - 8, 1, generator=g) < 0.1
    rows, cols = adj.nonzero(as_tuple=True)
    rowptr = torch.zeros(n + 1, dtype=torch.int64)
    rowptr[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    G = gat.GATGraph(rowptr.int(), cols.int(), wide=wide, part=1, parts_per_chunk=per_run)
    f = G.fmt
    assert int((f.window_of_part == 0).sum()) == parts
    rp = f.rowptr.cpu()
    dropped = torch.zeros(n, dtype=torch.bool)
    for k in bad:                          # the boundary behind part k moves into it: k and k + 1 are misaligned
        rp[2 * k + 1] -= wide // 2
        rp[2 * k + 2] -= wide // 2
        dropped[wide * k:wide * (k + 2)] = True
    f.rowptr = rp.cuda()
    keep = ~((rows < 8) & dropped[cols])
    X = (torch.rand(n, F, generator=g) * 2 - 1).to(dt)
    s0, s1 = torch.rand(2, 1, n, generator=g) * 2 - 1
    out = torch.empty(n, F, device="cuda")
    part = torch.empty(max(G.n_slots, 1) * 8 * (F + 2), device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = ops._p
    Xd, s0d, s1d = X.cuda(), s0.cuda(), s1.cuda()
    _lib.call("att_gat_forward", p(f.rowptr), p(f.col), p(G.mask), p(f.window_of_part), f.n_parts, p(G.chunk_begin),
              p(G.chunk_slot), G.n_chunks, p(G.multi), G.n_multi, 8, wide, p(Xd), ops._DT[dt], n, 1, F, F, 1, p(s0d),
              p(s1d), 0.2, p(out), F, None, None, p(part), p(err), ops._stream())
    assert int(err.item()) == 2
    r, c = rows[keep], cols[keep]
    e = s0[0, r].double() + s1[0, c].double()
    w = torch.exp(torch.where(e > 0, e, 0.2 * e))
    total = torch.zeros(n, dtype=torch.float64).index_add_(0, r, w)
    ref = torch.zeros(n, F, dtype=torch.float64).index_add_(0, r, w[:, None] * X[c].double())
    ref /= total.clamp_min(1e-300)[:, None]
    # weights rounded once to fp16 (2^-11 each way), or 3xTF32 products
    assert (out.cpu().double() - ref).abs().max() <= (2e-5 if dt == torch.float32 else 2.0 ** -10 + 1e-4)
