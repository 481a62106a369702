"""The chunk stream of the fused GAT forward at its edges: windows of every
length around the half (16 columns), the chunk (32), the part and the run of
parts (a window over several runs is merged from partials), every block width,
head and feature count, with and without softmax statistics.

Bounds per output value, relative to the largest feature (an output is a convex
combination of features): 2^-10 (fp16) or 2^-7 (bf16) for probabilities rounded
once to 16 bits, 1e-4 for the hi + lo pair that statistics ask for (and for the
logits' fp32 sums), 2e-5 for 3xTF32."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 48, 63, 65, 255, 256, 257, 700]


def _graph(seed):
    rng = np.random.default_rng(seed)
    n = 8 * 90 + 3  # not a multiple of the window
    rows, cols = [], []
    for w, length in enumerate(LENGTHS):
        for c in rng.choice(n, size=length, replace=False):
            rows.append(8 * w + int(rng.integers(0, 8)))
            cols.append(c)
    for r in range(8 * len(LENGTHS), n):  # the last, ragged window too
        rows.append(r)
        cols.append(r)
    order = np.lexsort((cols, rows))
    rows, cols = np.array(rows)[order], np.array(cols)[order]
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return torch.from_numpy(rowptr).int(), torch.from_numpy(cols).int(), torch.from_numpy(rows), n


def _reference(e, rows, cols, n, x, slope):
    e = torch.where(e > 0, e, slope * e)
    m = torch.full((n,), -np.inf, dtype=torch.float64).scatter_reduce_(0, rows, e, "amax")
    p = torch.exp(e - m[rows])
    s = torch.zeros(n, dtype=torch.float64).index_add_(0, rows, p)
    out = torch.zeros(n, x.shape[1], dtype=torch.float64).index_add_(0, rows, p[:, None] * x[cols])
    return out / s.clamp_min(1e-300)[:, None], m + torch.log(s)


@pytest.mark.parametrize("dt,F", [(torch.float16, 32), (torch.float16, 64), (torch.float16, 128), (torch.bfloat16, 64),
                                  (torch.float32, 32), (torch.float32, 64), (torch.float32, 128)])
@pytest.mark.parametrize("wide,part,run", [(8, 32, 4), (8, 1, 4), (4, 3, 2), (16, 2, 1)])
@pytest.mark.parametrize("H,mode,slope", [(1, 0, 0.2), (3, 1, 0.2), (2, 0, 1.5)])
def test_runs(cuda, dt, F, wide, part, run, H, mode, slope):
    from att_gb300 import gat
    rowptr, col, rows, n = _graph(F)
    G = gat.GATGraph(rowptr, col, wide=wide, part=part, parts_per_chunk=run)
    g = torch.Generator().manual_seed(H)
    X = (torch.rand(n, H * F, generator=g) * 2 - 1).to(dt)
    s0, s1 = torch.rand(2, H, n, generator=g) * 6 - 3
    cols = col.long()
    for stats in (False, True):
        out, rmax, rsum = G.attention(X.cuda(), n_heads=H, mode=mode, s0=s0.cuda(), s1=s1.cuda(), slope=slope,
                                      stats=stats)
        tol = 2e-5 if dt == torch.float32 else 1e-4 + (0 if stats else 2.0 ** (-10 if dt == torch.float16 else -7))
        for h in range(H):
            x = X[:, h * F:(h + 1) * F].double()
            e = (x[rows] * x[cols]).sum(1) if mode == 0 else s0[h, rows].double() + s1[h, cols].double()
            ref, lse = _reference(e, rows, cols, n, x, slope)
            got = out[:, h * F:(h + 1) * F].cpu().double()
            assert (got - ref).abs().max() <= tol * x.abs().max()
            if stats:
                has = torch.bincount(rows, minlength=n) > 0
                got = (rmax[h].cpu().double() + torch.log(rsum[h].cpu().double()))[has]
                assert (got - lse[has]).abs().max() <= 1e-4 * (1 + lse[has].abs().max())
                assert torch.all(rsum[h].cpu()[~has] == 0)


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("F,H", [(32, 3), (64, 1), (64, 4), (128, 2)])
def test_grad_prepare_forms(cuda, dt, F, H):
    """The 16-byte form of the backward's first pass keeps the scalar form's
    order of sums: the same bits (rows off the 16-byte grid take the latter)."""
    from att_gb300 import _lib, ops
    n = 1003
    g = torch.Generator().manual_seed(F)
    dout, out = (torch.rand(2, n, H * F, generator=g) * 2 - 1).cuda()
    off = torch.empty(n * H * F + 1, device="cuda")[1:].view(n, H * F).copy_(dout)
    got = []
    for d in (dout, off):
        hi, lo = torch.empty(2, n, H * F, dtype=dt, device="cuda")
        c = torch.empty(H, n, device="cuda")
        _lib.call("att_gat_grad_prepare", ops._p(d), H * F, ops._p(out), H * F, n, H, F, ops._p(hi), ops._p(lo),
                  ops._DT[dt], H * F, ops._p(c), ops._stream())
        got.append((hi, lo, c))
    for a, b in zip(*got):
        assert torch.equal(a, b)
    ref = (dout.double() * out.double()).view(n, H, F).sum(2).t()
    assert (got[0][2].double() - ref).abs().max() <= F * 2.0 ** -23
    assert torch.equal(got[0][0], dout.to(dt))
