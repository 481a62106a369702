"""The ordered SpMM of 16-bit features: the parts of split windows meet in part order, as in fp64, so
every run gives the same bits; unsplit windows are as ever."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [8, 0, 17, 64, 264, 265, 800, 3, 0, 800, 40]


def _format(W, wide, seed, n=800):
    """One block per part: windows of up to 100 parts, empty ones between."""
    from att_gb300 import ops
    rng = np.random.default_rng(seed)
    rowptr, col = [0], []
    for length in LENGTHS:
        cells = np.sort(rng.choice(n, length, replace=False))
        owner = rng.integers(0, W, length)
        for r in range(W):
            col.extend(cells[(owner == r) | (rng.random(length) < 0.3)] if length else [])
            rowptr.append(len(col))
    deg = torch.from_numpy(rng.uniform(0.1, 1.0, n)).half()
    f = ops.block_convert(torch.tensor(rowptr, dtype=torch.int32), torch.tensor(np.array(col), dtype=torch.int32), deg,
                          window=W, wide=wide, part=1, n_cols=n)
    return f, n


@pytest.mark.parametrize("dt,wide", [("fp16", 8), ("fp16", 16), ("bf16", 8), ("bf16", 16)])
@pytest.mark.parametrize("W", [8, 16])
@pytest.mark.parametrize("F", [16, 64, 144])
def test_one_order(cuda, dt, wide, W, F):
    """Equal to the parts' own tiles (each part as a window of its own), added in
    fp64 and rounded once; aligned and unaligned output rows; rows past m_out cut."""
    from att_gb300 import ops
    f, n = _format(W, wide, F)
    t = {"fp16": torch.float16, "bf16": torch.bfloat16}[dt]
    X = torch.from_numpy(np.random.default_rng(F).uniform(-1, 1, (n, F)).astype(np.float32)).to(t).cuda()
    val = f.val.to(t)
    kw = dict(window=W, wide=wide)
    P, m = f.n_parts, len(LENGTHS) * W - 3
    alone = ops.spmm(f.rowptr, f.col, val, torch.arange(P, dtype=torch.int32, device="cuda"),
                     torch.zeros(P, dtype=torch.int32, device="cuda"), X, P * W, **kw).cpu().view(P, W, F)
    win = f.window_of_part.cpu().long()
    assert int(torch.bincount(win).max()) >= 50
    ref = torch.zeros(len(LENGTHS), W, F, dtype=torch.float64).index_add_(0, win, alone.double())
    ref = ref.view(-1, F)[:m].float()
    out = torch.full((m, F + 1), float("nan"), device="cuda")[:, :F]
    for Y in (None, None, out):
        got = ops.spmm(f.rowptr, f.col, val, f.window_of_part, f.atomic, X, m, out=Y, ordered=True, **kw).cpu()
        assert torch.equal(got, ref)
    near = ops.spmm(f.rowptr, f.col, val, f.window_of_part, f.atomic, X, m, **kw).cpu()
    whole = (f.atomic.cpu() == 0).nonzero().flatten()
    rows = (win[whole][:, None] * W + torch.arange(W)).flatten()
    assert torch.equal(near[rows[rows < m]], ref[rows[rows < m]])  # unsplit windows: one chain either way


def test_infinities_and_other_orders(cuda):
    from att_gb300 import ops
    f, n = _format(8, 8, 3)
    X = torch.ones(n, 64, dtype=torch.float16)
    inf = float("inf")
    X[::7, 0], X[3::11, 1], X[5::13, 1], X[100, 2] = inf, inf, -inf, float("nan")
    m = len(LENGTHS) * 8
    args = (f.rowptr, f.col, f.val)
    a = ops.spmm(*args, f.window_of_part, f.atomic, X.cuda(), m, ordered=True).cpu()
    b = ops.spmm(*args, f.window_of_part, f.atomic, X.cuda(), m).cpu()
    for t in (a, b):
        assert torch.equal(torch.isnan(t), torch.isnan(b)) and torch.equal(t[:, :3] == inf, b[:, :3] == inf)
    order = torch.randperm(len(LENGTHS), generator=torch.Generator().manual_seed(1))
    win = order[f.window_of_part.cpu().long()].int().cuda()  # windows out of order: a small output takes them
    c = ops.spmm(*args, win, f.atomic, X.cuda(), m, ordered=True).cpu().view(-1, 8, 64)
    assert torch.equal(torch.nan_to_num(c[order], nan=7.0), torch.nan_to_num(a.view(-1, 8, 64), nan=7.0))


def test_capture_and_scratch(cuda):
    from att_gb300 import _lib, ops
    f, n = _format(8, 8, 5)
    X = torch.rand(n, 64, device="cuda").half()
    m = len(LENGTHS) * 8
    Y = torch.empty(m, 64, device="cuda")

    def call():
        ops.spmm(f.rowptr, f.col, f.val, f.window_of_part, f.atomic, X, m, out=Y, ordered=True)
    call()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    X.copy_(torch.rand(n, 64, device="cuda").half())
    g.replay()
    again = Y.clone()
    call()
    assert torch.equal(again, Y)
    need = _lib.lib().att_spmm_scratch_bytes(f.n_parts, 8, 64)
    assert need == f.n_parts * 8 * 64 * 4 and _lib.lib().att_spmm_scratch_bytes(0, 8, 64) == 0
    p = ops._p
    for scratch, size in ((None, need), (p(Y), need - 1), (p(Y) + 4, need)):
        with pytest.raises(_lib.AttError) as e:
            _lib.call("att_spmm_ordered", p(f.rowptr), p(f.col), p(f.val), _lib.F16, p(f.window_of_part), p(f.atomic),
                      f.n_parts, p(X), _lib.F16, None, n, 64, 64, p(Y), m, 64, 8, 8, None, scratch, size, None)
        assert "scratch" in str(e.value)


def test_gcn_layer_repeats_itself(cuda):
    """Output and gradients of a GCN layer with hubs: the same bits in every run."""
    from att_gb300 import layers
    g = torch.Generator().manual_seed(2)
    n = 6000
    src = torch.cat([torch.randint(0, n, (30000,), generator=g), torch.arange(4).repeat_interleave(5000)])
    dst = torch.cat([torch.randint(0, n, (30000,), generator=g), torch.randint(0, n, (20000,), generator=g)])
    src, dst = torch.cat([src, dst, torch.arange(n)]), torch.cat([dst, src, torch.arange(n)])
    info = layers.GCNInput(src, dst, n)
    layer = layers.GCNConv(48, 64).cuda()
    X = (torch.rand(n, 48, generator=g) * 2 - 1).cuda().requires_grad_()
    d = torch.rand(n, 64, generator=g).cuda()
    runs = []
    for _ in range(6):
        out = layer(X, info)
        runs.append([out.detach()] + list(torch.autograd.grad(out, [X, layer.weights], d.to(out.dtype))))
    for r in runs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(r, runs[0]))
