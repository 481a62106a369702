"""Row sums of split windows: the parts' sums meet in a fixed order, as in fp64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [8, 16])
@pytest.mark.parametrize("H", [1, 3, 4, 5])
@pytest.mark.parametrize("dt", [torch.float16, torch.float32])
@pytest.mark.parametrize("layout", ["h_m", "m_h"])
def test_split_windows_have_one_order(cuda, W, H, dt, layout):
    """Windows of 1 .. 100 parts: the sum of the parts' own sums (each computed
    as a window of its own), added in fp64 and rounded once, in every run."""
    from att_gb300 import gat_ops, ops
    rng = np.random.default_rng(H)
    n = 8 * 100  # columns; one 8-column block per part
    lengths = [8, 9, 17, 64, 264, 265, 800, 0, 800]
    rowptr, col = [0], []
    for length in lengths:
        cells = np.sort(rng.choice(n, length, replace=False))
        owner = rng.integers(0, W, length)
        for r in range(W):
            col.extend(cells[(owner == r) | (rng.random(length) < 0.5)] if length else [])
            rowptr.append(len(col))
    m = len(lengths) * W
    f = ops.block_convert(torch.tensor(rowptr, dtype=torch.int32), torch.tensor(np.array(col), dtype=torch.int32), None,
                          window=W, wide=8, part=1, want_val=False, want_map=True, n_cols=n)
    q = gat_ops.map_to_quad(f.map, W, 8)
    nnz = len(col)
    vals = torch.from_numpy(rng.uniform(0.1, 2.0, (H, nnz))).to(dt).cuda()
    args = (W, vals, nnz, 1, H)
    P = f.n_parts
    alone = gat_ops.rowsum(f.rowptr, q, torch.arange(P, dtype=torch.int32, device="cuda"),
                           torch.zeros(P, dtype=torch.int32, device="cuda"), *args, P * W).cpu()[..., 0]
    win = f.window_of_part.cpu().long()
    assert int(torch.bincount(win).max()) >= 90
    ref = torch.zeros(H, len(lengths), W, dtype=torch.float64).index_add_(1, win, alone.view(H, P, W).double())
    ref = ref.view(H, m).float()
    for _ in range(3):
        got = gat_ops.rowsum(f.rowptr, q, f.window_of_part, f.atomic, *args, m, layout).cpu()[..., 0]
        assert torch.equal(got if layout == "h_m" else got.t(), ref)


def test_scratch_is_checked(cuda):
    from att_gb300 import _lib
    one = torch.zeros(8, dtype=torch.int32, device="cuda")
    out = torch.zeros(8, device="cuda")
    assert _lib.lib().att_rowsum_scratch_bytes(3, 8, 2) == 4 * 3 * 8 * 2
    assert _lib.lib().att_rowsum_scratch_bytes(0, 8, 2) == 0
    p = one.data_ptr()
    for scratch, size in ((None, 1 << 20), (p, 31)):
        with pytest.raises(_lib.AttError) as e:
            _lib.call("att_rowsum_ordered", p, p, p, p, 1, 8, 4, out.data_ptr(), _lib.F32, 0, 1, 1, out.data_ptr(), 0, 1,
                      8, scratch, size, None)
        assert "scratch" in str(e.value)


@pytest.mark.parametrize("W", [8, 16])
def test_infinities_in_a_split_window(cuda, W):
    """inf, -inf, inf - inf and NaN among the parts' sums come out as they are."""
    from att_gb300 import gat_ops, ops
    n = 400
    rowptr = torch.arange(0, W * n + 1, n, dtype=torch.int32)
    f = ops.block_convert(rowptr, torch.arange(n, dtype=torch.int32).repeat(W), None, window=W, wide=8, part=1,
                          want_val=False, want_map=True, n_cols=n)
    vals = torch.ones(1, W * n, device="cuda")
    inf = float("inf")
    vals[0, [17, n + 399, 2 * n + 3, 2 * n + 300, 3 * n + 200]] = torch.tensor([inf, -inf, inf, -inf, float("nan")]).cuda()
    q = gat_ops.map_to_quad(f.map, W, 8)
    got = gat_ops.rowsum(f.rowptr, q, f.window_of_part, f.atomic, W, vals, W * n, 1, 1, W).cpu()[0, :, 0]
    assert torch.equal(torch.nan_to_num(got, nan=1e9), torch.nan_to_num(vals.view(W, n).sum(1).cpu(), nan=1e9))
