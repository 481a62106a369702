"""The ordered SpMM on both sides of the widest tile that its merge's grid holds: 65,535 blocks of
64 float4s, 4 rows' worth of which are F (16-row windows) or half of it (8-row ones).  Whole-number
features and values of 0.25: every result is exact."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,F", [(16, 1048552), (16, 1048560), (16, 1048568), (16, 1 << 20), (16, (1 << 20) + 8),
                                 (8, 1 << 20), (8, 2097120), (8, 2097128)])
def test_widest_tiles(cuda, W, F):
    from att_gb300 import ops
    rng = np.random.default_rng(W)
    n_cols, lengths = 28, [28, 3]
    rowptr, col = [0], []
    for length in lengths:
        cells = np.sort(rng.choice(n_cols, length, replace=False))
        owner = rng.integers(0, W, length)
        for r in range(W):
            col.extend(cells[owner == r])
            rowptr.append(len(col))
    rowptr, col = np.array(rowptr, np.int32), np.array(col, np.int32)
    f = ops.block_convert(torch.from_numpy(rowptr), torch.from_numpy(col), torch.full((max(n_cols, len(lengths) * W),), 0.5).half(),
                          window=W, wide=8, part=1, n_cols=n_cols)
    assert f.n_parts == 5 and 4 * f.n_parts * W * F <= 1 << 30  # a window of four parts; scratch is taken
    x = torch.randint(-4, 5, (n_cols, F), generator=torch.Generator("cuda").manual_seed(1), device="cuda").half()
    n = len(lengths) * W
    A = torch.zeros(n, n_cols, device="cuda")
    A[torch.from_numpy(np.repeat(np.arange(n), np.diff(rowptr))), torch.from_numpy(col).long()] = 0.25
    got = ops.spmm(f.rowptr, f.col, f.val, f.window_of_part, f.atomic, x, n, window=W, ordered=True)
    for r in range(n):  # each row has few neighbours: a sum of rows, exact in fp32
        c = A[r].nonzero().flatten()
        assert torch.equal(got[r], 0.25 * x[c].float().sum(0))
