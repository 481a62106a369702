"""Outputs of up to 32 MiB do not depend on the order of the windows in the part
list: every row is zeroed first, whoever stores it.  Whole-number features and
values of 0.25: every result is exact."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _parts(W, wide, seed):
    """Block format (one block per part) of windows of 0 .. 300 columns."""
    from att_gb300 import ops
    rng = np.random.default_rng(seed)
    lengths, n_cols = [3, 0, 300, 40, 8, 0, 9, 129, 16, 300, 1], 400
    rowptr, col = [0], []
    for length in lengths:
        cells = np.sort(rng.choice(n_cols, length, replace=False))
        owner = rng.integers(0, W, length)
        for r in range(W):
            col.extend(cells[owner == r])
            rowptr.append(len(col))
    rowptr, col = np.array(rowptr, np.int32), np.array(col, np.int32)
    n = len(lengths) * W
    deg = torch.full((max(n, n_cols),), 0.5, dtype=torch.float32 if wide == 4 else torch.float16)
    f = ops.block_convert(torch.from_numpy(rowptr), torch.from_numpy(col), deg, window=W, wide=wide, part=1,
                          n_cols=n_cols)
    rows = torch.from_numpy(np.repeat(np.arange(n), np.diff(rowptr)))
    return f, rows, torch.from_numpy(col).long(), len(lengths), n_cols


@pytest.mark.parametrize("dt,wide,shape,gather", [("fp16", 8, None, 0), ("fp16", 16, None, 0), ("fp16", 8, None, 1),
                                                  ("fp16", 8, None, 2), ("bf16", 8, None, 0), ("tf32", 4, None, 0),
                                                  ("fp8", 8, ("fp8", 1), 0), ("fp8", 8, ("fp8", 0), 0)])
@pytest.mark.parametrize("W", [8, 16])
@pytest.mark.parametrize("F", [32, 64, 144])
def test_windows_in_any_order(cuda, dt, wide, shape, gather, W, F):
    from att_gb300 import _lib, ops
    f, rows, cols, n_win, n_cols = _parts(W, wide, F)
    g = torch.Generator().manual_seed(F)
    x = torch.randint(-4, 5, (n_cols, F), generator=g).float()
    t = {"fp16": torch.float16, "bf16": torch.bfloat16, "tf32": torch.float32, "fp8": torch.float8_e4m3fn}[dt]
    val = f.val.to(torch.float16 if dt == "fp8" else t)
    scale = torch.ones(n_cols, device="cuda") if dt == "fp8" else None
    ref = torch.zeros(n_win * W, F).index_add_(0, rows, 0.25 * x[cols]).view(n_win, W, F)
    m_out = (n_win + 2) * W + 3
    for order in (torch.arange(n_win), torch.arange(n_win).flip(0), torch.randperm(n_win, generator=g)):
        win = (order[f.window_of_part.cpu().long()] + 1).int().cuda()  # window 0 and the last ones have no part
        want = torch.zeros(m_out, F)
        want[W:W + n_win * W].view(n_win, W, F)[order] = ref
        Y = torch.full((m_out, F), float("nan"), device="cuda")
        _lib.call("att_set_thread_option", b"spmm_gather", gather)
        try:
            ops.spmm(f.rowptr, f.col, val, win, f.atomic, x.to(t).cuda(), m_out, window=W, wide=wide, out=Y,
                     x_scale=scale, shape=shape)
        finally:
            _lib.call("att_set_thread_option", b"spmm_gather", -1)
        assert torch.equal(Y.cpu(), want)
