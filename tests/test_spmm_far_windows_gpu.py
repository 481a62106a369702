"""Parts whose window lies past the output are cut, up to the largest id that the kernels hold
(2^30 - 1): an id of 2^29 and more is not taken for a row before the output."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [1 << 20, (1 << 29) - 1, 1 << 29, (1 << 30) - 1])
@pytest.mark.parametrize("dt,wide,ordered", [("fp16", 8, False), ("fp16", 8, True), ("bf16", 16, True),
                                             ("tf32", 4, False), ("fp8", 8, False)])
@pytest.mark.parametrize("W", [8, 16])
def test_windows_past_the_output(cuda, dt, wide, ordered, W, far):
    from att_gb300 import ops
    rng = np.random.default_rng(W)
    lengths, n_cols, F = [40, 3, 100, 0, 9], 128, 64
    rowptr, col = [0], []
    for length in lengths:
        cells = np.sort(rng.choice(n_cols, length, replace=False))
        owner = rng.integers(0, W, length)
        for r in range(W):
            col.extend(cells[owner == r])
            rowptr.append(len(col))
    rowptr, col = np.array(rowptr, np.int32), np.array(col, np.int32)
    n = len(lengths) * W
    deg = torch.full((n_cols,), 0.5, dtype=torch.float32 if wide == 4 else torch.float16)
    f = ops.block_convert(torch.from_numpy(rowptr), torch.from_numpy(col), deg, window=W, wide=wide, part=1,
                          n_cols=n_cols)
    t = {"fp16": torch.float16, "bf16": torch.bfloat16, "tf32": torch.float32, "fp8": torch.float8_e4m3fn}[dt]
    x = torch.from_numpy(rng.integers(-4, 5, (n_cols, F)).astype(np.float32))
    rows = torch.from_numpy(np.repeat(np.arange(n), np.diff(rowptr)))
    want = torch.zeros(n, F).index_add_(0, rows, 0.25 * x[torch.from_numpy(col).long()])
    win = f.window_of_part.cpu()
    assert int((win == 2).sum()) > 3
    want[W:3 * W] = 0  # an unsplit and a split window go
    win[win == 1], win[win == 2] = far - 1, far
    val = f.val if dt in ("fp16", "fp8") else f.val.to(t)
    Y = torch.full((n, F), float("nan"), device="cuda")
    ops.spmm(f.rowptr, f.col, val, win.cuda(), f.atomic, x.to(t).cuda(), n, window=W, wide=wide, out=Y,
             x_scale=torch.ones(n_cols, device="cuda") if dt == "fp8" else None, ordered=ordered)
    assert torch.equal(Y.cpu(), want)
