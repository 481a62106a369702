"""The chunk stream of the SpMM kernels (32 condensed columns at a time) at its
edges: windows of every length around the 8-column block, the 16-row half and
the 32-column chunk, parts of one and several chunks, feature widths around the
item width, empty parts, an unaligned column list and an output whose rows are
not 16-byte aligned.

Bound per output value, from the arithmetic: with S = sum |v x| over its terms,
fp32 accumulation of exact products errs by at most (terms + 8) 2^-24 S; the
3xTF32 split by at most another 3 * 2^-20 S; the e4m3 kernel rounds each scaled
value once to fp16, 2^-11 S more."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 7, 8, 9, 15, 16, 17, 23, 24, 25, 31, 32, 33, 47, 48, 49, 63, 64, 65, 255, 256, 257, 300]


def _graph(window, seed):
    """A window per length: that many distinct columns, spread over its rows."""
    rng = np.random.default_rng(seed)
    n_cols = 700
    rows, cols = [], []
    for w, length in enumerate(LENGTHS):
        for c in rng.choice(n_cols, size=length, replace=False):
            rows.append(w * window + int(rng.integers(0, window)))
            cols.append(c)
    order = np.lexsort((cols, rows))
    rows, cols = np.array(rows)[order], np.array(cols)[order]
    n = len(LENGTHS) * window
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    return rowptr, cols.astype(np.int32), n, n_cols


CASES = [(dt, F, W, w, part) for dt, Fs, ws in (("fp16", (8, 32, 40, 64, 72, 128, 136), (8, 16)),
                                               ("bf16", (56, 64), (8,)),
                                               ("tf32", (4, 32, 36, 64, 68, 100, 128), (4, 8)),
                                               ("fp8", (16, 64, 80, 128, 144), (8, 16)))
         for F in Fs for W in (8, 16) for w in ws for part in (1, 32)]


@pytest.mark.parametrize("dt,F,W,w,part", CASES)
def test_stream_edges(cuda, dt, F, W, w, part):
    from att_gb300 import ops
    rowptr, col, n, n_cols = _graph(W, F + W)
    rng = np.random.default_rng(F)
    deg = rng.uniform(0.1, 1.0, max(n, n_cols)).astype(np.float32 if dt == "tf32" else np.float16)
    f = ops.block_convert(torch.from_numpy(rowptr), torch.from_numpy(col), torch.from_numpy(deg), window=W, wide=w,
                          part=part, emit_empty=(dt == "tf32"), val_dtype=torch.bfloat16 if dt == "bf16" else None)
    x = torch.from_numpy(rng.uniform(-1, 1, (n_cols, F)).astype(np.float32))
    scale = None
    if dt == "fp8":
        scale = (x.abs().amax(1) / 448).float()
        X = (x / scale[:, None]).to(torch.float8_e4m3fn)
        xd = X.double() * scale.double()[:, None]
    else:
        X = x.to({"fp16": torch.float16, "bf16": torch.bfloat16, "tf32": torch.float32}[dt])
        xd = X.double()
    vt = {"bf16": torch.bfloat16, "tf32": torch.float32}.get(dt, torch.float16)
    rows = np.repeat(np.arange(n), np.diff(rowptr))
    v = (torch.from_numpy(deg[rows]).float() * torch.from_numpy(deg[col]).float()).to(vt).double()
    ref = torch.zeros(n, F, dtype=torch.float64).index_add_(0, torch.from_numpy(rows), v[:, None] * xd[col])
    mag = torch.zeros(n, F, dtype=torch.float64).index_add_(0, torch.from_numpy(rows), v[:, None] * xd[col].abs())
    eps = (300 + 8) * 2.0 ** -24 + {"tf32": 3 * 2.0 ** -20, "fp8": 2.0 ** -11}.get(dt, 0.0)
    m_out = n + 3  # rows past the last window come back zero
    out = torch.full((m_out, F + 1), float("nan"), device="cuda")[:, :F]  # rows not 16-byte aligned
    shifted = torch.cat([f.col[:1], f.col])[1:]                            # ids at an address of 4 mod 16
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    shapes = {"tf32": [("tf32", k) for k in range(3)], "fp8": [("fp8", 1)]}.get(
        dt, [("spmm", fc, st) for fc in (64, 128) for st in (3, 4)])
    for c, Y, shape in [(f.col, None, None), (shifted, out, None)] + [(f.col, None, s) for s in shapes]:
        got = ops.spmm(f.rowptr, c, f.val, f.window_of_part, f.atomic, X.cuda(), m_out, window=W, wide=w, out=Y,
                       x_scale=None if scale is None else scale.cuda(), err_flag=err, shape=shape).cpu().double()
        assert torch.all(got[n:] == 0)
        assert torch.all((got[:n] - ref).abs() <= eps * mag)
    assert int(err.item()) == 0


def test_infinite_features_stay_in_their_rows(cuda):
    """A row that no window gathers, and one past the padding, never reach an output."""
    from att_gb300 import ops
    rowptr, col, n, n_cols = _graph(8, 1)
    deg = np.full(max(n, n_cols), 0.5, np.float16)
    f = ops.block_convert(torch.from_numpy(rowptr), torch.from_numpy(col), torch.from_numpy(deg))
    unused = sorted(set(range(n_cols)) - set(col.tolist()))
    assert unused
    X = torch.ones(n_cols, 64, dtype=torch.float16)
    X[unused] = float("inf")
    Y = ops.spmm(f.rowptr, f.col, f.val, f.window_of_part, f.atomic, X.cuda(), n)
    assert torch.isfinite(Y).all()


def test_capture_replays(cuda):
    """The zero pass and the kernel behind it, captured and replayed on new features."""
    from att_gb300 import ops
    rowptr, col, n, n_cols = _graph(8, 2)
    deg = np.full(max(n, n_cols), 0.5, np.float16)
    f = ops.block_convert(torch.from_numpy(rowptr), torch.from_numpy(col), torch.from_numpy(deg), part=1)
    X = torch.rand(n_cols, 64, device="cuda").half()
    Y = torch.empty(n, 64, device="cuda")

    def call():
        ops.spmm(f.rowptr, f.col, f.val, f.window_of_part, f.atomic, X, n, out=Y)
    call()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    X.copy_(torch.rand(n_cols, 64, device="cuda").half())
    for _ in range(3):
        g.replay()
    again = Y.clone()
    call()
    # parts of split windows add in any order
    assert torch.allclose(again, Y, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("W", [8, 16])
@pytest.mark.parametrize("F", [72, 96, 128, 136, 192, 256])
@pytest.mark.parametrize("n_windows", [4095, 4096])
def test_item_width_rule(cuda, W, F, n_windows):
    """Either side of the part count from which wide features take 128-feature
    items: the same bits as both widths asked for by name (unsplit windows, so
    every output is one chain of additions), and the FP64 result."""
    from att_gb300 import ops
    n = n_windows * W
    rng = np.random.default_rng(F)
    rowptr = np.arange(0, 2 * n + 1, 2, dtype=np.int32)
    col = np.sort(np.stack([rng.integers(0, n // 2, n), rng.integers(n // 2, n, n)], 1), 1).reshape(-1).astype(np.int32)
    deg = np.full(n, 0.5, np.float16)
    f = ops.block_convert(torch.from_numpy(rowptr), torch.from_numpy(col), torch.from_numpy(deg), window=W)
    assert f.n_parts == n_windows
    X = torch.from_numpy(rng.uniform(-1, 1, (n, F)).astype(np.float16))
    got = [ops.spmm(f.rowptr, f.col, f.val, f.window_of_part, f.atomic, X.cuda(), n, window=W, shape=s).cpu()
           for s in (None, ("spmm", 64, 3), ("spmm", 128, 3))]
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    ref = 0.25 * (X[col[0::2]].double() + X[col[1::2]].double())
    assert torch.all((got[0].double() - ref).abs() <= 2 * 2.0 ** -24)
