"""Feature matrices that the SpMM drop-in reshapes, takes as they are, or refuses.
No GPU: the launch is replaced."""
import pytest
import torch


def _call(monkeypatch, shape, dimN):
    from att_gb300 import ops
    from att_gb300.compat import SpMM_sr_bcrs as m
    seen = []
    monkeypatch.setattr(m, "_check", lambda t, name: None)
    monkeypatch.setattr(ops, "spmm", lambda *a, **k: seen.append(a[5]) or torch.zeros(4, a[5].shape[1]))
    i = torch.zeros(3, dtype=torch.int32)
    x = torch.arange(torch.Size(shape).numel()).half().view(shape)
    y = m.forward_fp16_gnn(i, i, x, i, i, x, 8, dimN, 4)[0]
    return seen[0], y


@pytest.mark.parametrize("shape,dimN,rows,width", [((4, 8), 8, 4, 8), ((32,), 8, 4, 8), ((2, 2, 8), 8, 4, 8),
                                                   ((4, 16), 8, 8, 8), ((4, 5), 5, 4, 8), ((20,), 5, 4, 8)])
def test_reshaped_or_taken(monkeypatch, shape, dimN, rows, width):
    X, Y = _call(monkeypatch, shape, dimN)
    assert X.shape == (rows, width) and Y.shape == (4, dimN)
    assert torch.equal(X[:, :dimN].flatten(), torch.arange(rows * dimN).half())


@pytest.mark.parametrize("shape,dimN", [((4, 0), 0), ((0,), 0), ((4, 8), 0), ((4, 8), 5)])
def test_refused(monkeypatch, shape, dimN):
    with pytest.raises(RuntimeError):
        _call(monkeypatch, shape, dimN)
