"""Jobs of the batched SpMM whose sizes do not fit 32-bit offsets: flagged and
left out, wherever they stand in the table; the others are computed."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field,value", [("F", (1 << 31) + 64), ("F", 1 << 31), ("ldx", 1 << 33), ("ldy", 1 << 31),
                                         ("m_out", 1 << 40)])
@pytest.mark.parametrize("where", [0, 1, 2])
def test_oversized_job(cuda, field, value, where):
    from att_gb300 import ops, serving
    n, F = 16, 64
    jobs = []
    for k in range(3):
        f = ops.block_convert(torch.arange(0, n + 1, dtype=torch.int32), torch.arange(n, dtype=torch.int32),
                              torch.full((n,), 0.5, dtype=torch.float16))
        g = serving.spmm_groups(f, m_out=n)
        assert (g.n_groups, g.n_red, g.n_empty) == (2, 0, 0)
        X = torch.randint(-8, 9, (n, F), generator=torch.Generator().manual_seed(k)).half().cuda()
        jobs.append(serving.Job(f, g, None, X, torch.full((n, F), float("nan"), device="cuda"), n))
    table, header = serving.build_job_table(jobs)
    setattr(table[where], field, value)
    items = 0
    for t in table:
        t.item_begin = items
        items += 2 * ((t.F + 63) // 64)
    b = serving.BatchedSpmm(3, use_graph=False)
    raw = bytearray(ctypes.string_at(ctypes.addressof(table), 3 * b.rec))
    b.table_d.copy_(torch.frombuffer(raw, dtype=torch.uint8))
    b.header_d.copy_(torch.tensor((3, items) + tuple(header[2:]), dtype=torch.int64))
    b._launch()
    assert int(b.err.item()) == 8
    for k, j in enumerate(jobs):
        if k == where:
            assert torch.isnan(j.Y).all()
        else:
            assert torch.equal(j.Y, 0.25 * j.X.float())
