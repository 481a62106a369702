"""The quad-layout forms of the map operators (row sums, slot scores and row
broadcasts, dense values) and the map conversion, at window lengths around the
4-column quad and the four quads in flight, for one head, a whole group of four
and more, against per-edge references on the CPU; vectorised node scores.

Whole-number inputs of a few bits: every result is exact."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 3, 4, 5, 15, 16, 17, 31, 33, 64, 130]


def _format(W, wide, part, seed):
    from att_gb300 import gat_ops, ops
    rng = np.random.default_rng(seed)
    n = len(LENGTHS) * W
    rows, cols = [], []
    for w, length in enumerate(LENGTHS):
        for c in rng.choice(n, size=min(length, n), replace=False):
            rows.append(w * W + int(rng.integers(0, W)))
            cols.append(c)
    order = np.lexsort((cols, rows))
    rows, cols = np.array(rows)[order], np.array(cols)[order]
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    f = ops.block_convert(torch.from_numpy(rowptr), torch.from_numpy(cols.astype(np.int32)), None, window=W, wide=wide,
                          part=part, want_val=False, want_map=True)
    return f, gat_ops.map_to_quad(f.map, W, wide), torch.from_numpy(rows), torch.from_numpy(cols), n


def _quad_reference(m, W, wide):
    """The same slots, one by one."""
    m = m.cpu().numpy()
    out = np.empty_like(m)
    for g in range(m.size // W):
        for r in range(W):
            out[(g - g % 4) * W + r * 4 + g % 4] = m[(g - g % wide) * W + r * wide + g % wide]
    return torch.from_numpy(out)


@pytest.mark.parametrize("W,wide", [(8, 4), (8, 8), (8, 16), (16, 8)])
@pytest.mark.parametrize("part", [1, 32])
def test_map_to_quad(cuda, W, wide, part):
    f, q, _, _, _ = _format(W, wide, part, 3)
    assert torch.equal(q.cpu(), _quad_reference(f.map, W, wide))


@pytest.mark.parametrize("W", [8, 16])
@pytest.mark.parametrize("H", [1, 3, 4, 5])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("layout", ["h_e", "e_h"])
@pytest.mark.parametrize("part", [1, 32])
def test_map_operators(cuda, W, H, dt, layout, part):
    from att_gb300 import gat_ops
    f, q, rows, cols, n = _format(W, 8, part, H)
    nnz = rows.numel()
    g = torch.Generator().manual_seed(H)
    s0, s1 = torch.randint(-8, 8, (2, H, n), generator=g).float()
    args = (f.rowptr, f.col, q, f.window_of_part, W)
    got = gat_ops.slot_scores(*args, s0.cuda(), s1.cuda(), n, nnz, dt, layout).cpu().float()
    ref = s0[:, rows] + s1[:, cols]
    assert torch.equal(got if layout == "h_e" else got.t(), ref)
    node = torch.randint(-8, 8, (n, H), generator=g).to(dt).cuda()
    got = gat_ops.slot_rows(*args, node, node.stride(1), node.stride(0), H, n, nnz, dt, layout).cpu().float()
    assert torch.equal(got if layout == "h_e" else got.t(), node.cpu().float().t()[:, rows])
    vals = torch.randint(-3, 4, (H, nnz) if layout == "h_e" else (nnz, H), generator=g).to(dt).cuda()
    v, sh, se = gat_ops.edge_view(vals, H, nnz)
    got = gat_ops.rowsum(f.rowptr, q, f.window_of_part, f.atomic, W, v, sh, se, H, n).cpu()[..., 0]
    vh = (vals if layout == "h_e" else vals.t()).cpu().float()
    ref = torch.zeros(H, n).index_add_(1, rows, vh)
    assert torch.equal(got, ref)
    for out_wide, odt in ((8, torch.float16), (8, torch.bfloat16), (4, torch.float32), (8, torch.float32)):
        V = gat_ops.gather_slot_values(q, W, out_wide, v, sh, se, H, odt).cpu().float()
        std = f.map.cpu() if out_wide == 8 else q.cpu()
        ref = torch.where(std >= 0, vh[:, std.clamp_min(0).long()], torch.zeros(()))
        assert torch.equal(V, ref)


@pytest.mark.parametrize("F", [8, 16, 24, 64, 256])
@pytest.mark.parametrize("xt,at", [(torch.float16, torch.float16), (torch.bfloat16, torch.float32),
                                   (torch.float32, torch.float32)])
def test_node_scores(cuda, F, xt, at):
    from att_gb300 import gat_ops
    g = torch.Generator().manual_seed(F)
    X = torch.randint(-4, 4, (37, 3 * F), generator=g).to(xt).cuda().view(37, 3, F).permute(1, 0, 2)
    a = torch.randint(-4, 4, (2, 3, F), generator=g).to(at).cuda()
    ref = torch.einsum("hmf,khf->khm", X.cpu().double(), a.cpu().double()).float()
    assert torch.equal(gat_ops.node_scores(X, a[0]).cpu(), ref[0])
    s0, s1 = gat_ops.node_scores_pair(X, a[0], a[1])
    assert torch.equal(s0.cpu(), ref[0]) and torch.equal(s1.cpu(), ref[1])
