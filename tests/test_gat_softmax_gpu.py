"""The online softmax of the fused GAT forward: its arithmetic does not depend
on where a row's columns fall in the stream, weights below the normal range
of fp32 count, and infinite scores give what leaky_relu and softmax do."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _graph(rows, n):
    """CSR of {row: columns}, every other row empty."""
    rowptr = torch.zeros(n + 1, dtype=torch.int32)
    for r, c in rows.items():
        rowptr[r + 1] = len(c)
    col = torch.cat([torch.tensor(sorted(rows[r]), dtype=torch.int32) for r in sorted(rows)])
    return torch.cumsum(rowptr, 0).to(torch.int32), col


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("F", [32, 64, 128])
@pytest.mark.parametrize("stats", [True, False])
def test_reference_move_does_not_depend_on_the_half(cuda, dt, F, stats):
    """Rows whose softmax reference moves between one group of 16 columns and
    the next: once both groups are halves of one 32-column chunk, once the
    second opens the next chunk (16 columns of another row stand before them).
    The same operations on the same numbers: the same bits."""
    from att_gb300 import gat
    pairs = 40
    n = 16 * pairs + 48
    first, second = range(n - 32, n - 16), range(n - 16, n)  # the groups; the 16 columns before are `pre`
    trigger = n - 1                                            # of row 0 alone: moves the whole window's references
    g = torch.Generator().manual_seed(F)
    rows = {}
    for k in range(pairs):
        for j in range(7):
            cols = [c for c in list(first) + list(second)[:-1] if torch.rand(1, generator=g).item() < 0.7]
            cols += [first[j], second[j]] + ([trigger] if j == 0 else [])
            rows[16 * k + j] = rows[16 * k + 8 + j] = set(cols)
        for j, c in enumerate(list(first) + list(second)[:-1]):  # every column is there in both windows
            for w in (0, 8):
                rows[16 * k + w + 1 + j % 6] = rows[16 * k + w + 1 + j % 6] | {c}
        rows[16 * k + 8 + 7] = set(range(n - 48, n - 32))
    G = gat.GATGraph(*_graph(rows, n))
    s0 = torch.zeros(1, n)
    s1 = torch.rand(1, n, generator=g) * 2 - 1
    s1[0, list(second)] += 1.0
    s1[0, trigger] = 12.0  # more than 8 above every other
    X = (torch.rand(n, F, generator=g) * 2 - 1).to(dt)
    out, rmax, rsum = G.attention(X.cuda(), mode=gat.MODE_ADD, s0=s0.cuda(), s1=s1.cuda(), stats=stats)
    a = torch.arange(pairs)[:, None] * 16 + torch.arange(7)
    for t in [out] + ([rmax[0], rsum[0]] if stats else []):
        assert torch.equal(t[a].cpu(), t[a + 8].cpu())
    if stats:
        assert torch.all(rsum[0][a] > 0)


@pytest.mark.parametrize("stats", [True, False])
def test_weights_below_the_normal_range(cuda, stats):
    """A weight e^-88 = 6.05e-39 is subnormal in fp32 and bf16 and still counts
    where the features are large: sum = 1, out = e^-88 2^126 = 0.515.
    Bound: bf16 rounds the weight to multiples of 2^-133; the argument of the
    exponential (88 log2 e, rounded) is 4e-6 off, the weight 2^-149 / 6e-39."""
    from att_gb300 import gat
    tol = 2.0 ** -134 / 6.05e-39 + 1e-4
    n = 64
    G = gat.GATGraph(*_graph({r: {8 + r, 32 + r} for r in range(8)}, n))
    X = torch.zeros(n, 32, dtype=torch.bfloat16)
    X[32:40] = 2.0 ** 126
    s1 = torch.zeros(1, n)
    s1[0, 32:40] = -88.0
    out, _, rsum = G.attention(X.cuda(), mode=gat.MODE_ADD, s0=torch.zeros(1, n).cuda(), s1=s1.cuda(), slope=1.0,
                               stats=stats)
    ref = 2.0 ** 126 * torch.exp(torch.tensor(-88.0, dtype=torch.float64)).item()
    assert ((out[:8].cpu().double() - ref).abs() <= tol * ref).all()
    if stats:
        assert torch.all(rsum[0, :8] == 1)


@pytest.mark.parametrize("slope", [0.0, 0.2, 1.0, 1.5, -0.5])
@pytest.mark.parametrize("value", [float("-inf"), float("inf"), float("nan")])
def test_infinite_and_nan_scores(cuda, slope, value):
    """A neighbour whose score is infinite or NaN, as leaky_relu and softmax have
    it: with slope 0 a score of -inf is 0 * -inf, a NaN."""
    from att_gb300 import gat
    n = 64
    G = gat.GATGraph(*_graph({r: {8 + r, 32 + r} for r in range(8)}, n))
    X = torch.ones(n, 32, dtype=torch.float16)
    s1 = torch.zeros(1, n)
    s1[0, 32:36] = value
    out, _, _ = G.attention(X.cuda(), mode=gat.MODE_ADD, s0=torch.zeros(1, n).cuda(), s1=s1.cuda(), slope=slope,
                            stats=False)
    e = torch.stack([s1[0, 8:16], s1[0, 32:40]], 1)
    ref = torch.softmax(torch.where(e > 0, e, slope * e), 1).sum(1)  # features of 1: the weights' sum
    got = out[:8].cpu()
    assert torch.equal(torch.isnan(got), torch.isnan(ref)[:, None].expand_as(got))
    ok = ~torch.isnan(ref)
    assert ((got[ok] - 1).abs() <= 1e-5).all()
