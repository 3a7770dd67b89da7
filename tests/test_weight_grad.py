"""Weight-grad kernel at the edges of its tiles: weight rows that end inside a CTA pair's 256, columns that end
inside a tile (and where rows allow 16-byte stores only), reductions shorter than, as long as and longer than the
row slots, one and two tiles a unit, groups without rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(groups, M, N, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    ends = torch.tensor(groups, device="cuda").cumsum(0).to(torch.int32)
    rows = sum(groups)
    a = torch.randn(rows, M, device="cuda", generator=g).bfloat16()
    b = torch.randn(rows, N, device="cuda", generator=g).bfloat16()
    return g, ends, a, b


@pytest.mark.parametrize("two", [0, 1])
@pytest.mark.parametrize("M, N", [(128, 8), (384, 40), (256, 264), (640, 512), (256, 1032)])
@pytest.mark.parametrize("groups", [[64, 0, 128], [320, 384, 0, 448, 512], [1152, 64, 832]])
def test_edges(groups, M, N, two, monkeypatch):
    from moonep_b200.ops import elementwise as ew
    from moonep_b200.ops import gemm
    monkeypatch.setattr(gemm, "TWO_CTA", two)
    gen, ends, a, b = _inputs(groups, M, N, M + N)
    G, lr = len(groups), 0.25
    grad = torch.full((G, M, N), float("nan"), device="cuda")
    gemm.wgrad(a, b, ends, grad)
    start = 0
    for g, n in enumerate(groups):
        want = a[start:start + n].double().t() @ b[start:start + n].double()
        # products are exact in fp32; n additions, each off by at most one unit of the running sum (truncated), which
        # stays below sum |a b|
        bound = 2.0 ** -23 * max(n, 1) * (a[start:start + n].double().abs().t() @ b[start:start + n].double().abs())
        assert bool(((grad[g].double() - want).abs() <= bound).all()), g
        start += n
    # accumulating adds the same sums
    base = torch.randn(G, M, N, device="cuda", generator=gen)
    acc = base.clone()
    gemm.wgrad(a, b, ends, acc, accumulate=True)
    assert torch.equal(acc, base + grad)
    # the SGD step in the epilogue: bit for bit the update by the stored grads
    w = torch.randn(G, M, N, device="cuda", generator=gen).bfloat16()
    want = w.clone()
    ew.sgd_update_(want, grad, lr)
    keep = torch.zeros(G, dtype=torch.int32, device="cuda")
    keep[G - 1] = 1
    want[G - 1] = w[G - 1]
    kept = torch.zeros(G, M, N, device="cuda")
    gemm.wgrad(a, b, ends, kept, sgd=(w, lr, keep))
    assert torch.equal(w, want)
    assert torch.equal(kept[G - 1], grad[G - 1]) and not bool(kept[:G - 1].any())
    gemm.check_status()


@pytest.mark.parametrize("two", [0, 1])
@pytest.mark.parametrize("M, N", [(128, 8), (384, 264), (640, 512)])
def test_two_products_equal_one_each(M, N, two, monkeypatch):
    """Bit for bit the two launches: stored, accumulated and applied grads, groups with slots and without rows."""
    from moonep_b200.ops import gemm
    monkeypatch.setattr(gemm, "TWO_CTA", two)
    groups, split = [320, 0, 512, 64, 0, 128], 4
    gen, ends, a, b0 = _inputs(groups, M, N, 3 * M + N)
    b = (b0, torch.randn(a.shape[0], N, device="cuda", generator=gen).bfloat16())
    rnd = lambda n: [torch.randn(n, M, N, device="cuda", generator=gen) for _ in range(2)]
    copy = lambda ts: [t.clone() for t in ts]
    local, slots = rnd(split), rnd(len(groups) - split)
    w = [t.bfloat16() for t in rnd(split)]
    keep = torch.tensor([0, 0, 1, 0], dtype=torch.int32, device="cuda")
    for form in (dict(), dict(accumulate=True), dict(sgd=0.25)):
        got, want = [], []
        l, s, ws = copy(local), copy(slots), copy(w)
        kw = dict(form, sgd=(ws, 0.25, keep)) if "sgd" in form else form
        gemm.wgrad2(a, b, ends, l, grad_slot=s, split=split, **kw)
        got += l + s + ws
        l, s, ws = copy(local), copy(slots), copy(w)
        for i in range(2):
            kw = dict(form, sgd=(ws[i], 0.25, keep)) if "sgd" in form else form
            gemm.wgrad(a, b[i], ends, l[i], grad_slot=s[i], split=split, **kw)
        want += l + s + ws
        assert all(torch.equal(x, y) for x, y in zip(got, want)), form
    gemm.check_status()


# average k-blocks that the launch is told -> with SGD two pieces and one, one and two tiles a unit (from eight blocks,
# from two, not at all)
@pytest.mark.parametrize("two", [0, 1])
@pytest.mark.parametrize("blocks", [1, 4, 8])
@pytest.mark.parametrize("M, N", [(384, 264), (256, 1000), (256, 2040)])
def test_every_geometry_computes_every_group(M, N, blocks, two, monkeypatch):
    """What the launch is told of the rows changes no bit, whatever the groups' real lengths."""
    from moonep_b200.ops import gemm
    monkeypatch.setattr(gemm, "TWO_CTA", two)
    groups = [64, 1472, 0, 128, 448]
    gen, ends, a, b = _inputs(groups, M, N, blocks)
    G, rows = len(groups), 64 * blocks * len(groups)
    spare = torch.zeros(max(0, rows - a.shape[0]), 1, device="cuda").bfloat16()      # (told rows are rows of a)
    a, b = (torch.cat([t, spare.expand(-1, t.shape[1])]) for t in (a, b))
    base, w = (torch.randn(G, M, N, device="cuda", generator=gen) for _ in range(2))
    start, want = 0, torch.empty_like(base)
    for g, n in enumerate(groups):       # each group alone, in the geometry of its own length
        gemm.wgrad(a[start:start + n], b[start:start + n], ends[:1] * 0 + n, want[g:g + 1]) if n else want[g].zero_()
        start += n
    grad, acc, ws = torch.empty_like(base), base.clone(), w.bfloat16()
    gemm.wgrad(a, b, ends, grad, rows=rows)
    gemm.wgrad(a, b, ends, acc, accumulate=True, rows=rows)
    gemm.wgrad(a, b, ends, base.clone(), sgd=(ws, 0.25, None), rows=rows)
    gemm.check_status()
    assert torch.equal(grad, want) and torch.equal(acc, base + want)
    assert torch.equal(ws, (w.bfloat16().float() - 0.25 * want).bfloat16())
