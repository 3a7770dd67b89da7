"""Cross-entropy over bf16 logits against PyTorch's, in fp64."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _kernel_at_all_sizes(monkeypatch):
    from moonep_b200.ops import elementwise as ew
    monkeypatch.setattr(ew, "CE_MIN_CLASSES", 0)
    monkeypatch.setattr(ew, "CE_MIN_LOGITS", 0)


# one class, rows below and above a block's stride, vector and scalar rows (odd classes, odd start)
@pytest.mark.parametrize("S,V,offset", [(1, 1, 0), (3, 8, 0), (5, 33, 0), (7, 4096, 0), (64, 4104, 0), (16, 32000, 0),
                                        (9, 50257, 0), (4, 64, 3)])
@pytest.mark.parametrize("ignored", [0, 2])
def test_matches_fp64(S, V, offset, ignored):
    from moonep_b200.ops import elementwise as ew
    g = torch.Generator(device="cuda").manual_seed(S + V)
    flat = (torch.randn(S * V + offset, device="cuda", generator=g) * 4).bfloat16()
    logits = flat[offset:].view(S, V)
    targets = torch.randint(0, V, (S,), device="cuda", generator=g)
    if ignored:
        targets[-1:] = -100
    if V > 4:
        logits[0, 1:4] = float("-inf")
        targets[0] = 0
    a = logits.detach().requires_grad_(True)
    loss = ew.cross_entropy(a, targets)
    (loss * 3.0).backward()
    b = logits.detach().double().requires_grad_(True)
    want = F.cross_entropy(b, targets)
    (want * 3.0).backward()
    assert loss.dtype == torch.float32
    if S == 1 and ignored:
        assert bool(torch.isnan(loss)) and bool(torch.isnan(want))
        return
    # fp32 sum of up to 5e4 terms: 1e-5; the gradient is bf16: half an ulp of 2^-8, and the exponential's 1e-5
    assert abs(float(loss) - float(want)) <= 1e-5 * (1 + abs(float(want)))
    assert bool(((a.grad.double() - b.grad).abs() <= b.grad.abs() * (2.0 ** -8) + 1e-7).all())


def test_odd_values_and_other_forms():
    from moonep_b200.ops import elementwise as ew
    x = torch.randn(4, 48, device="cuda").bfloat16()
    x[0] = float("-inf")
    x[1, 5] = float("nan")
    x[2, 7] = float("inf")
    t = torch.tensor([1, 2, 3, 4], device="cuda")
    for r in range(4):
        got, want = ew.cross_entropy(x[r:r + 1].contiguous(), t[r:r + 1]), F.cross_entropy(x[r:r + 1].float(), t[r:r + 1])
        assert bool(torch.isnan(got)) == bool(torch.isnan(want)) == (r < 3)
    # fp32 logits, strided logits and class probabilities take the general path
    y = torch.randn(4, 96, device="cuda").bfloat16()
    p = torch.softmax(torch.randn(4, 96, device="cuda"), 1)
    for a, b in ((y.float(), t), (y[:, ::2], t), (y, p)):
        assert torch.equal(ew.cross_entropy(a, b), F.cross_entropy(a.float(), b))


@pytest.mark.parametrize("V", [48, 49])
@pytest.mark.parametrize("bad", [-1, 49, 1 << 40])
def test_target_that_is_no_class(V, bad):
    from moonep_b200.ops import elementwise as ew, gemm
    gemm.check_status()
    x = torch.randn(5, V, device="cuda").bfloat16().requires_grad_(True)
    t = torch.tensor([1, -100, 2, bad, 3], device="cuda")
    loss = ew.cross_entropy(x, t)
    loss.backward()
    assert bool(torch.isnan(loss))
    assert bool(torch.isnan(x.grad[[0, 2, 3, 4]]).all()) and bool((x.grad[1] == 0).all())
    with pytest.raises(RuntimeError, match="row 3 is not one of"):
        gemm.check_status()
    gemm.reset_status()


def test_derivatives_and_transforms():
    """Whatever ``F.cross_entropy`` can be put through: second derivatives, forward mode, vmap, tracing."""
    from moonep_b200.ops import elementwise as ew
    from torch.autograd import forward_ad
    ref = lambda a, b: F.cross_entropy(a.float(), b)
    x = torch.randn(6, 40, device="cuda").bfloat16()
    t = torch.randint(0, 40, (6,), device="cuda")

    def second(fn):
        a = x.clone().requires_grad_(True)
        g, = torch.autograd.grad(fn(a, t), a, create_graph=True)
        return torch.autograd.grad((g.float() ** 2).sum(), a)[0]

    def forward(fn):
        with forward_ad.dual_level():
            return forward_ad.unpack_dual(fn(forward_ad.make_dual(x, torch.ones_like(x) * 0.5 + x), t)).tangent

    for case in (second, forward, lambda fn: torch.func.grad(lambda a: fn(a, t))(x),
                 lambda fn: torch.func.vmap(fn)(x.view(2, 3, 40), t.view(2, 3)),
                 lambda fn: torch.jit.trace(lambda a: fn(a, t), (x,))(-x)):
        got, want = case(ew.cross_entropy), case(ref)
        assert got is not None and torch.equal(got, want)
    # a plain first derivative beside a hook on the saved tensors
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda v: packed.append(v) or v.clone(), lambda v: v):
        a = x.clone().requires_grad_(True)
        loss = ew.cross_entropy(a, t)
    loss.backward()
    assert packed and bool(torch.isfinite(a.grad).all())


# scalar rows (odd classes, odd start) answer infinities and NaN as vector rows do
@pytest.mark.parametrize("V,offset", [(49, 0), (48, 3), (48, 0), (600, 1)])
def test_odd_values_in_scalar_rows(V, offset):
    from moonep_b200.ops import elementwise as ew
    inf = float("inf")
    rows = torch.randn(6, V, device="cuda")
    rows[0] = -inf
    rows[1, 5] = float("nan")
    rows[2, 7] = inf
    rows[3, V - 1] = inf
    rows[4, ::2] = -inf
    t = torch.tensor([1, 2, 7, 3, 5, 4], device="cuda")
    for r in range(6):
        flat = torch.zeros(V + offset, device="cuda", dtype=torch.bfloat16)
        flat[offset:] = rows[r].bfloat16()
        a, b = flat[offset:].view(1, V).detach().requires_grad_(True), rows[r:r + 1].bfloat16().double().requires_grad_(True)
        got, want = ew.cross_entropy(a, t[r:r + 1]), F.cross_entropy(b, t[r:r + 1])
        got.backward()
        want.backward()
        assert bool(torch.isnan(got)) == bool(torch.isnan(want)) == (r < 4)
        assert torch.equal(torch.isnan(a.grad), torch.isnan(b.grad))
        if r >= 4:
            assert abs(float(got.detach()) - float(want.detach())) <= 1e-5 * (1 + abs(float(want.detach())))


def test_small_logits_take_the_general_path(monkeypatch):
    from moonep_b200 import _native as nat
    from moonep_b200.ops import elementwise as ew
    monkeypatch.setattr(ew, "CE_MIN_CLASSES", 1000)
    monkeypatch.setattr(ew, "CE_MIN_LOGITS", 1 << 23)
    for S, V, kernel in ((16384, 512, False), (100, 32000, False), (263, 32000, True), (8389, 1000, True)):
        x, t = torch.randn(S, V, device="cuda").bfloat16(), torch.randint(0, V, (S,), device="cuda")
        before = nat.LAUNCHES
        got, want = ew.cross_entropy(x, t), F.cross_entropy(x.float(), t)
        assert (nat.LAUNCHES > before) == kernel
        assert abs(float(got) - float(want)) <= 1e-5 * (1 + abs(float(want)))
