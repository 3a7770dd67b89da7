"""Kernels around the layer's products at the edges of their ranges: SwiGLU backward by warps, the update of several
tensors in one launch, a lone rank's dispatch straight into the tensors that are kept."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hp", [8, 264, 520, 2048, 2312])       # part of a warp, one block of 256 columns and a bit, ...
@pytest.mark.parametrize("rows, valid", [(1, 1), (37, 0), (300, 261), (900, 790)])     # (wide rows a block each, else a warp)
def test_swiglu_bwd_widths(rows, valid, Hp):
    from moonep_b200.ops import elementwise as ew
    gen = torch.Generator(device="cuda").manual_seed(Hp + rows)
    d, g, u = [torch.randn(rows, Hp, device="cuda", generator=gen).bfloat16() for _ in range(3)]
    w = torch.rand(rows, device="cuda", generator=gen) + 0.5
    dg, du, ds = ew.swiglu_bwd(d, g, u, w, rows_ptr=torch.tensor([valid], dtype=torch.int32, device="cuda"))
    assert not bool(ds[valid:].any())
    d, g, u, w = d[:valid].double(), g[:valid].double(), u[:valid].double(), w[:valid].double()[:, None]
    s = torch.sigmoid(g)
    # |g| < 6: the exponential is off by at most 9 units of 2^-24, s and each product by one more; so 2^-19 of a
    # term's size.  bf16 results add 2^-8 of themselves, the sum at most Hp additions.
    factor = s * (1 + g * (1 - s))
    size = (d * u * w).abs() * (1 + g.abs())
    assert bool(((dg[:valid].double() - d * u * w * factor).abs() <= 2.0 ** -8 * (d * u * w * factor).abs() + 2.0 ** -19 * size).all())
    want = d * g * s * w
    assert bool(((du[:valid].double() - want).abs() <= (2.0 ** -8 + 2.0 ** -19) * want.abs()).all())
    terms = d * g * s * u
    assert bool(((ds[:valid].double() - terms.sum(1)).abs() <= (2.0 ** -19 + Hp * 2.0 ** -24) * terms.abs().sum(1)).all())


@pytest.mark.parametrize("sizes", [(5,), (8, 3, 4096), (1 << 20, 17, 8, 7, 300000, 1, 16, 2056)])
def test_update_of_several_tensors(sizes):
    from moonep_b200.ops import elementwise as ew
    gen = torch.Generator(device="cuda").manual_seed(len(sizes))
    w = [torch.randn(n, device="cuda", generator=gen).bfloat16() for n in sizes]
    g = [torch.randn(n, device="cuda", generator=gen) for n in sizes]
    # 0.25 g is exact, so the sum is rounded to fp32 once and then to bf16, as here
    want = [(a.float() - 0.25 * b).bfloat16() for a, b in zip(w, g)]
    ew.sgd_update_all_(list(zip(w, g)), 0.25)
    assert all(torch.equal(a, b) for a, b in zip(w, want))


def test_update_refuses_more_than_a_launch_takes():
    from moonep_b200.ops import elementwise as ew
    t = [(torch.zeros(8, device="cuda", dtype=torch.bfloat16), torch.zeros(8, device="cuda")) for _ in range(9)]
    with pytest.raises(RuntimeError):
        ew.sgd_update_all_(t, 1.0)


@pytest.mark.parametrize("shard", [0, 1])
@pytest.mark.parametrize("S, H, K, E, pad", [(1, 128, 1, 8, 64), (53, 1024, 4, 32, 64), (260, 7168, 8, 64, 128)])
def test_lone_dispatch_equals_dispatch(S, H, K, E, pad, shard):
    from moonep_b200 import Buffer
    buf = Buffer(S, H, K, E, 1, num_sms=4, token_padding=pad, timeout_s=5.0)
    if shard:
        buf.enable_second_shard()
    gen = torch.Generator(device="cuda").manual_seed(S)
    x = torch.randn(S, H, device="cuda", generator=gen).bfloat16()
    w = torch.rand(S, K, device="cuda", generator=gen)
    topk = torch.stack([torch.randperm(E, device="cuda", generator=gen)[:K] for _ in range(S)]).to(torch.int32)
    tpe = torch.bincount(topk.flatten().long(), minlength=E).to(torch.int32)
    rows, wr, cu, plan = buf.dispatch(x, w, topk, tpe)
    n = int(cu[-1])
    real = plan.src_info[:n] >= 0
    assert int(real.sum()) == S * K
    for keep in (True, False):
        # what is not written shows
        buf.hidden_view(shard).fill_(float("nan"))
        buf.router_weight_buffer_view.fill_(float("nan"))
        rows2, wr2, cu2, plan2 = buf._dispatch_lone(x, w, topk, tpe, keep=keep, shard=shard)
        for name in ("dst", "zero_fill_ranges", "cu_seqlens"):
            assert torch.equal(getattr(plan, name), getattr(plan2, name)), name
        for name in ("link", "src_info"):
            assert torch.equal(getattr(plan, name)[:n], getattr(plan2, name)[:n]), name
        assert torch.equal(rows[:n][real], rows2[:n][real])
        assert torch.equal(wr[:n], wr2[:n])
        padding = rows2[:n][~real]
        assert bool(torch.isnan(padding).all() if not keep else (padding == 0).all())
    buf.destroy()


@pytest.mark.parametrize("fused_combine", [True, False])
@pytest.mark.parametrize("in_place", [False, True])
def test_inference_reads_no_padding_row(fused_combine, in_place):
    """A pass without a backward pass leaves padding rows as they are: whatever they hold stays out of the result."""
    from moonep_b200 import Buffer
    from moonep_b200.models.moe_layer import MoELayer
    buf = Buffer(77, 256, 4, 16, 1, num_sms=8, token_padding=128, timeout_s=5.0)
    layer = MoELayer(buf, 192, seed=1, train=False, fused_combine=fused_combine, hidden_in_place=in_place)
    x = torch.randn(77, 256, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2)).bfloat16()
    got = []
    for fill in (0.0, float("nan"), float("inf")):
        for shard in range(1 + in_place):
            buf.hidden_view(shard).fill_(fill)
        with torch.no_grad():
            got.append(layer(x))
    assert bool(torch.isfinite(got[0]).all()) and bool(got[0].any())
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    buf.destroy()
