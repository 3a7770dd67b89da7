"""Token-major grouped products over ragged groups: token tiles of every size, padding ranges, column
tails, CTA pairs and single CTAs, against fp32 products of the same bf16 operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# real rows of the groups: around the 32-token step and the 256-token tile, several tiles, empty groups
VALID = [1, 0, 31, 32, 33, 64, 0, 160, 255, 256, 257, 300, 513, 700]


@pytest.mark.parametrize("two", [0, 1])
@pytest.mark.parametrize("pad,with_pads", [(64, True), (128, True), (64, False), (1, False)])
@pytest.mark.parametrize("H,Hp", [(256, 192), (640, 64), (1152, 328)])
def test_ragged_groups(H, Hp, pad, with_pads, two, monkeypatch):
    from moonep_b200.ops import gemm
    monkeypatch.setattr(gemm, "TWO_CTA", two)
    g = torch.Generator(device="cuda").manual_seed(H + pad)
    G, split = len(VALID), 9
    padded = [(v + pad - 1) // pad * pad for v in VALID]
    ends = torch.tensor(padded).cumsum(0)
    starts = ends - torch.tensor(padded)
    rows = int(ends[-1])
    cu = ends.to(torch.int32).cuda()
    pads = torch.tensor([[s + v, n - v] if n > v else [0, 0] for s, v, n in zip(starts.tolist(), VALID, padded)],
                        dtype=torch.int32).cuda()
    real = torch.zeros(rows, dtype=torch.bool, device="cuda")
    for s, v in zip(starts.tolist(), VALID):
        real[s:s + v] = True
    kw = dict(split=split, pads=pads if with_pads else None)

    def mk(*shape, std=1.0):
        t = (torch.randn(*shape, device="cuda", generator=g) * std).bfloat16()
        return t

    x, a, dg, du = mk(rows, H), mk(rows, Hp), mk(rows, Hp), mk(rows, Hp)
    for t in (x, a, dg, du):
        t[~real] = 0
    wg, wu, wd = (mk(G, H, Hp, std=0.05) for _ in range(3))
    sl = lambda w: (w[:split].contiguous(), w[split:].contiguous())
    (wg0, wg1), (wu0, wu1), (wd0, wd1) = sl(wg), sl(wu), sl(wd)
    scale = torch.rand(rows, device="cuda", generator=g) + 0.5

    def ref(fn):
        out = []
        for i, (s, n) in enumerate(zip(starts.tolist(), padded)):
            out.append(fn(slice(s, s + n), i))
        return torch.cat(out)

    def close(got, want):
        # bf16 result of an fp32 sum: half a bf16 ulp of the value (2^-9), and the order of the sum (<= 1200
        # terms of |a b| ~ 0.04: 1e-5); pads exactly zero
        assert torch.all(got[~real] == 0)
        assert torch.all((got.float() - want).abs() <= want.abs() * 2.0 ** -8 + 2e-4)

    new = lambda n: torch.full((rows, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    act, gate, up = gemm.gateup_swiglu(x, wg0, wu0, cu, wg_slot=wg1, wu_slot=wu1, row_scale=scale,
                                       out=(new(Hp), new(Hp), new(Hp)), **kw)
    close(gate, ref(lambda r, i: x[r].float() @ wg[i].float()))
    close(up, ref(lambda r, i: x[r].float() @ wu[i].float()))
    gf, uf = gate.float(), up.float()
    close(act, gf / (1 + torch.exp(-gf)) * uf * scale[:, None])
    act2, none_g, none_u = gemm.gateup_swiglu(x, wg0, wu0, cu, wg_slot=wg1, wu_slot=wu1, row_scale=scale,
                                              save_gate_up=False, **kw)
    assert none_g is None and none_u is None and torch.equal(act2[:rows], act)
    close(gemm.down(a, wd0, cu, wd_slot=wd1, out=new(H), **kw), ref(lambda r, i: a[r].float() @ wd[i].float().t()))
    close(gemm.down_dgrad(x, wd0, cu, wd_slot=wd1, out=new(Hp), **kw), ref(lambda r, i: x[r].float() @ wd[i].float()))
    close(gemm.gateup_dgrad(dg, du, wg0, wu0, cu, wg_slot=wg1, wu_slot=wu1, out=new(H), **kw),
          ref(lambda r, i: dg[r].float() @ wg[i].float().t() + du[r].float() @ wu[i].float().t()))
    # later groups only, on a limited grid: the first groups' rows stay untouched
    out = new(Hp)
    gemm.down_dgrad(x, wd0, cu, wd_slot=wd1, out=out, g_begin=split, grid=6, **kw)
    first = int(starts[split])
    assert torch.isnan(out[:first].float()).all()
    assert torch.equal(out[first:], gemm.down_dgrad(x, wd0, cu, wd_slot=wd1, **kw)[first:])
    # skipped blocks of zeros leave the weight grads as they are, bit for bit
    if with_pads and H % 128 == 0:
        mkg = lambda: (torch.zeros(split, H, Hp, device="cuda"), torch.zeros(G - split, H, Hp, device="cuda"))
        (l0, s0), (l1, s1) = mkg(), mkg()
        gemm.wgrad(x, a, cu, l0, grad_slot=s0, split=split)
        gemm.wgrad(x, a, cu, l1, grad_slot=s1, split=split, pads=pads)
        assert torch.equal(l0, l1) and torch.equal(s0, s1)
    gemm.check_status()


@pytest.mark.parametrize("two", [0, 1])
@pytest.mark.parametrize("pad,with_pads", [(64, True), (128, False), (1, False)])
@pytest.mark.parametrize("H,Hp", [(256, 192), (640, 64), (328, 128)])
def test_pushed_rows_of_ragged_groups(H, Hp, pad, with_pads, two, monkeypatch):
    """The push epilogue stores what the plain one stores, each real row at its entry's slot, and nothing else."""
    from moonep_b200.ops import gemm
    monkeypatch.setattr(gemm, "TWO_CTA", two)
    g = torch.Generator(device="cuda").manual_seed(H + pad)
    G, split, ranks = len(VALID), 9, 3
    padded = torch.tensor([(v + pad - 1) // pad * pad for v in VALID])
    ends = padded.cumsum(0)
    starts, rows, n_real = (ends - padded).tolist(), int(ends[-1]), sum(VALID)
    cu = ends.to(torch.int32).cuda()
    pads = torch.tensor([[s + v, n - v] if n > v else [0, 0] for s, v, n in zip(starts, VALID, padded.tolist())],
                        dtype=torch.int32).cuda()
    real = torch.cat([torch.arange(s, s + v) for s, v in zip(starts, VALID)]).cuda()
    entries = n_real // ranks + 40                        # (of which some get no row)
    slots = torch.randperm(ranks * entries, device="cuda", generator=g)[:n_real]
    src = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
    src[real] = slots.to(torch.int32)
    stride = entries * H + 64                             # elements between the ranks' staging buffers

    def mk(*shape, std=1.0):
        return (torch.randn(*shape, device="cuda", generator=g) * std).bfloat16()

    a, dg, du = mk(rows, Hp), mk(rows, Hp), mk(rows, Hp)
    for t in (a, dg, du):
        t[src < 0] = 0
    wd, wg, wu = (mk(G, H, Hp, std=0.05) for _ in range(3))
    sl = lambda w: (w[:split].contiguous(), w[split:].contiguous())
    (wd0, wd1), (wg0, wg1), (wu0, wu1) = sl(wd), sl(wg), sl(wu)
    kw = dict(split=split, pads=pads if with_pads else None)
    down = lambda **k: gemm.down(a, wd0, cu, wd_slot=wd1, **kw, **k)
    dgrad = lambda **k: gemm.gateup_dgrad(dg, du, wg0, wu0, cu, wg_slot=wg1, wu_slot=wu1, **kw, **k)
    for op in (down, dgrad):
        staging = torch.full((ranks, stride), float("nan"), dtype=torch.bfloat16, device="cuda")
        assert op(push=dict(src_info=src, push_base=staging, push_rank_stride=stride, push_entries=entries,
                            push_ranks=ranks)) is None
        want = torch.full((ranks * entries, H), float("nan"), dtype=torch.bfloat16, device="cuda")
        want[slots] = op()[real]
        bits = lambda t: t.contiguous().view(torch.int16)
        assert torch.equal(bits(staging[:, :entries * H]), bits(want.view(ranks, -1)))
        assert torch.isnan(staging[:, entries * H:].float()).all()
    gemm.check_status()
