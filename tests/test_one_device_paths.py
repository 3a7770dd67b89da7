"""Dispatch and combine within one device (a virtual group or a lone rank) move the duplicate rows
themselves; groups over several devices expand and pre-reduce them in kernels of their own.  Both
ways make the same rows and, bit for bit, the same sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (R, S, K, E, H, padding, CTAs a rank): one token; K = 1, an odd K, K above the ring's depth; groups of one
# row; every expert on one rank; rings of 16 / 8 / 3 rows
CASES = [(1, 1, 1, 1, 8, 8, 1), (1, 37, 8, 64, 7168, 128, 16), (1, 200, 5, 16, 1024, 16, 32),
         (2, 33, 3, 8, 2560, 64, 4), (4, 19, 8, 64, 512, 16, 32), (8, 17, 8, 128, 2560, 16, 18),
         (8, 65, 1, 16, 256, 8, 2), (2, 9, 32, 64, 16384, 8, 3), (3, 50, 12, 96, 4096, 32, 49),
         # rows summed by all warps: just above 7168 elements, around 14336, several tokens a CTA
         (1, 300, 6, 16, 7176, 16, 8), (2, 160, 8, 32, 10240, 16, 8), (1, 170, 3, 8, 14336, 8, 4), (2, 90, 4, 16, 14344, 8, 2),
         (1, 200, 8, 8, 16384, 8, 32)]


@pytest.mark.parametrize("R,S,K,E,H,tp,sms", CASES)
def test_duplicates_moved_directly_match_the_separate_kernels(R, S, K, E, H, tp, sms):
    from moonep_b200 import Buffer
    buf = Buffer(S, H, K, E, R, num_sms=sms, token_padding=tp, virtual=R > 1, timeout_s=2.0)
    g = torch.Generator().manual_seed(S * 31 + K)
    lead = (R,) if R > 1 else ()
    pop = torch.rand(E, generator=g) * 3
    topk = (torch.rand(R, S, E, generator=g) + pop).topk(K, dim=2).indices.to(torch.int32)
    tpe = torch.stack([torch.bincount(topk[r].flatten().long(), minlength=E) for r in range(R)]).to(torch.int32)
    topk, tpe = topk.reshape(*lead, S, K).cuda(), tpe.reshape(*lead, E).cuda()
    x = torch.randn(*lead, S, H, generator=g).bfloat16().cuda()
    w = torch.rand(*lead, S, K, generator=g).cuda()

    def rounds():
        h, wn, cu, plan = buf.dispatch(x, w, topk, tpe)
        scale = torch.linspace(0.1, 2.0, buf.NvS, device="cuda")[:, None]
        h2, _, _, _ = buf.dispatch(-x, plan=plan)
        y, wb, _ = buf.combine(plan, (h.float() * scale).bfloat16(), wn)
        buf.check()
        rows = cu.reshape(R, -1)[:, -1].tolist()
        cut = lambda t: [t.reshape(R, *t.shape[len(lead):])[r, :rows[r]] for r in range(R)]
        return cut(h) + cut(h2) + cut(wn) + cut(plan.link) + cut(plan.src_info) + [y, wb, plan.dst, cu]

    assert buf._one_device
    direct = rounds()
    buf._one_device = False
    separate = rounds()
    for a, b in zip(direct, separate):
        assert torch.equal(a, b)
    assert torch.equal(direct[-3], w)
    buf.destroy()


# (R, experts a rank, elements an expert): one chunk, ragged last chunks, several chunks; CTAs a rank
WEIGHT_CASES = [(2, 1, 8, 1), (2, 3, 4096, 2), (4, 8, 20000, 5), (8, 16, 70008, 18), (3, 5, 4104, 32)]


@pytest.mark.parametrize("R,epn,n,sms", WEIGHT_CASES)
@pytest.mark.parametrize("zero", [True, False])
def test_weights_moved_from_one_list_match_one_list_a_rank(R, epn, n, sms, zero):
    """``prefetch_weight`` / ``reduce_grad`` share one work list between all ranks' CTAs within one device;
    same bytes, same order of the additions."""
    from moonep_b200 import Buffer, CommPlan
    buf = Buffer(16, 64, 1, R * epn, R, num_sms=sms, token_padding=8, virtual=True, timeout_s=2.0)
    g = torch.Generator().manual_seed(n + R)
    etc = torch.where(torch.rand(R, epn, generator=g) < 0.6, torch.randint(0, R * epn, (R, epn), generator=g),
                      torch.full((R, epn), -1)).to(torch.int32).cuda()[None].expand(R, R, epn).contiguous()
    z = lambda *s: torch.zeros(*s, dtype=torch.int32, device="cuda")
    plan = CommPlan(dst=z(R, buf.N), experts_to_copy=etc, zero_fill_ranges=z(R, 2 * epn, 2), remote_stats=z(R, 2),
                    cu_seqlens=z(R, 2 * epn), link=z(R, buf.NvS), N=buf.N, R=R, E=buf.E, NvS=buf.NvS, K=buf.K)
    rnd = lambda: torch.randn(R, epn, n, generator=g).cuda()
    w, grads, slots = [rnd().bfloat16() for _ in range(3)], [rnd() for _ in range(3)], [rnd() for _ in range(3)]
    names = ("gate", "up", "down")

    def both(one):
        buf._one_device = one
        pool = [torch.full_like(t, 7.0) for t in w]
        buf.prefetch_weight(plan, **{f"local_{a}_weight": t for a, t in zip(names, w)},
                            **{f"{a}_prefetch_buffer": t for a, t in zip(names, pool)})
        gr, sl = [t.clone() for t in grads], [t.clone() for t in slots]
        buf.reduce_grad(plan, zero_consumed=zero, **{f"local_{a}_grad": t for a, t in zip(names, gr)},
                        **{f"{a}_reduce_buffer": t for a, t in zip(names, sl)})
        buf.check()
        return pool + gr + sl

    for a, b in zip(both(True), both(False)):
        assert torch.equal(a, b)
    buf.destroy()
