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
         (8, 65, 1, 16, 256, 8, 2), (2, 9, 32, 64, 16384, 8, 3), (3, 50, 12, 96, 4096, 32, 49)]


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
