"""Launches by Buffer.  Shared memory of dispatch and planner over several devices: they and the weight
ops wait for other ranks on two streams, so where they can share an SM they have to keep room for one another."""
import pytest

from moonep_b200 import _native as nat
import moonep_b200.api  # noqa: F401  (declares the entries)

SM_SHARED, PER_CTA = 228 * 1024, 1024 + 1024      # what the system keeps for a CTA, and static parts


@pytest.fixture
def ctx():
    made = []

    def make(R, E, S, K, H, num_sms=32, virt=0, local=148):
        c = nat.call("mep_ctx_create", 0, R, virt, E, S, K, H, 128, num_sms, local, num_sms, 0, 0, 0, 0, 0, 0, 0, 10 ** 9)
        assert c, nat.last_error()
        made.append(c)
        return c

    yield make
    for c in made:
        nat.call("mep_ctx_destroy", c)


@pytest.mark.parametrize("R", [2, 8])
@pytest.mark.parametrize("H", [256, 1024, 2048, 2560, 4096, 5120])
def test_dispatch_beside_reduce_grad(ctx, R, H):
    E = 256
    smem = nat.call("mep_dispatch_smem_bytes", ctx(R, E, 4096, 8, H))
    lists = 4 * (3 * (E // R) + E)
    assert smem + (128 * 1024 + lists) + 2 * PER_CTA <= SM_SHARED
    assert nat.call("mep_dispatch_smem_bytes", ctx(1, E, 4096, 8, H)) == 17 * 2 * H      # one device: the deep ring


@pytest.mark.parametrize("R", [2, 8])
@pytest.mark.parametrize("E", [64, 256, 1024])
@pytest.mark.parametrize("S,num_sms", [(16, 32), (4096, 32), (8192, 8)])
def test_planner_beside_prefetch_weight(ctx, R, E, S, num_sms):
    smem = nat.call("mep_plan_launch_smem_bytes", ctx(R, E, S, 8, 1024, num_sms))
    lists = 4 * (4 * (E // R) + E)
    assert smem + (192 * 1024 + lists) + 2 * PER_CTA <= SM_SHARED


# ranks on the device, num_sms, local SMs -> CTAs a rank
@pytest.mark.parametrize("R,num_sms,local,want", [(1, 8, 148, 148), (1, 32, 148, 148), (1, 148, 148, 148), (1, 32, 16, 32),
                                                  (8, 2, 148, 18), (8, 18, 148, 18), (8, 32, 148, 32), (2, 8, 148, 74)])
def test_few_communication_sms_on_one_device(ctx, R, num_sms, local, want):
    """Dispatch and combine that move all rows themselves run on no fewer SMs than the local kernels they replace."""
    assert nat.call("mep_ctx_direct_ctas", ctx(R, 64, 512, 8, 1024, num_sms, int(R > 1), local)) == want


# ranks of a virtual group, CTAs a rank for its copy kernels -> CTAs a rank of the planner
@pytest.mark.parametrize("R,num_sms,S,want", [(8, 18, 4096, 18), (32, 8, 512, 4), (128, 2, 512, 1), (2, 148, 8192, 74),
                                              (32, 8, 16, 1), (1, 96, 4096, 96)])
def test_planner_of_a_virtual_group_fits_one_cta_an_sm(ctx, R, num_sms, S, want):
    c = ctx(R, 6 * R, S, 8, 1024, num_sms, int(R > 1))
    assert nat.call("mep_plan_launch_ctas", c) == want
    assert want * R <= 148 and nat.call("mep_plan_launch_smem_bytes", c) <= 227 * 1024 - 1024


@pytest.mark.gpu
def test_virtual_group_of_more_ctas_than_sms():
    """32 ranks x 8 CTAs: the copy kernels' CTAs share SMs, the planner's cannot."""
    import torch
    from moonep_b200 import Buffer, reference as ref
    from moonep_b200.utils.routing import routing_for_maxvio, tokens_per_expert
    R, S, H, K, E, tp = 32, 40, 256, 4, 96, 16
    buf = Buffer(S, H, K, E, R, num_sms=8, token_padding=tp, virtual=True, timeout_s=5.0)
    topk, w, _, _ = routing_for_maxvio(S, K, E, R, 1.0, seed=4)
    tpe = torch.stack([tokens_per_expert(topk[r], E) for r in range(R)])
    x = torch.randn(R, S, H, generator=torch.Generator().manual_seed(2)).bfloat16()
    rows, wn, _, plan = buf.dispatch(x.cuda(), w.cuda(), topk.cuda(), tpe.cuda())
    y, wb, _ = buf.combine(plan, rows, wn)
    buf.check()
    assert torch.equal(plan.dst.cpu(), ref.plan_all_ranks(topk, S, K, E, tp, tpe)[1])
    assert torch.equal(y.cpu(), (x.float() * K).bfloat16()) and torch.equal(wb.cpu(), w)
    buf.destroy()
