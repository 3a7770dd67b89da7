"""Launch shapes of the pushed combine's local sum: with several devices it has to fit on an SM beside
``reduce_grad`` (both wait for other ranks), and a virtual group may want more CTAs than there are SMs."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

SM_REGISTERS, SM_SHARED = 65536, 228 * 1024


@pytest.mark.parametrize("R,E", [(2, 256), (8, 256), (8, 2048)])
def test_fits_beside_reduce_grad(R, E):
    from moonep_b200 import _native as nat
    import moonep_b200.api  # noqa: F401  (declares the entries)
    v = [ctypes.c_int() for _ in range(4)]
    p = [ctypes.byref(x) for x in v]
    assert nat.call("mep_push_reduce_footprint", p[0], p[1]) == 0, nat.last_error()
    assert nat.call("mep_grad_reduce_footprint", R, E, p[2], p[3]) == 0, nat.last_error()
    push_regs, push_smem, reduce_regs, reduce_smem = [x.value for x in v]
    assert push_regs + reduce_regs <= SM_REGISTERS and push_smem + reduce_smem <= SM_SHARED


# (ranks, CTAs a rank): within the SMs, and two CTAs an SM; an H with a ragged share of vectors a thread
@pytest.mark.parametrize("R,sms", [(2, 8), (2, 148), (4, 74)])
@pytest.mark.parametrize("S,K,H", [(5, 3, 8), (300, 9, 1032)])
def test_sum_at_both_launch_shapes(R, sms, S, K, H):
    from moonep_b200 import Buffer
    E = 16 * R
    g = torch.Generator(device="cuda").manual_seed(S + R)
    topk = torch.rand(R, S, E, device="cuda", generator=g).topk(K, dim=2).indices.to(torch.int32)
    tpe = torch.stack([torch.bincount(t.flatten().long(), minlength=E) for t in topk]).to(torch.int32)
    mk = lambda n: Buffer(S, H, K, E, R, num_sms=n, token_padding=8, virtual=True, timeout_s=2.0)
    plans, buf = mk(4), mk(sms)      # (a plan of any Buffer of these sizes will do)
    plan = plans.dispatch(torch.zeros(R, S, H, dtype=torch.bfloat16, device="cuda"), None, topk, tpe)[3]
    buf.enable_push()
    rows = torch.randn(R, S, K, H, device="cuda", generator=g).bfloat16()
    buf.push_buf.view(R, buf.push_stride)[:, :S * K * H] = rows.reshape(R, -1)
    scalar = torch.rand(R, buf.NvS, device="cuda", generator=g)
    want = torch.zeros(R, S, H, device="cuda")
    for k in range(K):
        want += rows[:, :, k].float()
    raw = torch.where(plan.dst < 0, -plan.dst - 1, plan.dst).long()
    for sc in (None, scalar):        # without scalars there is no barrier
        y, w = buf.combine_pushed(plan, sc)
        buf.check()
        assert torch.equal(y, want.bfloat16())
    assert torch.equal(w.reshape(R, -1), scalar.reshape(-1)[raw])
    plans.destroy()
    buf.destroy()
