"""Row sizes whose rings take just under 48 KB of dynamic shared memory: with the kernels' static part
the launch needs more than 48 KB, which has to be allowed explicitly."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [1728, 1920, 2048, 2688, 2880, 3072])
def test_dispatch_combine_just_below_48k(H):
    from moonep_b200 import Buffer
    from moonep_b200.utils.routing import pattern_topk
    R, S, K, epn = 2, 8, 2, 2
    buf = Buffer(S, H, K, R * epn, R, num_sms=2, token_padding=8, virtual=True, timeout_s=2.0)
    pairs = [pattern_topk("all_remote", S, K, epn, R, r) for r in range(R)]
    topk, tpe = (torch.stack([p[i] for p in pairs]).cuda() for i in range(2))
    x = torch.randn(R, S, H, device="cuda").bfloat16()
    rows, _, _, plan = buf.dispatch(x, None, topk, tpe)
    y, _, _ = buf.combine(plan, rows)
    buf.check()
    assert torch.equal(y, (x.float() * K).bfloat16())
    buf.destroy()
