"""The communication tests once more with the kernels that groups over several devices use (the planner's exchange of
counts, expansion, pre-reduction, barriers between launches, one work list a rank): a virtual group takes them too when it is told
that its ranks are not on one device."""
import pytest
import torch

from tests.test_large_shapes import (test_dispatch_combine_large_stride,  # noqa: F401
                                     test_prefetch_offsets_beyond_4gib, test_reduce_grad_offsets_beyond_4gib,
                                     test_shard_is_bound_at_launch)
from tests.test_virtual_comm import (_cleanup, test_combine_scaled_rows_and_plan_reuse,  # noqa: F401
                                     test_plan_dispatch_combine_vs_oracle,
                                     test_programmatic_dependent_launch_gives_identical_results,
                                     test_zero_copy_async_and_bad_inputs)
from tests.test_virtual_weights import (test_prefetch_bf16, test_prefetch_uint8_with_scales_async,  # noqa: F401
                                        test_reduce_grad_bitwise)

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _separate(monkeypatch):
    from moonep_b200.api import Buffer
    init = Buffer.__init__

    def patched(self, *args, **kw):
        init(self, *args, **kw)
        self._one_device = False

    monkeypatch.setattr(Buffer, "__init__", patched)


@pytest.mark.parametrize("R", [1, 4])
def test_planner_exchanges_counts(R):
    """The exchange is a barrier of its own: the ranks' epochs count it, and the plan is the one made without."""
    from moonep_b200 import Buffer
    S, H, K, E = 40, 64, 2, 4 * R
    buf = Buffer(S, H, K, E, R, num_sms=3, token_padding=8, virtual=R > 1, timeout_s=2.0)
    lead = (R,) if R > 1 else ()
    gen = torch.Generator().manual_seed(R)
    topk = torch.rand(R, S, E, generator=gen).topk(K, dim=2).indices.to(torch.int32)
    tpe = torch.stack([torch.bincount(topk[r].flatten().long(), minlength=E) for r in range(R)]).to(torch.int32)
    topk, tpe = topk.reshape(*lead, S, K).cuda(), tpe.reshape(*lead, E).cuda()
    plans = []
    for one, epoch in ((False, 1), (True, 1), (False, 2)):
        buf._one_device = one
        plans.append(buf._fresh_plan(topk, tpe, topk.device, buf._stream()))
        buf.check()
        assert buf.sync_state[0, :, 1].tolist() == [epoch] * R
    for name in ("dst", "cu_seqlens", "zero_fill_ranges", "experts_to_copy", "remote_stats", "send_order"):
        a, b, c = (getattr(p, name) for p in plans)
        assert torch.equal(a, b) and torch.equal(a, c), name
    buf.destroy()
