"""The communication tests once more with the kernels that groups over several devices use (expansion,
pre-reduction, barriers between launches, one work list a rank): a virtual group takes them too when it is told
that its ranks are not on one device."""
import pytest

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
