"""``combine`` without ``zero_copy`` copies the caller's rows into the Buffer's memory outside autograd: whatever mode
the Buffer's views were first used in, rows with a grad history are accepted and leave none behind."""
import contextlib

import pytest
import torch

from moonep_b200 import _native as nat
from moonep_b200.api import Buffer

MODES = {"grad": contextlib.nullcontext, "no_grad": torch.no_grad, "inference": torch.inference_mode}


def _host_buffer(R, H=16, NvS=8, S=4, K=2):
    """The state that ``combine`` works on, in host memory: no context, launches left out."""
    buf = object.__new__(Buffer)
    meta = 4 * NvS
    vars(buf).update(R=R, virtual=R > 1, rank=0, S=S, H=H, K=K, N=S * K, NvS=NvS, Rv=R, hidden_stride=NvS + 3, meta_stride=meta,
                     weights_off=NvS, hidden_buf=torch.zeros(R * (NvS + 3), H, dtype=torch.bfloat16), hidden_buf2=None,
                     meta_buf=torch.zeros(R * meta, dtype=torch.int32), _own_views={}, _one_device=True, _destroyed=True,
                     _ctx=0, _stats=dict(combine=0, bytes_combine=0))
    return buf


class _Plan:
    dst = torch.zeros(1, dtype=torch.int32)


@pytest.mark.parametrize("R", [1, 3])
@pytest.mark.parametrize("first", MODES)
@pytest.mark.parametrize("then", MODES)
def test_rows_with_history(monkeypatch, R, first, then):
    monkeypatch.setattr(nat, "call", lambda *a: 0)
    monkeypatch.setattr(Buffer, "_stream", staticmethod(lambda: 0))
    buf = _host_buffer(R)
    with MODES[first]():
        buf._hidden_own(), buf._weights_own()
    with MODES[then]():
        rows = torch.randn(buf._shape(buf.NvS, buf.H)).bfloat16().requires_grad_(then == "grad") * 2
        w = torch.rand(buf._shape(buf.NvS)).requires_grad_(then == "grad") * 2
        assert rows.requires_grad == (then == "grad")
        out, w_out = buf._combine_on_current_stream(_Plan, rows, w, True, False, False)
    assert not out.requires_grad and not w_out.requires_grad
    for view, want in ((buf._hidden_own(), rows), (buf._weights_own(), w)):
        assert torch.equal(view, want.detach()) and not view.requires_grad
        assert not view.detach().clone().requires_grad
    assert not buf.hidden_buf.requires_grad and not buf.meta_buf.requires_grad


@pytest.mark.gpu
def test_combine_after_a_pass_without_grad():
    S, H, K, E = 9, 128, 2, 4
    buf = Buffer(S, H, K, E, 1, num_sms=2, token_padding=16, timeout_s=2.0)
    topk = torch.tensor([[0, 1]] * 5 + [[2, 3]] * 4, dtype=torch.int32, device="cuda")
    tpe = torch.bincount(topk.flatten().long(), minlength=E).to(torch.int32)
    x = torch.randn(S, H, device="cuda").bfloat16()
    with torch.no_grad():
        rows, w, _, plan = buf.dispatch(x, torch.rand(S, K, device="cuda"), topk, tpe)
    y, _, _ = buf.combine(plan, rows.requires_grad_() * 2, w.requires_grad_() * 2)
    assert torch.equal(y, (x.float() * 4).bfloat16())
    again = buf.dispatch(x, plan=plan)[0]
    assert not again.requires_grad and not buf.hidden_nvsh_buffer_view.requires_grad
    buf.check()
    buf.destroy()
