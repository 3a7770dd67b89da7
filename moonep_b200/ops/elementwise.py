"""Wrappers of the bandwidth kernels in ``csrc/device/elementwise.cu`` (router top-k / softmax /
histogram and its backward, SwiGLU backward, cross-entropy, fused SGD).  None of these exist in the reference,
which stops at communication; they are the remaining hot ops of the MoE layer."""
from __future__ import annotations

import torch

from .. import _native as nat
from .._native import F, I, L, P
from .gemm import status_word

nat.declare("mep_router_topk", I, [P, P, I, I, I, P, P, P, P])
nat.declare("mep_router_topk_bwd", I, [P, P, P, I, I, I, P, P])
nat.declare("mep_swiglu_bwd", I, [P, P, P, P, P, I, I, P, P, P, P])
nat.declare("mep_ce_fwd", I, [P, P, L, I, I, P, P, P, P, P])
nat.declare("mep_ce_bwd", I, [P, P, L, I, I, P, P, P, P, P])
nat.declare("mep_sgd_update", I, [P, P, P, I, F, P])
nat.declare("mep_sgd_update_masked", I, [P, P, L, L, P, F, P])


def _st():
    return nat.stream()


def _rc(rc, what):
    if rc != 0:
        raise RuntimeError(f"{what}: {nat.last_error()} (code {rc})")


def router_topk(logits: torch.Tensor, K: int, bias: torch.Tensor | None = None):
    """Top-``K`` experts of ``logits + bias`` per token, softmax gate weights over the selected
    unbiased logits, and the tokens-per-expert histogram.  Returns ``(topk[S,K] int32,
    weights[S,K] fp32, tpe[E] int32)``."""
    assert logits.dtype == torch.float32 and logits.is_contiguous() and logits.is_cuda
    S, E = logits.shape
    topk = torch.empty(S, K, dtype=torch.int32, device=logits.device)
    w = torch.empty(S, K, dtype=torch.float32, device=logits.device)
    tpe = torch.empty(E, dtype=torch.int32, device=logits.device)
    if bias is not None:
        assert bias.dtype == torch.float32 and bias.numel() == E
    _rc(nat.call("mep_router_topk", logits.data_ptr(), nat.ptr(bias), S, E, K, topk.data_ptr(),
                 w.data_ptr(), tpe.data_ptr(), _st()), "router_topk")
    return topk, w, tpe


def router_topk_bwd(weights, dweights, topk, E: int) -> torch.Tensor:
    """``dlogits[S,E]`` bf16 (softmax backward, zero outside the selected experts)."""
    S, K = weights.shape
    assert dweights.dtype == torch.float32 and dweights.is_contiguous()
    out = torch.empty(S, E, dtype=torch.bfloat16, device=weights.device)
    _rc(nat.call("mep_router_topk_bwd", weights.data_ptr(), dweights.data_ptr(), topk.data_ptr(),
                 S, E, K, out.data_ptr(), _st()), "router_topk_bwd")
    return out


def swiglu_bwd(dact, gate, up, row_scale=None, rows_ptr=None, want_dscale=True):
    """Backward of ``act = silu(gate) * up * row_scale``: ``(dgate, dup, dscale[rows] | None)``.
    ``rows_ptr`` (device int32) bounds the rows that are processed without a host sync."""
    rows, Hp = dact.shape
    for t in (dact, gate, up):
        assert t.dtype == torch.bfloat16 and t.is_contiguous()
    dgate, dup = torch.empty_like(dact), torch.empty_like(dact)
    dscale = torch.empty(rows, dtype=torch.float32, device=dact.device) if want_dscale else None
    _rc(nat.call("mep_swiglu_bwd", dact.data_ptr(), gate.data_ptr(), up.data_ptr(),
                 nat.ptr(row_scale), nat.ptr(rows_ptr), rows, Hp, dgate.data_ptr(), dup.data_ptr(),
                 nat.ptr(dscale), _st()), "swiglu_bwd")
    return dgate, dup, dscale


def _sgd_pair(w, g):
    assert w.dtype == torch.bfloat16 and g.dtype == torch.float32 and w.numel() == g.numel()
    assert w.is_contiguous() and g.is_contiguous()


def sgd_update_all_(pairs, lr: float) -> None:
    """:func:`sgd_update_` of up to eight ``(w, g)`` pairs in one launch."""
    n = len(pairs)
    w, g, size = (P * n)(), (P * n)(), (L * n)()
    for i, (wi, gi) in enumerate(pairs):
        _sgd_pair(wi, gi)
        w[i], g[i], size[i] = wi.data_ptr(), gi.data_ptr(), wi.numel()
    _rc(nat.call("mep_sgd_update", w, g, size, n, float(lr), _st()), "sgd_update")


def sgd_update_(w: torch.Tensor, g: torch.Tensor, lr: float, only: torch.Tensor = None) -> None:
    """In place ``w(bf16) = bf16(w - lr * g(fp32))``.  ``only`` (int32 ``[experts]``, with ``w`` and
    ``g`` shaped ``[experts, ...]``) restricts the update to the experts whose flag is non-zero."""
    if only is None:
        sgd_update_all_(((w, g),), lr)
        return
    _sgd_pair(w, g)
    assert only.dtype == torch.int32 and only.is_cuda and only.numel() >= w.shape[0]
    _rc(nat.call("mep_sgd_update_masked", w.data_ptr(), g.data_ptr(), w.shape[0], w[0].numel(),
                 only.data_ptr(), float(lr), _st()), "sgd_update")


class _CrossEntropy(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logits, targets, ignore_index):
        S, V = logits.shape
        f32 = dict(dtype=torch.float32, device=logits.device)
        lse, loss, mean_n = torch.empty(S, **f32), torch.empty(S, **f32), torch.empty(2, **f32)
        _rc(nat.call("mep_ce_fwd", logits.data_ptr(), targets.data_ptr(), ignore_index, S, V, lse.data_ptr(),
                     loss.data_ptr(), mean_n.data_ptr(), status_word(logits.device).data_ptr(), _st()), "cross_entropy")
        ctx.ignore_index = ignore_index
        ctx.save_for_backward(logits, targets, lse, mean_n)
        return mean_n[0].clone()

    @staticmethod
    def backward(ctx, g):
        logits, targets, lse, mean_n = ctx.saved_tensors
        if torch.is_grad_enabled():        # create_graph: a gradient that can be differentiated again
            loss = torch.nn.functional.cross_entropy(logits.float(), targets, ignore_index=ctx.ignore_index)
            return torch.autograd.grad(loss, logits, g, create_graph=True)[0], None, None
        S, V = logits.shape
        grad = torch.empty_like(logits)
        _rc(nat.call("mep_ce_bwd", logits.data_ptr(), targets.data_ptr(), ctx.ignore_index, S, V, lse.data_ptr(),
                     mean_n.data_ptr(), g.contiguous().data_ptr(), grad.data_ptr(), _st()), "cross_entropy backward")
        return grad, None, None


# Where the kernel is the faster way (forward + backward, against F.cross_entropy).  It gives a block to a row,
# which with few classes idles: 32768 x 512 239 us against 198, x 1000 274 against 325, 65536 x 128 429 against 179.
# Issued eagerly its host work is 105 us whatever the size, F.cross_entropy's 90: 4M logits 106 against 90, 8M 105
# against 105 - 115, 16M 105 against 175 - 215.  Captured in a graph only the device counts: 2M 23 against 49.
CE_MIN_CLASSES, CE_MIN_LOGITS = 1000, 1 << 23


def _kernel_pays(S: int, V: int) -> bool:
    return V >= CE_MIN_CLASSES and (S * V >= CE_MIN_LOGITS or torch.cuda.is_current_stream_capturing())


def _eager(*tensors) -> bool:
    """True if nothing stands between these tensors and their memory: no tracer, dispatch mode, subclass,
    functorch transform or forward-mode tangent, which a kernel of our own would pass by."""
    return (not torch.jit.is_tracing() and not torch.compiler.is_compiling()
            and torch._C._len_torch_dispatch_stack() == 0
            and all(type(t) in (torch.Tensor, torch.nn.Parameter) and not torch._C._functorch.is_functorch_wrapped_tensor(t)
                    and torch.autograd.forward_ad.unpack_dual(t).tangent is None for t in tensors))


def cross_entropy(logits: torch.Tensor, targets: torch.Tensor, ignore_index: int = -100) -> torch.Tensor:
    """``F.cross_entropy(logits.float(), targets)`` (mean over the rows whose target is not
    ``ignore_index``) for bf16 ``logits [S, V]`` and int64 ``targets [S]`` on the GPU, without the
    fp32 copies; the gradient is rounded to bf16 once, as there.  Other sizes (``CE_MIN_LOGITS``),
    other forms of the arguments, other devices than the current one, tracing, ``vmap``, forward-mode
    and second derivatives go to ``F.cross_entropy``.

    For a target that is neither ``ignore_index`` nor a class ``F.cross_entropy`` stops the device with
    an assertion; the kernel makes the loss and all gradients NaN, and ``gemm.check_status`` raises."""
    if (logits.is_cuda and logits.dtype == torch.bfloat16 and logits.dim() == 2 and _kernel_pays(*logits.shape)
            and _eager(logits, targets)
            and logits.device.index == torch.cuda.current_device() and logits.is_contiguous()
            and targets.device == logits.device and targets.dtype == torch.int64
            and tuple(targets.shape) == (logits.shape[0],) and targets.is_contiguous()):
        return _CrossEntropy.apply(logits, targets, ignore_index)
    return torch.nn.functional.cross_entropy(logits.float(), targets, ignore_index=ignore_index)
