"""The work that programs built on this framework have it do, as cases of one pass each.

Sizes are those of the repository's own configurations (the DeepSeek-V3-shaped layer with H=7168,
H'=2048, top-8; the decoder with hidden 2048, H'=768, 128 experts; the reduced benchmark layer with
H=1024, H'=512) and generic ones between them.  One GPU holds either one rank's share of a layer
(R = 1, the per-rank workload of an expert-parallel group) or a whole virtual group of R ranks.

Kinds of case
  step      MoE layer: forward, backward, optimizer step (applied in the weight-grad kernels, or fp32
            grads stored for an optimizer of the user's own)
  forward   MoE layer, inference
  group     dispatch / combine of a whole group in both directions: fresh plan, rows out, rows
            home, then the gradients back through the same plan
  weights   the redundant experts' weights out, their gradients home
  decoder   decoder stack, loss and gradients
"""
import sys

import torch

from moonep_b200 import Buffer
from moonep_b200 import reference
from moonep_b200.models.decoder import MoEDecoder
from moonep_b200.models.moe_layer import MoELayer
from moonep_b200.utils.graph import GraphedStep


def listed():
    return [
        # a decoding batch of 16 sequences on a rank that holds 32 experts: the weights of nearly
        # every expert are read for a handful of rows each, launches and latency count
        dict(name="forward_decode_16", kind="forward", S=16, H=7168, Hp=2048, K=8, E=32, pad=128, zipf=0.3),
        # prompt processing with a ragged number of tokens on the same rank
        dict(name="forward_prefill_1531", kind="forward", S=1531, H=7168, Hp=2048, K=8, E=32, pad=128, zipf=0.5),
        # training step of the benchmark layer, one rank's share of 8 ranks (1024 rows an expert)
        dict(name="step_32_experts", kind="step", S=4096, H=7168, Hp=2048, K=8, E=32, pad=128, zipf=0.5, sgd=True, graph=True),
        # the same layer sharded over 2 ranks: 128 experts of 256 rows, a stream over the weights
        dict(name="step_128_experts", kind="step", S=4096, H=7168, Hp=2048, K=8, E=128, pad=128, zipf=0.5, sgd=True, graph=True),
        # the decoder's layer with fp32 grads kept for the user's optimizer, issued eagerly
        dict(name="step_stored_grads", kind="step", S=4096, H=2048, Hp=768, K=8, E=128, pad=128, zipf=0.5, sgd=False, graph=False),
        # the reduced layer with an odd number of tokens and short padding (stand-alone dispatch)
        dict(name="step_small_odd", kind="step", S=509, H=1024, Hp=512, K=4, E=32, pad=64, zipf=0.5, sgd=False, graph=False),
        # the communication benchmark's shape, all 8 ranks
        dict(name="group_8x4096", kind="group", R=8, S=4096, H=7168, K=8, E=256, pad=128, zipf=0.6),
        # a few tokens a rank, as while decoding
        dict(name="group_8x17", kind="group", R=8, S=17, H=2560, K=8, E=128, pad=16, zipf=0.3),
        # one rank on its own: every expert is local, all K rows of a token are copies
        dict(name="group_1x4096", kind="group", R=1, S=4096, H=7168, K=8, E=256, pad=128, zipf=0.6),
        # weight movement for a strongly skewed routing, decoder's expert size
        dict(name="weights_8x16", kind="weights", R=8, S=512, H=2048, Hp=768, K=8, E=128, pad=128, zipf=1.0),
        # two blocks of the decoder with its vocabulary
        dict(name="decoder_2_blocks", kind="decoder", S=4096, H=2048, Hp=768, K=8, E=128, pad=128, zipf=0.8,
             layers=2, heads=16, vocab=32000),
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], spread over its logarithm."""
    return int(round(lo * (hi / lo) ** rng.random()))


def _multiple(rng, of, lo, hi):
    return max(lo, min(hi, int(round(_log_int(rng, lo, hi) / of)) * of))


HIDDEN = (1024, 1536, 2048, 2560, 4096, 5120, 7168)


def draw(rng):
    kind = rng.choice(["forward", "forward", "step", "step", "step", "group", "group", "weights", "decoder"])
    c = dict(kind=kind, K=rng.choice([2, 4, 6, 8, 8]), zipf=round(rng.uniform(0.0, 1.0), 2))
    if kind == "forward":
        c.update(S=_log_int(rng, 1, 4096), H=rng.choice(HIDDEN), Hp=_multiple(rng, 64, 512, 2048),
                 E=8 * _log_int(rng, 1, 16), pad=rng.choice([64, 128, 128]))
    elif kind == "step":
        graph = rng.random() < 0.5
        c.update(S=_log_int(rng, 256, 4096), H=rng.choice(HIDDEN), Hp=_multiple(rng, 64, 512, 2048),
                 E=8 * _log_int(rng, 1, 16), pad=rng.choice([64, 128, 128]), sgd=rng.random() < 0.5, graph=graph)
    elif kind == "group":
        R = rng.choice([1, 2, 4, 8])
        c.update(R=R, S=_log_int(rng, 4, 4096), H=rng.choice((512, 1024, 1536, 2560, 4096, 5120, 7168)), E=R * _log_int(rng, 8, 32),
                 pad=rng.choice([16, 64, 128, 128]))
    elif kind == "weights":
        R = rng.choice([2, 4, 8])
        c.update(R=R, S=_log_int(rng, 64, 1024), H=_multiple(rng, 128, 512, 2048), Hp=_multiple(rng, 64, 256, 1024),
                 E=R * _log_int(rng, 8, 16), pad=128, zipf=round(rng.uniform(0.5, 1.5), 2))
    else:
        heads = rng.choice([8, 16])
        c.update(S=8 * _log_int(rng, 16, 512), H=heads * 128, Hp=_multiple(rng, 64, 256, 768), E=8 * _log_int(rng, 2, 16),
                 pad=128, layers=rng.choice([1, 2]), heads=heads, vocab=8 * _log_int(rng, 500, 4000))
    return c


# ---- state ------------------------------------------------------------------------------------
class State:
    """What a program keeps between passes.  A Buffer's peer mappings are given back explicitly."""

    buf = step = None

    def __del__(self):
        self.step = None
        if self.buf is not None and not sys.is_finalizing():
            self.buf.destroy()


def _generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + salt)


def _popularity(E, zipf, gen):
    """Logarithm of a Zipf popularity over a random order of the experts."""
    ranks = torch.randperm(E, device="cuda", generator=gen).float() + 1.0
    return -float(zipf) * torch.log(ranks)


def _layer(buf, case, seed, train, **kw):
    layer = MoELayer(buf, case["Hp"], None, seed=int(seed), train=train, **kw)
    layer.router_bias = _popularity(case["E"], case["zipf"], _generator(seed, 3)).contiguous()
    return layer


def _prepare_layer(case, seed):
    st = State()
    S, H = case["S"], case["H"]
    train = case["kind"] == "step"
    # one GPU: the dispatch is a local copy, 96 CTAs as in the benchmark
    st.buf = Buffer(S, H, case["K"], case["E"], 1, num_sms=96, token_padding=case["pad"])
    st.layer = layer = _layer(st.buf, case, seed, train, hidden_in_place=train)
    g = _generator(seed, 5)
    st.x = torch.randn(S, H, device="cuda", generator=g).bfloat16()
    if not train:
        return st
    # upstream gradient; it changes its sign from pass to pass, so that the weights of a state that
    # is stepped many times stay where they are
    st.dy = torch.randn(S, H, device="cuda", generator=g).bfloat16()
    st.dy = [st.dy, -st.dy]
    lr = 0.005 / (S * case["K"] / case["E"])      # a step changes a weight by a few hundredths
    if case["sgd"]:
        layer.fuse_sgd(lr)

    def step(x, dy):
        x = x.detach().requires_grad_(True)
        y = layer(x)
        y.backward(dy)
        layer.sgd_step(lr)
        return y.detach(), x.grad

    st.step = GraphedStep(step, [st.x, st.dy[0]], warmup=1) if case["graph"] else step
    return st


def _routing(case, seed, device="cuda"):
    """``topk [R, S, K]``, softmax gate weights, ``tokens_per_expert [R, E]``."""
    R, S, E = case["R"], case["S"], case["E"]
    if device == "cuda":
        g = _generator(seed, 7)
        logits = torch.randn(R, S, E, device="cuda", generator=g) + _popularity(E, case["zipf"], g)
    else:
        g = torch.Generator().manual_seed(int(seed))
        logits = torch.randn(R, S, E, generator=g) - case["zipf"] * torch.log(torch.randperm(E, generator=g).float() + 1.0)
    val, idx = torch.topk(logits, case["K"], dim=2)
    tpe = torch.zeros(R, E, dtype=torch.int32, device=device)
    flat = idx.reshape(R, -1)
    tpe.scatter_add_(1, flat, torch.ones_like(flat, dtype=torch.int32))
    return idx.to(torch.int32).contiguous(), torch.softmax(val, dim=2).contiguous(), tpe


def _group_buffer(case):
    R = case["R"]
    # as many CTAs a rank as the ranks of a virtual group can have at once; 96 for a lone rank
    return Buffer(case["S"], case["H"], case["K"], case["E"], R, num_sms=min(32, 144 // R) if R > 1 else 96,
                  token_padding=case["pad"], virtual=R > 1)


def _prepare_group(case, seed):
    st = State()
    st.buf = _group_buffer(case)
    lead = (case["R"],) if case["R"] > 1 else ()
    topk, w, tpe = _routing(case, seed)
    st.topk, st.w, st.tpe = (t if lead else t[0] for t in (topk, w, tpe))
    g = _generator(seed, 11)
    st.x = torch.randn(*lead, case["S"], case["H"], device="cuda", generator=g).bfloat16()
    st.dy = torch.randn(*lead, case["S"], case["H"], device="cuda", generator=g).bfloat16()
    # gradients of the dispatched route weights, as the expert FFN's backward leaves them
    st.dw = torch.randn(*lead, st.buf.NvS, device="cuda", generator=g)
    return st


def _prepare_weights(case, seed):
    st = State()
    st.buf = _group_buffer(case)
    R, epn, H, Hp = case["R"], case["E"] // case["R"], case["H"], case["Hp"]
    topk, w, tpe = _routing(case, seed)
    g = _generator(seed, 13)
    x = torch.zeros(R, case["S"], H, dtype=torch.bfloat16, device="cuda")
    st.plan = st.buf.dispatch(x, w, topk, tpe, zero_copy=True)[3]

    def normal(std, dtype):
        return (torch.randn(R, epn, H, Hp, device="cuda", generator=g) * std).to(dtype)

    names = ("gate", "up", "down")
    st.weights = {f"local_{n}_weight": normal(0.02, torch.bfloat16) for n in names}
    st.slots = {f"{n}_prefetch_buffer": torch.zeros(R, epn, H, Hp, dtype=torch.bfloat16, device="cuda") for n in names}
    st.grads = {f"local_{n}_grad": normal(1e-3, torch.float32) for n in names}
    st.replicas = {f"{n}_reduce_buffer": normal(1e-3, torch.float32) for n in names}
    return st


def _prepare_decoder(case, seed):
    st = State()
    st.buf = Buffer(case["S"], case["H"], case["K"], case["E"], 1, num_sms=96, token_padding=case["pad"])
    torch.manual_seed(int(seed))
    with torch.device("cuda"):
        st.model = MoEDecoder(case["vocab"], case["H"], case["layers"], case["heads"],
                              lambda i: _layer(st.buf, case, int(seed) + 31 * i, True))
    g = _generator(seed, 17)
    st.tokens = torch.randint(0, case["vocab"], (case["S"],), device="cuda", generator=g)
    st.targets = (st.tokens * 31 + 7) % case["vocab"]
    return st


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "forward"):
        st = _prepare_layer(case, seed)
    else:
        st = {"group": _prepare_group, "weights": _prepare_weights, "decoder": _prepare_decoder}[kind](case, seed)
    st.kind = kind
    st.sgd = case.get("sgd", False)
    return st


# ---- one pass ---------------------------------------------------------------------------------
def run(st):
    if st.kind == "forward":
        with torch.no_grad():
            return st.layer(st.x)
    if st.kind == "step":
        y, dx = st.step(st.x, st.dy[0])
        st.dy.reverse()
        out = dict(y=y, dx=dx)
        # with the optimizer inside the weight-grad kernels the weights are the result, else the
        # grads are kept too
        out.update(st.layer.parameters() if st.sgd else st.layer.grads())
        return out
    if st.kind == "group":
        buf = st.buf
        rows, _, cu, plan = buf.dispatch(st.x, st.w, st.topk, st.tpe, zero_copy=True, router_weights_zero_copy=True)
        y, _, _ = buf.combine(plan, rows, None, zero_copy=True)
        rows, _, _, _ = buf.dispatch(st.dy, plan=plan, zero_copy=True)
        dx, dw, _ = buf.combine(plan, rows, st.dw, zero_copy=True)
        return dict(y=y, dx=dx, dw=dw, cu_seqlens=cu, dst=plan.dst)
    if st.kind == "weights":
        st.buf.prefetch_weight(st.plan, **st.weights, **st.slots)
        st.buf.reduce_grad(st.plan, **st.grads, **st.replicas)
        return dict(**st.slots, **st.grads, **st.replicas)
    model = st.model
    for p in model.parameters():
        p.grad = None
    loss = model(st.tokens, st.targets)
    loss.backward()
    out = dict(loss=loss.detach(), dense=[p.grad for p in model.parameters()])
    out["experts"] = [m.grads() for m in model.moe_layers()]
    return out


# ---- what a pass cannot do without --------------------------------------------------------------
def _experts_used(S, K, E):
    return E * (1.0 - (1.0 - K / E) ** S) if K < E else E


def work(case):
    S, H, K, E = case["S"], case["H"], case["K"], case["E"]
    kind = case["kind"]
    if kind in ("group", "weights"):
        R = case["R"]
    if kind == "group":
        # forward and backward: token rows read, K rows each written, read again, token rows written
        return {"bytes": 2.0 * R * S * H * 2 * (2 + 2 * K) + 8.0 * R * S * K * 4, "flops": 2.0 * R * S * K * H}
    if kind == "weights":
        topk, _, tpe = _routing(case, 0, "cpu")
        etc = reference.plan_all_ranks(topk, S, K, E, case["pad"], tpe)[0].experts_to_copy
        slots = int((etc >= 0).sum())
        homes = len(set(etc[etc >= 0].tolist()))
        n = 3.0 * H * case["Hp"]
        # weights: each expert read once, each slot written; grads: slots read and cleared, home
        # grads read and written
        return {"bytes": n * (2 * (homes + slots) + 4 * (2 * slots + 2 * homes)), "flops": n * slots}
    Hp, layers = case["Hp"], case.get("layers", 1)
    used = _experts_used(S, K, E)
    expert = 3.0 * H * Hp
    router = H * E
    if kind == "forward":
        return {"bytes": 2 * (used * expert + router + 2 * S * H), "flops": 2.0 * S * (K * expert + router)}
    # forward, grads of the rows, grads of the weights: three contractions; the weights are read,
    # and updated in place or their fp32 grads written
    step_flops = 6.0 * S * (K * expert + router)
    step_bytes = 2 * (used * expert + router) + (2 * used if case.get("sgd") else 4 * E) * expert + 2.0 * 4 * S * H
    if kind == "step":
        return {"bytes": step_bytes, "flops": step_flops}
    V = case["vocab"]
    dense = 4.0 * H * H
    attention = 2.0 * 2.0 * S * S * H / 2
    return {"bytes": layers * (step_bytes + 4 * dense) + 4.0 * 2 * V * H,
            "flops": layers * (step_flops + 6.0 * S * dense + 3.5 * attention) + 6.0 * S * V * H}


def tolerance(case):
    # bf16 rows, weights and outputs around fp32 sums.  A token whose K-th and next logit agree to
    # fp32 rounding may take the other expert, which changes that row alone ("max").
    if case["kind"] == "group":
        return {"rel": 4e-3, "max": 0.02}
    if case["kind"] == "weights":
        return {"rel": 1e-6, "max": 1e-5}
    return {"rel": 1e-2, "max": 0.9}
