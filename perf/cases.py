"""What a user of this framework has it do, as cases that can be timed and whose outputs can be compared.

Kinds of case, each through the call that a user's program makes:

  steps      ``TrainEngine``: optimiser steps on [B, S] token batches held in pinned host memory, one at a time
             (``train_step``) or as the pipelined loop (``train_steps``), in every training mode
  evaluate   ``TrainEngine.evaluate``: the forward-only loop over host batches between training phases
  pool_ffn   ``cluster_pool_swiglu``: the statically routed cluster-pool FFN, forward and backward
  svd_ffn    ``svd_sparse_ffn``: the per-token top-k FFN with its low-rank selector, forward and backward
  packed_ffn ``kernels.packed_swiglu_ffn``: the packed SwiGLU FFN of the operator table, forward and backward
  attention  the operator table's attention half of a block (norm, projections, rotary, causal attention, output
             projection), forward alone or with its backward
  logits     the operator table's head: final norm, tied logits, per-token cross entropy, and their backward

A training state is one in the middle of a run: seeded weights, gains and biases that have moved off their initial
values, AdamW moments and step counts of a run a thousand steps old.  Token streams are Zipf(1.1).
"""
from __future__ import annotations

import math

import torch

from speedup_thingy_b200 import kernels as K
from speedup_thingy_b200.cluster_pool import StaticClusterPoolSwiGLU, cluster_pool_swiglu
from speedup_thingy_b200.config import ExperimentConfig, ModelConfig, OutputConfig, TrainingConfig
from speedup_thingy_b200.engine import TrainEngine, parameter_shapes
from speedup_thingy_b200.svd_ffn import SVDFactorSparseFFN, svd_sparse_ffn
from speedup_thingy_b200.workloads import train_flops_per_token

DEV = "cuda:0"
STEPS = dict(kind="steps", mode="recursive_macro", B=128, S=64, d=512, heads=8, F=2048, V=2048, T=4, blocks=1, audit=0, clip=False, batches=4)


# --------------------------------------------------------------------------- the cases
def listed():
    def steps(name, **kw):
        return dict(name=name, **{**STEPS, **kw})

    return [
        # the smallest model anybody trains here (it is the one that also runs on a CPU), one synchronous step at a time
        steps("step_small", B=8, d=128, heads=4, F=512, batches=1),
        # the headline workload: depth 4, one audited sample per batch, in the pipelined loop
        steps("steps_macro_audit", audit=1),
        # the dense model it is compared with: four blocks
        steps("steps_dense", mode="dense_exact", blocks=4),
        # the shortlist head: depth 8, longer sequences, two audited samples
        steps("steps_shortlist", mode="recursive_macro_shortlist", S=128, T=8, audit=2),
        # the scale-up model, per GPU: wide, large vocabulary, longest sequences
        steps("steps_wide", B=32, S=256, d=1024, heads=16, F=4096, V=32768, T=16, batches=2),
        # the exact teacher: every sample runs the recurrent core; ragged sizes, gradient clipping
        steps("steps_exact_ragged", mode="recursive_exact", B=21, S=50, d=384, heads=6, F=1152, V=5000, clip=True),
        # the evaluation between training phases, on sizes that are no multiple of anything
        dict(name="evaluate_ragged", kind="evaluate", mode="recursive_macro", B=50, S=100, d=384, heads=6, F=1536, V=5000, T=4, blocks=1, audit=1, clip=False,
             batches=4),
        # sparse FFN modules at the benchmark's widths
        dict(name="pool_ffn", kind="pool_ffn", N=8192, d=512, F=2048, C=16, Mc=128, rank=32, dtype="float32"),
        dict(name="svd_ffn", kind="svd_ffn", N=16384, d=512, F=2048, rank=128, k=256, dtype="float32"),
        # operator table: the packed FFN over the active union of neurons
        dict(name="packed_ffn", kind="packed_ffn", N=8192, d=512, m=320, dtype="float32"),
        # ... the smallest call: the attention half of a block for a few short sequences, forward alone
        dict(name="attention_small", kind="attention", B=4, S=64, d=128, heads=4, dtype="bfloat16", backward=False),
        # ... and the head over an odd number of tokens, in training
        dict(name="logits_ragged", kind="logits", N=4107, d=512, V=8192, dtype="float32"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_model(rng):
    hd = rng.choice([32, 64, 64, 128])
    heads = max(1, round(_log(rng, 128, 1024) / hd))
    d = hd * heads
    return dict(d=d, heads=heads, F=64 * max(2, round(d * rng.uniform(2.0, 4.0) / 64)), V=8 * round(_log(rng, 1024, 32768) / 8))


def _draw_once(rng):
    kind = rng.choice(["steps"] * 6 + ["evaluate", "pool_ffn", "svd_ffn", "packed_ffn", "attention", "logits"])
    if kind in ("steps", "evaluate"):
        mode = rng.choice(["recursive_macro", "recursive_macro", "recursive_macro", "dense_exact", "recursive_macro_shortlist", "recursive_exact"])
        model = _draw_model(rng)
        S = 2 * rng.randint(8, 64 if model["d"] == 128 * model["heads"] else 128)      # (heads of 128: at most 128 positions)
        B = max(4, round(_log(rng, 256, 16384) / S))
        audited = mode in ("recursive_macro", "recursive_macro_shortlist")
        return dict(kind=kind, mode=mode, B=B, S=S, **model, T=rng.choice([4, 4, 8]), blocks=rng.choice([2, 3, 4]) if mode == "dense_exact" else 1,
                    audit=rng.choice([0, 1, 1, 2]) if audited else 0, clip=rng.random() < 0.3, batches=rng.choice([1, 4]))
    dtype = rng.choice(["float32", "bfloat16"])
    if kind == "attention":
        hd = rng.choice([32, 64, 128])
        heads = max(1, round(_log(rng, 128, 1024) / hd))
        S = rng.randint(16, 128 if hd == 128 else 256)
        return dict(kind=kind, B=max(1, round(_log(rng, 256, 16384) / S)), S=S, d=hd * heads, heads=heads, dtype=dtype, backward=rng.random() < 0.7)
    N, d = round(_log(rng, 256, 16384)), 64 * round(_log(rng, 128, 1024) / 64)
    if kind == "logits":
        return dict(kind=kind, N=N, d=d, V=8 * round(_log(rng, 1024, 32768) / 8), dtype=dtype)
    if kind == "packed_ffn":
        return dict(kind=kind, N=N, d=d, m=8 * round(_log(rng, 64, 2048) / 8), dtype=dtype)
    F = 64 * max(4, round(d * rng.uniform(2.0, 4.0) / 64))
    if kind == "pool_ffn":
        return dict(kind=kind, N=N, d=d, F=F, C=rng.choice([4, 8, 16, 32, 64]), Mc=64 * rng.randint(1, min(8, F // 64)), rank=4 * rng.randint(2, 16), dtype=dtype)
    return dict(kind=kind, N=N, d=d, F=F, rank=8 * rng.randint(4, 16), k=max(8, round(F * rng.uniform(0.05, 0.2))), dtype=dtype)


def _cost(case):
    """A bound on how long a pass takes, in the units of the largest listed one."""
    w = work(case)
    return max(w["flops"] / 5e14, w["bytes"] / 3e12)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        case = _draw_once(rng)
        if _cost(case) <= most:
            return case


# --------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(gen, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=gen, device=DEV) * std).to(dtype)


def _zipf(gen, n, vocab):
    weight = torch.arange(1, vocab + 1, device=DEV, dtype=torch.float64).pow(-1.1)
    edges = weight.cumsum(0) / weight.sum()
    return torch.searchsorted(edges, torch.rand(n, generator=gen, device=DEV, dtype=torch.float64)).clamp_(max=vocab - 1)


def _config(c):
    dense = c["mode"] == "dense_exact"
    slabs = 16 if c["F"] % 16 == 0 else 8
    model = dict(vocab_size=c["V"], d_model=c["d"], n_heads=c["heads"], d_ff=c["F"])
    if dense:
        model.update(topology="dense", n_dense_layers=c["blocks"], head_groups=1, active_head_groups=1, ffn_groups=8)
    else:
        depths = tuple(1 << i for i in range(c["T"].bit_length()))
        model.update(n_prelude=c["blocks"], n_coda=c["blocks"], t_max=c["T"], depth_choices=depths, attn_banks=1, ffn_banks=1, head_groups=c["heads"],
                     active_head_groups=max(1, c["heads"] // 4), ffn_groups=slabs, active_ffn_groups=slabs // 4, recipe_count=5, macro_rank=32)
    train = dict(mode=c["mode"], lr=3e-4, weight_decay=0.1, batch_size=c["B"], seq_len=c["S"], seed=0)
    if not dense:
        train["fixed_depth"] = c["T"]
    if c["audit"]:
        train["audit_fixed_count_per_batch"] = c["audit"]
    if c["clip"]:
        train["grad_clip_norm"] = 1.0
    out = dict(mode="shortlist", num_clusters=64, shortlist_top_clusters=2, shortlist_max_tokens=128, hard_negatives=32, random_negatives=32)
    return ExperimentConfig(ModelConfig(**model), TrainingConfig(**train), OutputConfig(**(out if c["mode"] == "recursive_macro_shortlist" else {})))


def _weights(gen, cfg):
    """Seeded weights of a run under way: matrices N(0, 0.02), gains around one, biases and FiLM vectors off zero."""
    shapes = parameter_shapes(cfg.model, cfg.output.num_clusters)
    flat = _randn(gen, sum(math.prod(s) for _, s in shapes), std=0.02)
    out, at = {}, 0
    for name, shape in shapes:
        n = math.prod(shape)
        t = flat[at:at + n].view(shape)
        at += n
        if name.endswith(("norm1.weight", "norm2.weight", "final_norm.weight", "pass_attn_scale", "pass_mlp_scale")):
            t = t + 1.0
        elif name == "core.alpha_inj":
            t = t + 0.1
        out[name] = t
    return out


def _prepare_engine(c, seed):
    gen = _gen(seed)
    cfg = _config(c)
    engine = TrainEngine(cfg, _weights(gen, cfg), device=DEV)
    for name in engine.exp_avg:                         # a run a thousand steps old
        engine.exp_avg_sq[name].fill_(1e-5)
    engine.plan.step_count.fill_(1000)
    B, S = c["B"], c["S"]
    stream = _zipf(gen, c["batches"] * B * (S + 1), c["V"]).view(c["batches"], B, S + 1).cpu()
    batches = [(s[:, :-1].contiguous().pin_memory(), s[:, 1:].contiguous().pin_memory()) for s in stream]
    return dict(kind=c["kind"], engine=engine, batches=batches)


def _leaves(*tensors):
    return [t.requires_grad_() for t in tensors]


def prepare(case, seed):
    c = dict(case)
    if c["kind"] in ("steps", "evaluate"):
        return _prepare_engine(c, seed)
    gen = _gen(seed)
    dt = getattr(torch, c["dtype"])
    d = c["d"]
    if c["kind"] == "attention":
        B, S, H = c["B"], c["S"], c["heads"]
        x, gain = _randn(gen, B, S, d, dtype=dt), 1.0 + _randn(gen, d, std=0.05)
        ws = [_randn(gen, d, d, std=d ** -0.5, dtype=dt) for _ in range(4)]
        pos = torch.arange(S, device=DEV, dtype=torch.float32)[:, None]
        freq = 10000.0 ** (-torch.arange(0, d // H, 2, device=DEV, dtype=torch.float32) / (d // H))
        angle = (pos * freq).repeat_interleave(2, dim=-1)
        state = dict(x=x, gain=gain.to(dt), ws=ws, cos=angle.cos(), sin=angle.sin(), rows=torch.arange(d, device=DEV), dims=(B, S, H, d // H), kind=c["kind"],
                     dy=_randn(gen, B, S, d, dtype=dt) if c["backward"] else None)
        if c["backward"]:
            state["leaves"] = _leaves(state["x"], state["gain"], *ws)
        return state
    N = c["N"]
    if c["kind"] == "logits":
        leaves = _leaves(_randn(gen, N, d, dtype=dt), (1.0 + _randn(gen, d, std=0.05)).to(dt), _randn(gen, c["V"], d, std=d ** -0.5, dtype=dt))
        return dict(kind=c["kind"], leaves=leaves, targets=_zipf(gen, N, c["V"]), dloss=torch.full((N,), 1.0 / N, device=DEV))
    dy = _randn(gen, N, d)
    if c["kind"] == "packed_ffn":
        m = c["m"]
        leaves = _leaves(_randn(gen, N, d, dtype=dt), _randn(gen, 2 * m, d, std=d ** -0.5, dtype=dt), _randn(gen, m, d, std=m ** -0.5, dtype=dt))
        return dict(kind=c["kind"], leaves=leaves, dy=dy.to(dt))
    F, r = c["F"], c["rank"]
    x = _randn(gen, N, d, dtype=dt)
    if c["kind"] == "pool_ffn":
        # tokens around one prototype direction per cluster, clusters of unequal popularity; the centres are what a
        # codebook build over such tokens ends with: the prototypes' selector features, normalised
        C = c["C"]
        protos = _randn(gen, C, d, std=2.0)
        share = torch.rand(C, generator=gen, device=DEV) + 0.2
        which = torch.searchsorted((share.cumsum(0) / share.sum()).contiguous(), torch.rand(N, generator=gen, device=DEV)).clamp_(max=C - 1)
        x = (protos[which] + 0.25 * _randn(gen, N, d)).to(dt)
        up_a, gate_a = (_randn(gen, d, r, std=d ** -0.5) for _ in range(2))
        centers = torch.nn.functional.normalize(torch.cat([protos @ up_a, protos @ gate_a], dim=-1), dim=-1)
        ids = torch.rand(C, F, generator=gen, device=DEV).argsort(dim=-1)[:, :c["Mc"]]
        wug, wd = _randn(gen, 2 * F, d, std=d ** -0.5), _randn(gen, d, F, std=F ** -0.5)
        module = StaticClusterPoolSwiGLU(wug, wd, dict(up_a=up_a, gate_a=gate_a), dict(centers=centers, candidate_ids=ids), rank=r, max_tokens=N)
        return dict(kind=c["kind"], module=module, leaves=_leaves(x, wug, wd), dy=dy)
    # selector factors that describe the weights they select for: the leading part of each weight is what they span
    up_a, gate_a = (_randn(gen, d, r, std=d ** -0.5) for _ in range(2))
    up_b, gate_b = (_randn(gen, r, F, std=r ** -0.5) for _ in range(2))
    w_up, w_gate = ((a @ b).t() + _randn(gen, F, d, std=0.5 * d ** -0.5) for a, b in ((up_a, up_b), (gate_a, gate_b)))
    w_down = _randn(gen, F, d, std=F ** -0.5)
    w = [t.contiguous() for t in (w_up, w_gate, w_down)]
    module = SVDFactorSparseFFN(*w, up_a, up_b, gate_a, gate_b, top_k=c["k"], up_m=c["k"], product_m=c["k"], max_tokens=N)
    return dict(kind=c["kind"], module=module, leaves=_leaves(x, *w), dy=dy)


# --------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "steps":
        engine, batches = state["engine"], state["batches"]
        if len(batches) == 1:
            losses = [engine.train_step(batches[0]).loss]
        else:
            losses = [result.loss for result in engine.train_steps(batches)]
        return dict(losses=losses, params={n: engine.params[n] for n in engine.trainable}, gradient=engine.grad_flat)
    if kind == "evaluate":
        out = state["engine"].evaluate(state["batches"])
        return dict(loss=out["eval_loss_per_sample"], nll=out["eval_nll_per_token"], last_per_sample=state["engine"].loss_per_sample)
    if kind == "attention":
        B, S, H, hd = state["dims"]
        wq, wk, wv, wo = state["ws"]
        normed, _ = K.k_fused_rmsnorm(state["x"], state["gain"])
        q, k, v = (t.view(B, S, H, hd).transpose(1, 2) for t in K.k_qkv_dense(normed, wq, wk, wv))
        q, k = K.k_rope_apply(q, k, state["cos"], state["sin"])
        y = K.k_flash_causal_dense(q, k, v)
        out = K.k_out_proj_grouped(y.transpose(1, 2).reshape(B, S, H * hd), wo, state["rows"])
        if state["dy"] is None:
            return out
        return dict(out=out.detach(), grads=torch.autograd.grad(out, state["leaves"], state["dy"]))
    leaves = state["leaves"]
    if kind == "logits":
        hidden, gain, table = leaves
        normed, _ = K.k_fused_rmsnorm(hidden, gain)
        loss = K.k_cross_entropy_unreduced(K.k_logits_full(normed, table), state["targets"])
        return dict(loss=loss.detach(), grads=torch.autograd.grad(loss, leaves, state["dloss"]))
    if kind == "packed_ffn":
        out = K.packed_swiglu_ffn(*leaves)
    elif kind == "pool_ffn":
        out = cluster_pool_swiglu(state["module"], leaves[0])
    else:
        out = svd_sparse_ffn(state["module"], leaves[0])
    return dict(out=out.detach(), grads=torch.autograd.grad(out, leaves, state["dy"]))


# --------------------------------------------------------------------------- what a pass cannot do without
def _engine_work(c):
    cfg = _config(c)
    m, tokens = cfg.model, c["B"] * c["S"]
    block = 8 * c["d"] ** 2 + 6 * c["d"] * c["F"] + 4 * c["S"] * c["d"]
    core = 3.0 * (c["T"] + (m.n_prelude + m.n_coda if c["mode"] != "dense_exact" else 0)) * block
    if c["mode"] == "recursive_exact":
        flops = tokens * (core + 6.0 * c["d"] * c["V"])
    else:
        flops = tokens * train_flops_per_token(cfg)
        if c["audit"]:                                  # the audited samples also run the recurrent core and the coda
            flops += c["audit"] * c["S"] * (core + 6.0 * c["d"] * c["V"])
    used = ["embed.", "prelude.", "coda.", "blocks.", "final_norm.", "router.recipe_mlp.", "router.depth_mlp."]
    used += ["macro."] if c["mode"] != "recursive_exact" else []
    used += ["core."] if c["mode"] == "recursive_exact" or c["audit"] else []
    n = sum(math.prod(s) for name, s in parameter_shapes(m, cfg.output.num_clusters) if name.startswith(tuple(used)))
    if c["kind"] == "evaluate":
        return dict(bytes=c["batches"] * 16.0 * tokens + 4.0 * n, flops=c["batches"] * tokens * train_flops_per_token(cfg) / 3.0)
    # per step: weights and two moments read and written, the gradient written; tokens and targets
    return dict(bytes=c["batches"] * (28.0 * n + 16.0 * tokens), flops=c["batches"] * flops)


def work(case):
    c = dict(case)
    if c["kind"] in ("steps", "evaluate"):
        return _engine_work(c)
    e, d = (4.0 if c["dtype"] == "float32" else 2.0), c["d"]
    if c["kind"] == "attention":
        N, half = c["B"] * c["S"], 8.0 * d * d + 2.0 * c["S"] * d            # (causal: half the score matrix)
        passes = 3.0 if c["backward"] else 1.0
        return dict(bytes=e * (2 * N * d + 4 * d * d) * (2.0 if c["backward"] else 1.0), flops=passes * N * half)
    N = c["N"]
    if c["kind"] == "logits":
        return dict(bytes=2 * e * (N * d + c["V"] * d) + 16.0 * N, flops=6.0 * N * d * c["V"])
    if c["kind"] == "packed_ffn":
        return dict(bytes=e * (4 * N * d + 6 * c["m"] * d), flops=18.0 * N * d * c["m"])
    io = N * d * (2 * e + 8.0) + 24.0 * c["F"] * d                               # x, dx; out, dout; dense weights and their gradients
    if c["kind"] == "pool_ffn":
        return dict(bytes=io, flops=N * (18.0 * d * c["Mc"] + 4.0 * d * c["rank"] + 4.0 * c["rank"] * c["C"]))
    # selector (two products per half), then the selected neurons, forward and backward
    return dict(bytes=io, flops=N * (4.0 * d * c["rank"] + 4.0 * c["rank"] * c["F"] + 18.0 * d * c["k"]))


def tolerance(case):
    """bf16 operands with fp32 accumulation throughout: about 1e-2 for one pass; a training run carries each step's
    rounding into the next, and a router or top-k decision on two nearly equal scores can fall the other way."""
    return {"rel": 2e-2 if case["kind"] == "steps" else 1e-2, "max": 0.9 if case["kind"] in ("steps", "pool_ffn", "svd_ffn") else 0.4}
