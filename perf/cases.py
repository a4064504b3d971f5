"""What is measured of this engine's speed: its whole steps and its layers, through the entry points a program calls.

`listed` names the cases, `draw` gives more of the same ranges, `prepare` makes what a program holds before the call (weights,
caches, a step's context, inputs), `run` is the call, `work` what the call cannot do without, `exact` the same results in
64 bits from plain torch.

Kinds:
    decode      one decode step of a Qwen3 dense model through the engine's captured graphs (`Engine.graphs.run`): what every
                generated token costs.  The sampled tokens are read back, the logits are what is compared.
    step        one step of prompt portions, alone or beside decoding requests, through the step function
                (`ModelRunner.step`): prompts as a server takes them in.
    attention   a grouped-query attention layer over a prompt (`parts`: what a program that builds its own model calls).
    wkv, state_space, delta, linear, latent
                the mixers of the other designs, over a batch of prompts and, behind it, one more token a request (the
                recurrent state is carried from the one step to the other), or in two portions.
    experts     a routed feed-forward over a step's tokens.
Weights follow the law the engine's own random mode uses (matrices N(0, 0.02), norms 1 + N(0, 0.01)); decays are spread over
the values trained models of the kind have.
"""
from __future__ import annotations

import math
import random
from types import SimpleNamespace

import torch
import torch.nn.functional as F

BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
DTYPES = {"bfloat16": BF16, "float32": F32}
DEV = "cuda"

SHAPES = {   # hidden, intermediate, query heads, kv heads, tied head; heads of 128
    "8b": dict(hidden=4096, inter=12288, heads=32, kv_heads=8, tied=False),
    "0.6b": dict(hidden=1024, inter=3072, heads=16, kv_heads=8, tied=True),
}
THETA, EPS = 1e6, 1e-6


# ------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # a chat with one user on a small model: launches and their latency
        dict(name="decode 0.6b x1", kind="decode", shape="0.6b", layers=28, vocab=151936, batch=1, context=512, ragged=False),
        # the headline workload's batch and context, four of its layers
        dict(name="decode 8b x8", kind="decode", shape="8b", layers=4, vocab=32768, batch=8, context=2048, ragged=False),
        # a full server: requests of very different age
        dict(name="decode 8b x64", kind="decode", shape="8b", layers=2, vocab=32768, batch=64, context=3000, ragged=True),
        # the headline prompt, whole
        dict(name="prompt 8b 2048", kind="step", shape="8b", layers=4, vocab=32768, portions=1, tokens=2048, behind=0, decoding=0,
             context=0),
        # two prompts coming in 256 tokens a step (the default portion) beside requests that decode
        dict(name="mixed 8b 2x256+24", kind="step", shape="8b", layers=4, vocab=32768, portions=2, tokens=256, behind=1536,
             decoding=24, context=1100),
        # a long document, not a multiple of any tile
        dict(name="attention 8191", kind="attention", dtype="bfloat16", hidden=4096, heads=32, kv_heads=8, seqs=1, tokens=8191,
             ragged=False, window=0),
        # Kolorax's recurrent mixer over a batch of prompts of different length
        dict(name="wkv 8 prompts", kind="wkv", dtype="bfloat16", hidden=2048, heads=32, rank=64, seqs=8, tokens=1024, ragged=True,
             tail=1),
        # Pepolorn's state-space mixer: four prompts of 2048 tokens, the design benchmark's batch
        dict(name="state space 4x2048", kind="state_space", dtype="bfloat16", hidden=1024, state=128, groups=8, seqs=4, tokens=2048,
             ragged=False, tail=1),
        # Kefisun's delta rule, the same batch
        dict(name="delta 4x2048", kind="delta", dtype="bfloat16", hidden=1024, heads=8, kv_heads=4, decay="channel", seqs=4,
             tokens=2048, ragged=False, tail=1),
        # Gatutar's gated linear attention: few prompts, cut into two portions, odd lengths
        dict(name="linear 3x1500", kind="linear", dtype="bfloat16", hidden=2048, heads=16, dim=64, decay="channel", seqs=3, tokens=1501,
             ragged=True, tail=333),
        # Papusun's latent attention inside a window
        dict(name="latent 8x2048", kind="latent", dtype="bfloat16", hidden=1024, heads=8, q_rank=512, window=1024, seqs=8, tokens=2048,
             ragged=True),
        # Mumopel's routed feed-forward over a full step
        dict(name="experts 8192", kind="experts", form="chosen", hidden=1024, ff=512, shared_ff=1024, experts=16, top=4, tokens=8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "step", "attention", "wkv", "state_space", "delta", "linear", "latent", "experts"])
    if kind == "decode":
        shape = rng.choice(["0.6b", "8b"])
        batch = _log_int(rng, 1, 64)
        return dict(kind=kind, shape=shape, layers=rng.randint(2, 4) if shape == "8b" else rng.randint(4, 28), vocab=32768, batch=batch,
                    context=_log_int(rng, 64, 4096 if batch <= 32 else 2500), ragged=rng.random() < 0.5)
    if kind == "step":
        shape = rng.choice(["0.6b", "8b"])
        portions = rng.randint(1, 4)
        decoding = rng.choice([0, 0, _log_int(rng, 1, 48)])
        return dict(kind=kind, shape=shape, layers=rng.randint(2, 4), vocab=32768, portions=portions,
                    tokens=_log_int(rng, 65, 2048 // portions), behind=rng.choice([0, rng.randint(1, 2000)]), decoding=decoding,
                    context=rng.randint(100, 2000) if decoding else 0)
    if kind == "experts":
        width = rng.choice([1024, 2048])
        form = rng.choice(["chosen", "groups", "on_input"])
        return dict(kind=kind, form=form, hidden=width, ff=width // 2, shared_ff=width, experts=rng.choice([16, 32]), top=4,
                    tokens=_log_int(rng, 600, 8192))
    seqs = _log_int(rng, 1, 12)
    tokens = _log_int(rng, 150, min(4096, 12288 // seqs))
    out = dict(kind=kind, dtype="bfloat16", seqs=seqs, tokens=tokens, ragged=rng.random() < 0.5)
    if kind == "attention":
        hidden, heads, kv = rng.choice([(4096, 32, 8), (1024, 16, 8), (1024, 8, 2), (5120, 64, 8)])
        return dict(out, hidden=hidden, heads=heads, kv_heads=kv, window=rng.choice([0, 0, 1024]))
    width = rng.choice([1024, 2048])
    out["hidden"] = width
    if kind == "latent":
        form = rng.choice([dict(q_rank=0, window=0), dict(q_rank=width // 2, window=1024)])
        return dict(out, heads=width // (64 if not form["q_rank"] else 128), **form)
    out["tail"] = rng.choice([1, 1, rng.randint(2, 700)])
    if rng.random() < 1 / 6:      # the 32-bit engine that checks the other
        out.update(dtype="float32", tokens=min(tokens, 1 + 3072 // seqs))
    if kind == "wkv":
        return dict(out, heads=width // 64, rank=64)
    if kind == "state_space":
        return dict(out, state=rng.choice([64, 128]), groups=rng.choice([1, 8]))
    heads = width // 128
    if kind == "delta":
        return dict(out, heads=heads, kv_heads=max(1, heads // 2), decay=rng.choice(["channel", "head"]))
    decay = rng.choice(["constant", "channel"])
    return dict(out, heads=heads, dim=128 if decay == "constant" else 64, decay=decay)


def _lens(n, tokens, ragged):
    """The requests' lengths: all alike, or spread from about a fifth of the longest up to it."""
    if not ragged or n == 1:
        return [tokens] * n
    r = random.Random(1000 * n + tokens)
    return [tokens] + [max(1, int(tokens * r.uniform(0.2, 1.0))) for _ in range(n - 1)]


# ------------------------------------------------------------------------------------------------ inputs
class _Rand:
    """Draws on the device, the same for the same seed."""

    def __init__(self, seed, dtype):
        self.g, self.dtype = torch.Generator(device=DEV).manual_seed(int(seed) * 1009 + 5), dtype

    def mat(self, *shape, std=0.02):
        return (torch.randn(*shape, generator=self.g, device=DEV, dtype=F32) * std).to(self.dtype)

    def norm(self, *shape):
        return (1 + 0.01 * torch.randn(*shape, generator=self.g, device=DEV, dtype=F32)).to(self.dtype)

    def vec(self, *shape, std=1.0, mean=0.0):
        return torch.randn(*shape, generator=self.g, device=DEV, dtype=F32) * std + mean

    def uniform(self, lo, hi, *shape):
        return torch.rand(*shape, generator=self.g, device=DEV, dtype=F32) * (hi - lo) + lo

    def ids(self, vocab, n):
        return torch.randint(0, vocab, (n,), generator=self.g, device=DEV).tolist()

    def step_bias(self, *shape):
        """The inverse softplus of steps spread over their logarithm from 0.001 to 0.1."""
        step = torch.exp(self.uniform(math.log(1e-3), math.log(1e-1), *shape))
        return step + torch.log(-torch.expm1(-step))


def _qwen_config(case):
    s = SHAPES[case["shape"]]
    return dict(architectures=["Qwen3ForCausalLM"], hidden_size=s["hidden"], intermediate_size=s["inter"], num_hidden_layers=case["layers"],
                num_attention_heads=s["heads"], num_key_value_heads=s["kv_heads"], head_dim=128, vocab_size=case["vocab"],
                max_position_embeddings=8192, rms_norm_eps=EPS, rope_theta=THETA, tie_word_embeddings=s["tied"])


def _qwen_weights(case, rnd):
    s, V = SHAPES[case["shape"]], case["vocab"]
    H, I, nq, nkv, d = s["hidden"], s["inter"], s["heads"], s["kv_heads"], 128
    w = {"model.embed_tokens.weight": rnd.mat(V, H)}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        w.update({p + "self_attn.q_proj.weight": rnd.mat(nq * d, H), p + "self_attn.k_proj.weight": rnd.mat(nkv * d, H),
                  p + "self_attn.v_proj.weight": rnd.mat(nkv * d, H), p + "self_attn.o_proj.weight": rnd.mat(H, nq * d),
                  p + "self_attn.q_norm.weight": rnd.norm(d), p + "self_attn.k_norm.weight": rnd.norm(d),
                  p + "mlp.gate_proj.weight": rnd.mat(I, H), p + "mlp.up_proj.weight": rnd.mat(I, H), p + "mlp.down_proj.weight": rnd.mat(H, I),
                  p + "input_layernorm.weight": rnd.norm(H), p + "post_attention_layernorm.weight": rnd.norm(H)})
    w["model.norm.weight"] = rnd.norm(H)
    if not s["tied"]:
        w["lm_head.weight"] = rnd.mat(V, H)
    return w


def _requests(case):
    """(tokens in the cache, new tokens) of every request of a whole-model case, decoding ones first."""
    if case["kind"] == "decode":
        return [(n, 1) for n in _lens(case["batch"], case["context"], case["ragged"])]
    return [(n, 1) for n in _lens(case["decoding"], max(1, case["context"]), True)] + [(case["behind"], case["tokens"])] * case["portions"]


def _qwen_inputs(case, seed):
    rnd = _Rand(seed, BF16)
    w = _qwen_weights(case, rnd)
    return w, [rnd.ids(case["vocab"], old + new) for old, new in _requests(case)]


def _part_inputs(case, seed):
    """(kind of part, its parameters, its position part's parameters or None, weights, input rows of the steps)."""
    dtype = DTYPES[case.get("dtype", "bfloat16")]
    rnd = _Rand(seed, dtype)
    kind, W = case["kind"], case["hidden"]
    pos = None
    if kind == "attention":
        nq, nkv, d = case["heads"], case["kv_heads"], 128
        par = ("gqa_attention", dict(hidden_size=W, num_heads=nq, num_kv_heads=nkv, head_dim=d, qk_norm=True, qk_norm_eps=EPS,
                                     window=case["window"] or None))
        pos = dict(head_dim=d, rotary_dim=d, theta=THETA, max_positions=8192)
        w = {"q_proj.weight": rnd.mat(nq * d, W), "k_proj.weight": rnd.mat(nkv * d, W), "v_proj.weight": rnd.mat(nkv * d, W),
             "o_proj.weight": rnd.mat(W, nq * d), "q_norm.weight": rnd.norm(d), "k_norm.weight": rnd.norm(d)}
    elif kind == "wkv":
        h, hd, r = case["heads"], case["heads"] * 64, case["rank"]
        par = ("wkv", dict(hidden_size=W, heads=h, dim=64, decay_rank=r, eps=EPS))
        w = {f"mu.{s}": rnd.uniform(0.0, 1.0, W) for s in "rkvgw"}
        w.update({s: rnd.mat(hd, W) for s in "rkvg"})
        # decays from long memory to short, as trained mixers of this kind start
        w.update({"w1": rnd.mat(r, W), "w2": rnd.mat(hd, r), "w0": rnd.uniform(-6.0, -1.0, hd), "u": rnd.vec(h, 64, std=0.3),
                  "norm": rnd.norm(hd).float(), "o": rnd.mat(W, hd)})
    elif kind == "state_space":
        V, N, G = 64, case["state"], case["groups"]
        inner = 2 * W
        h = inner // V
        C = inner + 2 * G * N
        par = ("state_space", dict(hidden_size=W, heads=h, vdim=V, state=N, groups=G, conv=4, norm_groups=G, eps=EPS))
        w = {"in": rnd.mat(2 * inner + 2 * G * N + h, W), "conv": rnd.vec(C, 4, std=0.3), "conv.b": rnd.vec(C, std=0.1),
             "dt_bias": rnd.step_bias(h), "A_log": torch.log(rnd.uniform(1.0, 16.0, h)), "D": torch.ones(h, device=DEV),
             "norm": rnd.norm(inner).float(), "o": rnd.mat(W, inner)}
    elif kind == "delta":
        h, g, D, V, r = case["heads"], case["kv_heads"], 128, 128, 64
        head = case["decay"] == "head"
        n_a = h if head else h * D
        params = dict(hidden_size=W, heads=h, kv_heads=g, dim=D, vdim=V, conv=4, eps=EPS)
        par = ("gated_delta", params) if head else ("channel_delta", dict(params, decay_rank=r, gate_rank=r))
        w = {"q": rnd.mat(g * D, W), "k": rnd.mat(g * D, W), "v": rnd.mat(h * V, W), "b": rnd.mat(h, W), "o": rnd.mat(W, h * V),
             "q.conv": rnd.vec(g * D, 4, std=0.3), "k.conv": rnd.vec(g * D, 4, std=0.3), "v.conv": rnd.vec(h * V, 4, std=0.3),
             "dt_bias": rnd.step_bias(n_a), "A_log": torch.log(rnd.uniform(1.0, 16.0, h)), "norm": rnd.norm(V).float()}
        if head:
            w.update({"a": rnd.mat(n_a, W), "g": rnd.mat(h * V, W)})
        else:
            w.update({"a1": rnd.mat(r, W), "a2": rnd.mat(n_a, r), "g1": rnd.mat(r, W), "g2": rnd.mat(h * V, r)})
    elif kind == "linear":
        h, D, V = case["heads"], case["dim"], 128
        params = dict(hidden_size=W, heads=h, dim=D, vdim=V, eps=EPS)
        w = {"q": rnd.mat(h * D, W), "k": rnd.mat(h * D, W), "v": rnd.mat(h * V, W), "g": rnd.mat(h * V, W), "o": rnd.mat(W, h * V)}
        if case["decay"] == "constant":
            par = ("linear_attention", dict(params, decay=_constant_decays(h)))
            w["norm"] = rnd.norm(h * V).float()
        else:
            par = ("gated_linear_attention", dict(params, decay_rank=16, tau=16.0))
            w.update({"a1": rnd.mat(16, W), "a2": rnd.mat(h * D, 16, std=0.1), "a2.b": rnd.vec(h * D), "norm": rnd.norm(V).float()})
    elif kind == "latent":
        h, rank = case["heads"], 192
        D = V = 128 if case["q_rank"] else 64
        params = dict(hidden_size=W, heads=h, dim=D, rot_dim=64, vdim=V, kv_rank=rank, scale=(D + 64) ** -0.5, eps=EPS)
        w = {"dkv": rnd.mat(rank + 64, W), "dkv.norm": rnd.norm(rank).float(), "uk": rnd.mat(h * D, rank, std=0.07), "uv": rnd.mat(h * V, rank, std=0.07),
             "o": rnd.mat(W, h * V)}
        pos = dict(head_dim=64, rotary_dim=64, theta=1e4, max_positions=0)
        if case["q_rank"]:
            params.update(q_rank=case["q_rank"], window=case["window"], gate="head")
            pos["pairing"] = "interleaved"
            w.update({"dq": rnd.mat(case["q_rank"], W), "dq.norm": rnd.norm(case["q_rank"]).float(),
                      "uq": rnd.mat(h * (D + 64), case["q_rank"], std=0.04), "g": rnd.mat(h, W)})
        else:
            w.update({"q": rnd.mat(h * (D + 64), W), "g": rnd.mat(h * V, W)})
        par = ("latent_attention", params)
    else:
        E, ff, sff = case["experts"], case["ff"], case["shared_ff"]
        params = dict(hidden_size=W, experts=E, top=case["top"], ff=ff, shared_ff=sff)
        w = {"router": rnd.mat(E, W)}
        gated = case["form"] != "on_input"
        for e in range(E):
            if gated:
                w[f"e{e}.gate"] = rnd.mat(ff, W)
            w.update({f"e{e}.up": rnd.mat(ff, W), f"e{e}.down": rnd.mat(W, ff)})
        if gated:
            w["shared.gate"] = rnd.mat(sff, W)
            params.update(limit=7.0, shared_limit=7.0)
        w.update({"shared.up": rnd.mat(sff, W), "shared.down": rnd.mat(W, sff)})
        if case["form"] == "chosen":
            params.update(score="chosen_softmax", renormalize=False, router_bias="router.b")
            w["router.b"] = rnd.vec(E, std=0.1)
        elif case["form"] == "groups":
            params.update(groups=4, keep=2)
        else:
            params.update(score="sigmoid", renormalize=False, activation="relu2", weight_on_input=True, shared_gate=True)
            w["shared.sg"] = rnd.mat(1, W)
        par = ("grouped_experts", params)
        return par[0], par[1], None, w, [rnd.vec(case["tokens"], W).to(dtype)]
    xs = [rnd.vec(sum(new for _, new in step), W).to(dtype) for step in _part_steps(case)]
    return par[0], par[1], pos, w, xs


def _constant_decays(h):
    return [1.0 - 2.0 ** -(3 + 5 * i / max(1, h - 1)) for i in range(h)]


def _part_steps(case):
    """Per step the requests' (tokens already taken in, new tokens)."""
    if case["kind"] == "experts":
        return [[(0, case["tokens"])]]
    lens = _lens(case["seqs"], case["tokens"], case["ragged"])
    steps = [[(0, n) for n in lens]]
    if case.get("tail"):
        steps.append([(n, case["tail"]) for n in lens])
    return steps


# ------------------------------------------------------------------------------------------------ the calls
def prepare(case, seed):
    return _prepare_model(case, seed) if case["kind"] in ("decode", "step") else _prepare_part(case, seed)


def _prepare_model(case, seed):
    from firefly_b200.engine.engine import Engine, EngineOptions
    from firefly_b200.engine.loading import parse_dtype, require_cuda
    from firefly_b200.engine.runner import StepEntry
    from firefly_b200.models import config_from_dict, spec_for
    from firefly_b200.models.decoder import DecoderModel
    from firefly_b200.ops import kernels as K
    from firefly_b200.parts import Runtime
    w, ids = _qwen_inputs(case, seed)
    cfg = config_from_dict(_qwen_config(case))
    K.set_exact_matmul()
    model = DecoderModel(spec_for(cfg), Runtime(require_cuda("cuda:0"), parse_dtype("bfloat16")))
    model.bind(w)
    reqs = _requests(case)
    n = len(reqs)
    batch = case.get("batch", 1)
    eng = Engine(model, cfg, options=EngineOptions(
        num_kv_blocks=sum(-(-(old + new) // 16) + 1 for old, new in reqs), max_batch_size_limit=max(n, 1), max_num_batched_tokens=8192,
        max_model_len=8192, eos_token_ids=[], graph_batch_sizes=(next(b for b in (1, 2, 4, 8, 16, 32, 64) if b >= min(batch, 64)),)))
    entries, starts = [], []
    room, part = 8192, []

    def feed():
        if part:
            eng.runner.step(part)
            part.clear()
    for i, ((old, new), toks) in enumerate(zip(reqs, ids)):
        rc = eng.cache.admit(f"r{i}")
        assert eng.cache.grow(rc, old + new)
        if old:
            if old > room:
                feed()
                room = 8192
            part.append(StepEntry(rc, toks[:old], []))
            room -= old
        entries.append(StepEntry(rc, toks[old:], _wanted(new)))
        starts.append(old)
    feed()
    eng.runner.check_status()
    return SimpleNamespace(kind=case["kind"], engine=eng, entries=entries, starts=starts)


def _wanted(new):
    """Places of a portion whose logits are asked for: the last, and up to fifteen before it spread over the portion."""
    return sorted({new - 1 - i * new // 16 for i in range(min(16, new))})


def _prepare_part(case, seed):
    from firefly_b200.cache.manager import CacheManager
    from firefly_b200.config.base import PartSpec
    from firefly_b200.engine.runner import ModelRunner, StepEntry
    from firefly_b200.ops import kernels as K
    from firefly_b200.parts import Runtime, build_part
    kind, params, pos, w, xs = _part_inputs(case, seed)
    K.set_exact_matmul()
    rt = Runtime(torch.device("cuda:0"), DTYPES[case.get("dtype", "bfloat16")])
    extra = {"position": build_part("position", PartSpec("rotary", pos), rt)} if pos else {}
    routed = case["kind"] == "experts"
    part = build_part("feed_forward" if routed else "mixer", PartSpec(kind, params, prefix=""), rt, **extra)
    part.bind(w)
    steps = _part_steps(case)
    n, total = len(steps[0]), [sum(s[i][1] for s in steps) for i in range(len(steps[0]))]
    cache = CacheManager({} if routed else {0: part.cache_spec()}, block_size=16, num_blocks=sum(-(-t // 16) + 1 for t in total), max_requests=n)
    cache.allocate_storage(rt.dtype, rt.device)
    runner = ModelRunner(SimpleNamespace(rt=rt, spec=SimpleNamespace(vocab_size=2)), cache, max_model_len=max(total) + 16,
                         max_batched_tokens=max(x.shape[0] for x in xs), max_seqs=n)
    rcs = [cache.admit(i) for i in range(n)]
    for rc, t in zip(rcs, total):
        assert cache.grow(rc, t)
    contexts = []
    for step in steps:
        size = 16 * (sum(new for _, new in step) + 64 * n) + 64 * n * (max(total) // 16 + 8)
        host, dev = torch.zeros(size, dtype=torch.int32).pin_memory(), torch.zeros(size, dtype=torch.int32, device=DEV)
        contexts.append(runner.build_context([StepEntry(rc, [0] * new, []) for rc, (_, new) in zip(rcs, step)], meta_host=host, meta_dev=dev))
        for rc, (_, new) in zip(rcs, step):
            cache.advance(rc, new)
    return SimpleNamespace(kind=case["kind"], part=part, contexts=contexts, xs=xs, keep=(cache, runner))


def run(state):
    if state.kind in ("decode", "step"):
        for e, start in zip(state.entries, state.starts):     # the same step again: its tokens are taken back first
            e.cache.num_tokens = start
        if state.kind == "decode":
            logits, _ = state.engine.graphs.run(state.entries)    # the tokens are read too, as the engine's loop does
            return {"logits": logits}
        return {"logits": state.engine.runner.step(state.entries)}
    if state.kind == "experts":
        return {"out0": state.part.forward(state.xs[0], state.contexts[0])}
    if len(state.xs) == 1:
        return {"out0": state.part.forward(state.xs[0], state.contexts[0], 0, True)}
    # the layer's own output buffer serves both steps: the first step's rows are kept, as a model keeps them in its stream
    first = state.part.forward(state.xs[0], state.contexts[0], 0, True).clone()
    return {"out0": first, "out1": state.part.forward(state.xs[1], state.contexts[1], 0, True)}


# ------------------------------------------------------------------------------------------------ what a call cannot do without
def work(case):
    kind = case["kind"]
    if kind in ("decode", "step"):
        s, L, V = SHAPES[case["shape"]], case["layers"], case["vocab"]
        H, I, nq, nkv = s["hidden"], s["inter"], s["heads"] * 128, s["kv_heads"] * 128
        reqs = _requests(case)
        T = sum(new for _, new in reqs)
        rows = sum(len(_wanted(new)) for _, new in reqs)
        layer = H * (nq + 2 * nkv) + nq * H + 3 * H * I
        pairs = sum(new * old + new * (new + 1) // 2 for old, new in reqs)
        return {"bytes": 2 * (L * layer + V * H) + 2 * L * 2 * nkv * sum(old + new for old, new in reqs) + T * H * 2 + rows * V * 4,
                "flops": 2 * T * L * layer + 2 * rows * V * H + 4 * L * nq * pairs}
    W = case["hidden"]
    es = 4 if case.get("dtype") == "float32" else 2
    if kind == "experts":
        E, top, T, ff, sff = case["experts"], case["top"], case["tokens"], case["ff"], case["shared_ff"]
        mats = 2 if case["form"] == "on_input" else 3
        return {"bytes": es * (E * mats * ff * W + mats * sff * W + E * W + T * W) + 4 * T * W,
                "flops": 2 * T * W * (top * mats * ff + mats * sff + E)}
    T = sum(new for step in _part_steps(case) for _, new in step)
    n = case["seqs"]
    if kind == "attention":
        nq, nkv = case["heads"] * 128, case["kv_heads"] * 128
        pairs = sum(_pairs(new, case["window"]) for _, new in _part_steps(case)[0])
        mats = W * (2 * nq + 2 * nkv)
        return {"bytes": es * (mats + 2 * T * W + 2 * T * nkv), "flops": 2 * T * mats + 4 * nq * pairs}
    if kind == "latent":
        h, q, D = case["heads"], case["q_rank"], 128 if case["q_rank"] else 64
        mats = (W * q + q * h * (D + 64) if q else W * h * (D + 64)) + W * 256 + 2 * h * D * 192 + W * (h if q else h * D) + h * D * W
        pairs = sum(_pairs(new, case["window"]) for _, new in _part_steps(case)[0])
        return {"bytes": es * (mats + 2 * T * W + T * 256), "flops": 2 * T * mats + 2 * h * (2 * D + 64) * pairs}
    # the recurrences: the products, and per token and head four operations an element of the state
    if kind == "wkv":
        hd, N, V = case["heads"] * 64, 64, 64
        mats, h, state = 5 * W * hd + case["rank"] * (W + hd), case["heads"], case["heads"] * N * V
    elif kind == "state_space":
        inner, N, V = 2 * W, case["state"], 64
        h = inner // V
        mats, state = W * (2 * inner + 2 * case["groups"] * N + h) + W * inner, h * N * V
    elif kind == "delta":
        h, N, V = case["heads"], 128, 128
        low = W * (h + h * V) if case["decay"] == "head" else 128 * W + 64 * (h * N + h * V)
        mats, state = W * (2 * case["kv_heads"] * N + 2 * h * V + h) + low, h * N * V
    else:
        h, N, V = case["heads"], case["dim"], 128
        mats, state = W * (2 * h * N + 3 * h * V) + (16 * (W + h * N) if case["decay"] == "channel" else 0), h * N * V
    return {"bytes": es * (mats + 2 * T * W) + 2 * 4 * n * state, "flops": 2 * T * mats + (6 if kind == "delta" else 4) * T * state}


def _pairs(n, window):
    full = n * (n + 1) // 2
    return full if not window or n <= window else window * (window + 1) // 2 + (n - window) * window


def tolerance(case):
    if case.get("dtype") == "float32":
        return {"rel": 2e-5, "max": 2e-3}
    if case["kind"] in ("decode", "step"):
        return {"rel": 2.5e-2, "max": 0.25}      # either side of two correct ones is up to 1.3e-2 off the 64-bit logits
    return {"rel": 1e-2, "max": 0.25}            # one layer: up to 0.53e-2 off


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, w=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w


def _rope(x, positions, theta, interleaved=False):
    """x [n, heads, r], all of r turned."""
    r = x.shape[-1]
    ang = positions.to(F64)[:, None] * torch.pow(torch.tensor(theta, dtype=F64, device=x.device), -2.0 * torch.arange(r // 2, dtype=F64, device=x.device) / r)
    c, s = torch.cos(ang)[:, None, :], torch.sin(ang)[:, None, :]
    if interleaved:
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)
    a, b = x[..., : r // 2], x[..., r // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _attend(q, k, v, scale, rows, window=0):
    """q [m, h, d] at positions `rows`, k [n, g, d], v [n, g, e] -> [m, h, e]."""
    m, h, _ = q.shape
    n, g, e = v.shape
    out = torch.empty(m, h, e, dtype=F64, device=q.device)
    pos = torch.arange(n, device=q.device)
    for i in range(g):
        kk, vv = k[:, i], v[:, i]
        for j in range(i * (h // g), (i + 1) * (h // g)):
            for lo in range(0, m, 4096):
                hi = min(m, lo + 4096)
                s = q[lo:hi, j] @ kk.T * scale
                gap = rows[lo:hi, None] - pos[None]
                s.masked_fill_((gap < 0) | ((gap >= window) if window else (gap < 0)), -math.inf)
                out[lo:hi, j] = torch.softmax(s, -1) @ vv
    return out


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] in ("decode", "step"):
            return _exact_model(case, seed)
        _, _, _, w, xs = _part_inputs(case, seed)
        w = {k: t.to(F64) for k, t in w.items()}
        if case["kind"] == "experts":
            return {"out0": _exact_experts(case, w, xs[0].to(F64))}
        # one long sequence a request, cut again afterwards
        steps = _part_steps(case)
        seqs = [[] for _ in steps[0]]
        for step, x in zip(steps, xs):
            for i, piece in enumerate(torch.split(x.to(F64), [new for _, new in step])):
                seqs[i].append(piece)
        seqs = [torch.cat(s) for s in seqs]
        one = {"attention": _exact_attention, "latent": _exact_latent}.get(case["kind"])
        outs = [one(case, w, s) for s in seqs] if one else _exact_recurrent(case, w, seqs)
        return {f"out{k}": torch.cat([o[old: old + new] for o, (old, new) in zip(outs, step)]) for k, step in enumerate(steps)}


def _exact_model(case, seed):
    w, ids = _qwen_inputs(case, seed)
    s, reqs = SHAPES[case["shape"]], _requests(case)
    nq, nkv, L = s["heads"], s["kv_heads"], case["layers"]
    embed = w["model.embed_tokens.weight"]
    hs = [embed[torch.tensor(t, device=DEV)].to(F64) for t in ids]
    wanted = [torch.tensor([old + p for p in _wanted(new)], device=DEV) for old, new in reqs]
    for i in range(L):
        g = {k: t.to(F64) for k, t in w.items() if k.startswith(f"model.layers.{i}.")}
        p = f"model.layers.{i}."
        for j, h in enumerate(hs):
            n = h.shape[0]
            every = torch.arange(n, device=DEV)
            rows = every if i + 1 < L else wanted[j]       # the last layer's other rows are not read
            x = _rms(h, g[p + "input_layernorm.weight"])
            k = _rope(_rms((x @ g[p + "self_attn.k_proj.weight"].T).view(n, nkv, 128), g[p + "self_attn.k_norm.weight"]), every, THETA)
            v = (x @ g[p + "self_attn.v_proj.weight"].T).view(n, nkv, 128)
            q = _rope(_rms((x[rows] @ g[p + "self_attn.q_proj.weight"].T).view(-1, nq, 128), g[p + "self_attn.q_norm.weight"]), rows, THETA)
            a = _attend(q, k, v, 128 ** -0.5, rows).flatten(1)
            h = h[rows] + a @ g[p + "self_attn.o_proj.weight"].T
            x = _rms(h, g[p + "post_attention_layernorm.weight"])
            hs[j] = h + (F.silu(x @ g[p + "mlp.gate_proj.weight"].T) * (x @ g[p + "mlp.up_proj.weight"].T)) @ g[p + "mlp.down_proj.weight"].T
        del g
    x = _rms(torch.cat(hs), w["model.norm.weight"].to(F64))
    logits = x @ (embed if s["tied"] else w["lm_head.weight"]).to(F64).T
    return {"logits": logits}


def _exact_attention(case, w, x):
    n, nq, nkv = x.shape[0], case["heads"], case["kv_heads"]
    pos = torch.arange(n, device=x.device)
    q = _rope(_rms((x @ w["q_proj.weight"].T).view(n, nq, 128), w["q_norm.weight"]), pos, THETA)
    k = _rope(_rms((x @ w["k_proj.weight"].T).view(n, nkv, 128), w["k_norm.weight"]), pos, THETA)
    v = (x @ w["v_proj.weight"].T).view(n, nkv, 128)
    return _attend(q, k, v, 128 ** -0.5, pos, case["window"]).flatten(1) @ w["o_proj.weight"].T


def _exact_latent(case, w, x):
    n, h = x.shape[0], case["heads"]
    inter = bool(case["q_rank"])
    D = V = 128 if inter else 64
    pos = torch.arange(n, device=x.device)
    q = (_rms(x @ w["dq"].T, w["dq.norm"]) @ w["uq"].T if inter else x @ w["q"].T).view(n, h, D + 64)
    q = torch.cat([q[..., :D], _rope(q[..., D:], pos, 1e4, inter)], -1)
    d = x @ w["dkv"].T
    c = _rms(d[:, :192], w["dkv.norm"])
    rot = _rope(d[:, None, 192:], pos, 1e4, inter)
    k = torch.cat([(c @ w["uk"].T).view(n, h, D), rot.expand(n, h, 64)], -1)
    o = _attend(q, k, (c @ w["uv"].T).view(n, h, V), (D + 64) ** -0.5, pos, case["window"])
    gate = torch.sigmoid(x @ w["g"].T)
    o = o * gate[:, :, None] if inter else o * gate.view(n, h, V)
    return o.flatten(1) @ w["o"].T


def _conv(x, w):
    """Causal convolution per channel: x [n, C], w [C, taps], the last tap the current token's."""
    taps = w.shape[1]
    return F.conv1d(F.pad(x.T[None], (taps - 1, 0)), w[:, None], groups=w.shape[0])[0].T


def _padded(rows):
    """Sequences' rows [n_i, ...] side by side: [longest, sequences, ...]."""
    return torch.nn.utils.rnn.pad_sequence(rows)


def _exact_recurrent(case, w, seqs):
    """The recurrence token by token, all sequences and heads at once; the rest per sequence."""
    kind = case["kind"]
    parts = [_recurrent_inputs(case, w, x) for x in seqs]      # dicts of [n, heads, ...] rows
    col = {k: _padded([p[k] for p in parts]) for k in ("q", "k", "v", "decay", "beta") if k in parts[0]}
    n, B, h, N = col["k"].shape
    S = torch.zeros(B, h, N, col["v"].shape[-1], dtype=F64, device=DEV)
    o = torch.empty(n, B, h, col["v"].shape[-1], dtype=F64, device=DEV)
    for t in range(n):
        k, v, q = col["k"][t], col["v"][t], col["q"][t]
        if kind == "wkv":
            write = k[..., None] * v[..., None, :]
            o[t] = torch.einsum("bhn,bhnv->bhv", q, S + w["u"][None, :, :, None] * write)
            S = S * col["decay"][t][..., None] + write
            continue
        S = S * col["decay"][t][..., None]
        if kind == "delta":
            v = col["beta"][t][..., None] * (v - torch.einsum("bhn,bhnv->bhv", k, S))
        S = S + k[..., None] * v[..., None, :]
        o[t] = torch.einsum("bhn,bhnv->bhv", q, S)
    return [_recurrent_output(case, w, p, o[: x.shape[0], i]) for i, (p, x) in enumerate(zip(parts, seqs))]


def _recurrent_inputs(case, w, x):
    kind, n = case["kind"], x.shape[0]
    if kind == "wkv":
        h = case["heads"]
        before = F.pad(x, (0, 0, 1, 0))[:n]
        mix = {s: x + (before - x) * w[f"mu.{s}"] for s in "rkvgw"}
        z = torch.tanh(mix["w"] @ w["w1"].T) @ w["w2"].T + w["w0"]
        return {"q": (mix["r"] @ w["r"].T).view(n, h, 64), "k": (mix["k"] @ w["k"].T).view(n, h, 64), "v": (mix["v"] @ w["v"].T).view(n, h, 64),
                "decay": torch.exp(-torch.exp(z)).view(n, h, 64), "gate": F.silu(mix["g"] @ w["g"].T)}
    if kind == "state_space":
        inner, N, G = 2 * case["hidden"], case["state"], case["groups"]
        h = inner // 64
        z, xbc, step = torch.split(x @ w["in"].T, [inner, inner + 2 * G * N, h], -1)
        xbc = F.silu(_conv(xbc, w["conv"]) + w["conv.b"])
        v, b, c = torch.split(xbc, [inner, G * N, G * N], -1)
        step = F.softplus(step + w["dt_bias"], threshold=1e9)
        wide = lambda t: t.view(n, G, N).repeat_interleave(h // G, 1)  # noqa: E731
        return {"q": wide(c), "k": wide(b) * step[..., None], "v": v.view(n, h, 64),
                "decay": torch.exp(-torch.exp(w["A_log"]) * step)[..., None].expand(n, h, N), "z": z}
    h = case["heads"]
    if kind == "delta":
        g, head = case["kv_heads"], case["decay"] == "head"
        q, k, v = (F.silu(_conv(x @ w[s].T, w[s + ".conv"])) for s in "qkv")
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        a = x @ w["a"].T if head else (x @ w["a1"].T) @ w["a2"].T
        a = F.softplus(a + w["dt_bias"], threshold=1e9).view(n, h, -1).expand(n, h, 128)
        wide = lambda t: unit(t.view(n, g, 128)).repeat_interleave(h // g, 1)  # noqa: E731
        gate = x @ w["g"].T if head else (x @ w["g1"].T) @ w["g2"].T
        return {"q": wide(q) * 128 ** -0.5, "k": wide(k), "v": v.view(n, h, 128), "decay": torch.exp(-torch.exp(w["A_log"])[None, :, None] * a),
                "beta": torch.sigmoid(x @ w["b"].T), "gate": F.silu(gate) if head else torch.sigmoid(gate)}
    D = case["dim"]
    q, k, v, gate = (x @ w[s].T for s in "qkvg")
    if case["decay"] == "constant":
        decay = torch.tensor(_constant_decays(h), dtype=F32, device=x.device).to(F64)[None, :, None].expand(n, h, D)
        return {"q": F.silu(q).view(n, h, D), "k": F.silu(k).view(n, h, D), "v": F.silu(v).view(n, h, 128), "decay": decay, "gate": torch.sigmoid(gate)}
    alpha = torch.exp(-F.softplus(-((x @ w["a1"].T) @ w["a2"].T + w["a2.b"]), threshold=1e9) / 16.0)
    return {"q": q.view(n, h, D) * D ** -0.5, "k": k.view(n, h, D), "v": v.view(n, h, 128), "decay": alpha.view(n, h, D), "gate": F.silu(gate)}


def _recurrent_output(case, w, p, o):
    n, kind = o.shape[0], case["kind"]
    if kind == "wkv":
        y = _rms(o).flatten(1) * w["norm"] * p["gate"]
    elif kind == "state_space":
        o = o + w["D"][None, :, None] * p["v"]
        y = (o.flatten(1) * F.silu(p["z"])).view(n, case["groups"], -1)
        y = _rms(y).flatten(1) * w["norm"]
    elif kind == "linear" and case["decay"] == "constant":
        y = _rms(o.flatten(1)) * w["norm"] * p["gate"]
    else:
        y = (_rms(o) * w["norm"]).flatten(1) * p["gate"]
    return y @ w["o"].T


def _exact_experts(case, w, x):
    E, top = case["experts"], case["top"]
    z = x @ w["router"].T
    if case["form"] == "chosen":
        z = z + w["router.b"]
        best, ids = z.topk(top, -1)
        wts = torch.softmax(best, -1)
    elif case["form"] == "groups":
        s = torch.softmax(z, -1)
        score = s.view(-1, 4, E // 4).amax(-1)
        open_ = torch.zeros_like(score).scatter_(1, score.topk(2, -1).indices, 1.0).repeat_interleave(E // 4, 1)
        best, ids = torch.where(open_ > 0, s, -1.0).topk(top, -1)
        wts = best / (best.sum(-1, keepdim=True) + 1e-20)
    else:
        best, ids = torch.sigmoid(z).topk(top, -1)
        wts = best

    def expert(prefix, rows):
        if case["form"] == "on_input":
            return F.relu(rows @ w[prefix + ".up"].T).square() @ w[prefix + ".down"].T
        g, u = (rows @ w[prefix + ".gate"].T).clamp(max=7.0), (rows @ w[prefix + ".up"].T).clamp(-7.0, 7.0)
        return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w[prefix + ".down"].T
    out = expert("shared", x)
    if case["form"] == "on_input":
        out = out * torch.sigmoid(x @ w["shared.sg"].T)
    for e in range(E):
        tok, place = (ids == e).nonzero(as_tuple=True)
        wt = wts[tok, place][:, None]
        out.index_add_(0, tok, expert(f"e{e}", x[tok] * wt) if case["form"] == "on_input" else expert(f"e{e}", x[tok]) * wt)
    return out
