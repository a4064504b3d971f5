"""The recurrences a chunk of tokens at a time (csrc/ssm.cu, csrc/wkv.cu, csrc/delta_rule.cu over csrc/chunk_scan.cuh) against
the same recurrence token by token in 64 bits: lengths around the chunk sizes of 16 and 32, key sizes of 64 and 128, value
sizes that fill no block of columns, decays from none to all, and numbers that are not finite.

Tolerance of the outputs' norm: 2^-24 (32 + L) for sequences of up to L tokens.  Every number and sum is 32-bit; a decay is rounded
once, and what a state keeps of a token passed at most L of them, each off by 2^-24 at most; the sums over key channels and
tokens, of terms of random sign, stay below 32 roundings."""
import math
from types import SimpleNamespace

import pytest
import torch
import torch.nn.functional as F

from firefly_b200.engine.context import Workspace
from firefly_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
# ends around chunks of 16 and 32; around the shortest length that goes by chunks, 24 to 64; all of them by chunks
LENS = [(15, 16, 17, 400), (31, 32, 33, 330), (1, 260), (112, 128, 144), (23, 24, 25, 47, 48, 49, 63, 64, 65)]


def _ctx(lens, fresh):
    n = len(lens)
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    return SimpleNamespace(cu_q=cu, num_seqs=n, q_lens=list(lens), state_slots=torch.arange(n, 0, -1, dtype=torch.int32, device="cuda"),
                           seq_fresh=torch.full((n,), fresh, dtype=torch.int32, device="cuda"), workspace=Workspace("cuda"))


def _walk(q, k, v, decay, beta=None, bonus=None, S=None):
    """One sequence in 64 bits: q, k, decay [T, h, N], v [T, h, V]."""
    q, k, v, decay = (x.double() for x in (q, k, v, decay))
    T, h, N = q.shape
    S = torch.zeros(h, N, v.shape[-1], dtype=torch.float64, device=q.device) if S is None else S
    o = torch.empty_like(v)
    for t in range(T):
        if bonus is not None:
            w = k[t][:, :, None] * v[t][:, None]
            o[t] = torch.einsum("hn,hnv->hv", q[t], S + bonus.double()[:, :, None] * w)
            S = S * decay[t][:, :, None] + w
            continue
        S = S * decay[t][:, :, None]
        u = v[t] if beta is None else beta[t].double()[:, None] * (v[t] - torch.einsum("hn,hnv->hv", k[t], S))
        S = S + k[t][:, :, None] * u[:, None]
        o[t] = torch.einsum("hn,hnv->hv", q[t], S)
    return o, S


def _check(call, inputs, lens, heads, V, T, chunk_min, bonus=None):
    """A step of prompts on fresh slots, then one of single tokens behind them, against `_walk`."""
    n, tol = len(lens), 2.0 ** -24 * (32 + max(lens))
    o, o1 = torch.empty(T, heads * V, device="cuda"), torch.empty(n, heads * V, device="cuda")
    before = K.LAUNCHES
    call(0, T, _ctx(lens, 1), o)
    assert K.LAUNCHES - before == 2 * (max(lens) >= chunk_min) + (min(lens) < chunk_min)      # two kernels for chunks, one that walks
    call(T, T + n, _ctx([1] * n, 0), o1)                   # token by token, from the state that the chunks left
    at = 0
    for i, L in enumerate(lens):
        want, S = _walk(*inputs(at, at + L), bonus=bonus)
        assert (o[at:at + L].view_as(want).double() - want).norm() <= tol * want.norm()
        want, _ = _walk(*inputs(T + i, T + i + 1), bonus=bonus, S=S)
        assert (o1[i].view_as(want).double() - want).norm() <= tol * want.norm()
        at += L


def _rand(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return lambda *s: torch.randn(*s, generator=g, device="cuda")


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("N,V,heads,groups,mode", [(64, 64, 4, 1, "step"), (128, 40, 6, 3, "step"), (128, 128, 2, 2, "constant"),
                                                   (64, 72, 3, 3, "channel"), (128, 8, 2, 2, "channel"),
                                                   # a group's heads in three blocks, the last of them half empty; in two, as many groups fill the GPU
                                                   (64, 8, 10, 1, "step"), (64, 8, 400, 40, "step")])
def test_decay_scans(lens, N, V, heads, groups, mode):
    rn = _rand(N + V)
    T, n = sum(lens), len(lens)
    x = rn(T + n, heads * V + 2 * groups * N).to(BF)
    raw = rn(T + n, heads).to(BF)
    bias, a_log, skip = rn(heads) - 2, rn(heads) + 1, rn(heads)
    const = torch.tensor([-0.5, 0.999], device="cuda")
    # per channel: from keeping everything to forgetting everything at once
    alpha = torch.sigmoid(6 * rn(T + n, heads * N)) ** 2
    alpha[:, 0], alpha[:, 1] = 0.0, 1.0
    state = torch.full((n + 1, K.scan_state_floats(heads, N, V)), 7.0, device="cuda")
    kw = {"step": lambda a, b: dict(step=(raw[a:b], 0), step_bias=bias, a_log=a_log, skip=skip), "constant": lambda a, b: dict(decay=const),
          "channel": lambda a, b: dict(channel_decay=(alpha[a:b], 0), q_scale=0.125)}[mode]

    def values(a, b):
        return x[a:b, : heads * V].double().view(b - a, heads, V)

    def call(a, b, ctx, o):
        K.scalar_decay_scan((x[a:b], heads * V), (x[a:b], heads * V + groups * N), (x[a:b], 0), state, 0, ctx, o, heads, N, V,
                            heads_per_group=heads // groups, **kw(a, b))
        if mode == "step":                                 # the skip term is taken off again
            o.copy_((o.double() - (skip.double()[None, :, None] * values(a, b)).view(b - a, -1)).float())

    def inputs(a, b):
        xx, v = x[a:b].double(), values(a, b)
        q, k = (xx[:, heads * V + i * groups * N:][:, : groups * N].view(b - a, groups, N).repeat_interleave(heads // groups, 1) for i in (0, 1))
        if mode == "step":
            s = F.softplus(raw[a:b].double() + bias.double(), threshold=1e9)
            return q, k * s[:, :, None], v, torch.exp(-torch.exp(a_log.double()) * s)[:, :, None].expand_as(k)
        if mode == "constant":
            return q, k, v, const.double()[None, :, None].expand_as(k)
        return q * 0.125, k, v, alpha[a:b].view(b - a, heads, N)
    _check(call, inputs, lens, heads, V, T, 1 << 30 if mode == "constant" else K._lib("ssm").ff_scan_chunk_min(2 if mode == "channel" else 1))


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("dim,heads", [(64, 3), (128, 2)])
def test_wkv_scan(lens, dim, heads):
    rn = _rand(dim)
    T, n, hd = sum(lens), len(lens), heads * dim
    rkvg, rkvg1 = rn(4, T, hd).to(BF), rn(4, n, hd).to(BF)
    dlog, w0, u = rn(T + n, hd), 2.5 * rn(hd) - 2, rn(hd)
    x = rn(T + n, 48).to(BF)
    state = torch.full((n + 1, heads * dim * dim + 48), 7.0, device="cuda")

    def call(a, b, ctx, o):
        K.wkv_scan(rkvg if a == 0 else rkvg1, dlog[a:b].contiguous(), w0, u, state, heads * dim * dim, x[a:b].contiguous(), ctx, o, heads, dim)
        assert torch.equal(state[ctx.state_slots.long(), heads * dim * dim:], x[a:b][ctx.cu_q[1:].long() - 1].float())

    def inputs(a, b):
        r = (rkvg[:, a:b] if a < T else rkvg1[:, a - T:b - T]).reshape(4, b - a, heads, dim)
        return r[0], r[1], r[2], torch.exp(-torch.exp(dlog[a:b].double() + w0.double())).view(b - a, heads, dim)
    _check(call, inputs, lens, heads, dim, T, K._lib("wkv").ff_wkv_chunk_min(), bonus=u.view(heads, dim))


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("N,V,heads,per_group,per_head", [(64, 40, 4, 2, False), (128, 128, 2, 1, False), (128, 72, 2, 2, True)])
def test_delta_rule_scan(lens, N, V, heads, per_group, per_head):
    rn = _rand(N + V + per_head)
    T, n, G = sum(lens), len(lens), heads // per_group
    x, beta = rn(T + n, 2 * G * N + heads * V).to(BF), (2 * rn(T + n, heads)).to(BF)
    wide = heads if per_head else heads * N
    a_raw, bias, a_log = 3 * rn(T + n, wide), rn(wide) - 1, rn(heads)
    state = torch.full((n + 1, K.delta_state_floats_plan(heads, N, V)), 7.0, device="cuda")
    assert K.delta_state_floats(heads, N, V) == K.delta_state_floats_plan(heads, N, V)

    def call(a, b, ctx, o):
        xs, bs, rs = x[a:b], beta[a:b], a_raw[a:b]
        K.delta_rule_scan((xs, 0), (xs, G * N), (xs, 2 * G * N), (bs, 0), (rs, 0), bias, a_log, state, 0, ctx, o, heads, N, V,
                          heads_per_group=per_group, q_scale=N ** -0.5, unit_eps=1e-6, decay_per_head=per_head)

    def inputs(a, b):
        xx = x[a:b].double()
        q, k = (xx[:, i * G * N:][:, : G * N].view(b - a, G, N).repeat_interleave(per_group, 1) for i in (0, 1))
        q, k = (y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6) for y in (q, k))
        s = F.softplus(a_raw[a:b].double() + bias.double(), threshold=1e9).view(b - a, heads, -1).expand(b - a, heads, N)
        return (q * N ** -0.5, k, xx[:, 2 * G * N:].view(b - a, heads, V), torch.exp(-torch.exp(a_log.double())[None, :, None] * s),
                torch.sigmoid(beta[a:b].double()))
    _check(call, inputs, lens, heads, V, T, K._lib("delta_rule").ff_delta_chunk_min())


@pytest.mark.parametrize("bad", [math.nan, math.inf])
@pytest.mark.parametrize("kind", ["step", "channel", "wkv", "delta"])
def test_not_finite_values_stay_behind_their_token(kind, bad):
    """A value that is not finite spoils its own column from its token on, as token by token, and nothing in front of it."""
    rn = _rand(3)
    T, N, V, at, col = 100, 64, 64, 37, 21
    x = rn(T, 2 * N + V).to(BF)
    x[at, 2 * N + col] = bad
    zeros = lambda *s: torch.zeros(*s, device="cuda")  # noqa: E731
    out = []
    for workspace in (Workspace("cuda"), None):
        ctx = _ctx([T], 1)
        ctx.workspace = workspace
        o, state = zeros(T, V), zeros(2, N * V + 8)
        q, k, v = (x, 0), (x, N), (x, 2 * N)
        if kind == "step":
            K.scalar_decay_scan(q, k, v, state, 0, ctx, o, 1, N, V, step=(x, 0), step_bias=zeros(1), a_log=zeros(1))
        elif kind == "channel":
            K.scalar_decay_scan(q, k, v, state, 0, ctx, o, 1, N, V, channel_decay=(zeros(T, N) + 0.9, 0))
        elif kind == "wkv":
            rkvg = torch.stack([x[:, :N], x[:, N:2 * N], x[:, 2 * N:], x[:, :N]]).contiguous()
            K.wkv_scan(rkvg, zeros(T, N), zeros(N), zeros(N) + 1, state, N * V, x[:, :8].contiguous(), ctx, o, 1, N)
        else:
            K.delta_rule_scan(q, k, v, (x, 0), (zeros(T, N), 0), zeros(N), zeros(1), state, 0, ctx, o, 1, N, V)
        out.append(o)
    chunked, walked = out
    spoilt = ~torch.isfinite(walked)
    assert torch.equal(~torch.isfinite(chunked), spoilt)
    assert spoilt[at:, col].all() and not spoilt[:at].any() and not spoilt[:, :col].any()
    assert (chunked[~spoilt] - walked[~spoilt]).norm() <= 2.0 ** -23 * (32 + T) * walked[~spoilt].norm()


# what of a token's inputs is spoilt, for every kind of recurrence; "step" is whatever its decay is made of
INPUTS = [(kind, part) for kind in ("step", "channel", "wkv", "delta") for part in ("q", "k", "v", "step", "beta")
          if kind == "delta" or part != "beta"]


@pytest.mark.parametrize("bad", [math.nan, math.inf, 3e38])
@pytest.mark.parametrize("at", [37, 40, 95])
@pytest.mark.parametrize("kind,part", INPUTS)
def test_spoilt_inputs_stay_behind_their_token(kind, part, at, bad):
    """A number of any input that is not finite, or so large that sums behind it overflow, leaves the tokens in front of it as the
    walk token by token does; behind one that is not finite, what the walk leaves finite is finite here (sums next to the
    largest 32-bit number may overflow in one order and not in another)."""
    rn = _rand(5)
    T, N, V = 100, 64, 64
    x, beta, decay = rn(T, 2 * N + V).to(BF), rn(T, 1).to(BF), 0.8 + 0.1 * torch.rand(T, N, device="cuda")
    raw = (beta if kind == "step" else rn(T, N)).clone()
    if kind == "channel":
        raw = decay
    if part in "qkv":
        x[at, {"q": 0, "k": N, "v": 2 * N}[part] + 21] = bad
    else:
        (beta if part == "beta" else raw)[at, 0] = bad
    zeros = lambda *s: torch.zeros(*s, device="cuda")  # noqa: E731
    out = []
    for workspace in (Workspace("cuda"), None):
        ctx = _ctx([T], 1)
        ctx.workspace = workspace
        o, state = zeros(T, V), zeros(2, N * V + 8)
        q, k, v = (x, 0), (x, N), (x, 2 * N)
        if kind == "step":
            K.scalar_decay_scan(q, k, v, state, 0, ctx, o, 1, N, V, step=(raw, 0), step_bias=zeros(1), a_log=zeros(1))
        elif kind == "channel":
            K.scalar_decay_scan(q, k, v, state, 0, ctx, o, 1, N, V, channel_decay=(raw, 0))
        elif kind == "wkv":
            rkvg = torch.stack([x[:, :N], x[:, N:2 * N], x[:, 2 * N:], x[:, :N]]).contiguous()
            K.wkv_scan(rkvg, raw, zeros(N), zeros(N) + 1, state, N * V, x[:, :8].contiguous(), ctx, o, 1, N)
        else:
            K.delta_rule_scan(q, k, v, (beta, 0), (raw, 0), zeros(N), zeros(1), state, 0, ctx, o, 1, N, V)
        out.append(o)
    chunked, walked = out
    assert torch.isfinite(walked[:at]).all() and torch.isfinite(chunked[:at]).all()
    assert (chunked[:at] - walked[:at]).norm() <= 2.0 ** -23 * (32 + T) * walked[:at].norm()
    if not math.isfinite(bad):
        assert not (torch.isfinite(walked) & ~torch.isfinite(chunked)).any()


@pytest.mark.parametrize("L", [97, 112])
def test_delta_rule_without_an_epsilon(L):
    """unit_eps = 0: the rows that fill a sequence's last chunk up are zeros, which have no unit vector."""
    rn = _rand(9)
    N = V = 64
    x, beta, raw = rn(L, 2 * N + V).to(BF), rn(L, 1).to(BF), rn(L, N)
    state, o = torch.zeros(2, N * V, device="cuda"), torch.zeros(L, V, device="cuda")
    zeros = lambda *s: torch.zeros(*s, device="cuda")  # noqa: E731
    K.delta_rule_scan((x, 0), (x, N), (x, 2 * N), (beta, 0), (raw, 0), zeros(N), zeros(1), state, 0, _ctx([L], 1), o, 1, N, V, unit_eps=0.0)
    q, k = (x[:, i:i + N].double().view(L, 1, N) for i in (0, N))
    q, k = (y / y.norm(dim=-1, keepdim=True) for y in (q, k))
    want, S = _walk(q, k, x[:, 2 * N:].double().view(L, 1, V), torch.exp(-F.softplus(raw.double())).view(L, 1, N), torch.sigmoid(beta.double()))
    tol = 2.0 ** -24 * (32 + L)
    assert (o.view_as(want).double() - want).norm() <= tol * want.norm()
    assert (state[1].view(1, V, N).transpose(1, 2).double() - S).norm() <= tol * S.norm()


def test_rows_off_a_boundary_are_walked_without_scratch_memory():
    """Rows that 16-byte copies do not take are walked token by token and counted as one kernel; no scratch memory is taken for them."""
    rn = _rand(2)
    T, N = 100, 64
    zeros = lambda *s: torch.zeros(*s, device="cuda")  # noqa: E731
    for shift, kernels in ((0, 2), (1, 1)):
        x, ctx, o = rn(T, 3 * N + 8).to(BF), _ctx([T], 1), zeros(T, N)
        q, k, v = ((x, i * N + shift) for i in range(3))
        for call in (lambda: K.scalar_decay_scan(q, k, v, zeros(2, N * N), 0, ctx, o, 1, N, N, step=(x, 0), step_bias=zeros(1), a_log=zeros(1)),
                     lambda: K.scalar_decay_scan(q, k, v, zeros(2, N * N), 0, ctx, o, 1, N, N, channel_decay=(zeros(T, N), 0)),
                     lambda: K.delta_rule_scan(q, k, v, (x, 0), (zeros(T, N), 0), zeros(N), zeros(1), zeros(2, N * N), 0, ctx, o, 1, N, N)):
            before = K.LAUNCHES
            call()
            assert K.LAUNCHES - before == kernels and (ctx.workspace.bytes() > 0) == (kernels == 2)
            ctx.workspace = Workspace("cuda")


@pytest.mark.parametrize("kind", ["step", "channel", "wkv", "delta"])
@pytest.mark.parametrize("lens", [[1] * 24 + [256, 200], [30, 20, 500, 70, 1], [64] * 40])
@pytest.mark.parametrize("known", [True, False])
def test_company_changes_nothing(kind, lens, known):
    """A sequence's outputs and state are bit for bit those of the sequence alone in a step, beside single tokens or beside prompts,
    whether the host knows the lengths or not."""
    rn = _rand(7)
    H, N, V, T = 4, 64, 64, sum(lens)
    x, beta, raw = rn(T, (2 * N + V) * H).to(BF), rn(T, H).to(BF), rn(T, H * N)
    alpha, one, many = torch.sigmoid(4 * raw), rn(H), rn(H * N)
    start = rn(len(lens) + 1, H * V * N + 8)

    def step(a, b, step_lens, state):
        ctx, o = _ctx(step_lens, 0), torch.zeros(b - a, H * V, device="cuda")
        if not known:
            del ctx.q_lens
        q, k, v = ((x[a:b], i * H * N) for i in range(3))
        if kind == "step":
            K.scalar_decay_scan(q, k, v, state, 0, ctx, o, H, N, V, step=(beta[a:b], 0), step_bias=one, a_log=one, skip=one)
        elif kind == "channel":
            K.scalar_decay_scan(q, k, v, state, 0, ctx, o, H, N, V, channel_decay=(alpha[a:b], 0))
        elif kind == "wkv":
            rkvg = torch.stack([x[a:b, i * H * N:(i + 1) * H * N] for i in (0, 1, 2, 0)]).contiguous()
            K.wkv_scan(rkvg, raw[a:b], many, many, state, H * N * N, x[a:b, :8].contiguous(), ctx, o, H, N)
        else:
            K.delta_rule_scan(q, k, v, (beta[a:b], 0), (raw[a:b], 0), many, one, state, 0, ctx, o, H, N, V)
        return o

    together = start.clone()
    o, at = step(0, T, lens, together), 0
    for i, L in enumerate(lens):
        alone = start[len(lens) - i - 1:len(lens) - i + 1].clone()       # the sequence's slot is the second of two
        assert torch.equal(step(at, at + L, [L], alone), o[at:at + L]) and torch.equal(alone[1], together[len(lens) - i])
        at += L
