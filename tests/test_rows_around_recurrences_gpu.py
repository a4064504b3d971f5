"""The element-wise kernels around the recurrences and the latent attention, and the sum of experts' rows, in their forms with vector loads and without
(csrc/ssm.cu, csrc/wkv.cu, csrc/delta_rule.cu, csrc/latent_attention.cu, csrc/moe.cu), against the formulas in 64 bits: sequences that end
around the rows a thread takes (4) and a block's tile (32 and 16), sizes that vectors divide and that they do not, rows that
start off a 16-byte boundary.

Tolerance: a result is rounded to bfloat16 once (2^-9 of it; twice that is allowed) behind a few dozen 32-bit roundings of
terms no larger than the largest value (2^-18 of that)."""
from types import SimpleNamespace

import pytest
import torch

from firefly_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
BF, F32, F64 = torch.bfloat16, torch.float32, torch.float64
LENS = [(1, 2, 3, 4, 5, 31, 32, 33), (63, 1, 64, 65, 7), (4500, 1, 130)]


def _rand(*shape, dtype=F32, seed=0):
    g = torch.Generator("cuda").manual_seed(seed + sum(shape))
    return torch.randn(*shape, generator=g, device="cuda").to(dtype)


def _close(got, want):
    assert got.dtype == BF
    err = (got.double() - want).abs()
    assert bool((err <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * want.abs().max()).all())


def _ctx(lens):
    n = len(lens)
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    seq = torch.repeat_interleave(torch.arange(n), torch.tensor(lens)).to(torch.int32).cuda()
    return SimpleNamespace(cu_q=cu, token_seq=seq, num_seqs=n, state_slots=torch.arange(n, 0, -1, dtype=torch.int32, device="cuda"),
                           seq_fresh=(torch.arange(n) % 2).to(torch.int32).cuda())


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("channels,col0,taps", [(256, 0, 4), (136, 8, 4), (70, 3, 4), (128, 0, 3), (64, 64, 2)])
def test_convolution(lens, channels, col0, taps):
    ctx, T = _ctx(lens), sum(lens)
    x, w, b = _rand(T, channels + col0 + 5, dtype=BF), _rand(channels, taps), _rand(channels)
    state = _rand(len(lens) + 1, (taps - 1) * channels)
    old, out = state.clone(), torch.empty(T, channels, dtype=BF, device="cuda")
    K.causal_conv_silu(x, col0, channels, w, b, state, 0, ctx, out)
    at = 0
    for i, n in enumerate(lens):
        slot = len(lens) - i
        front = old[slot].view(taps - 1, channels).double() * (0 if i % 2 else 1)
        rows = torch.cat([front, x[at:at + n, col0:col0 + channels].double()])
        want = b.double() + sum(w[:, j].double() * rows[j:j + n] for j in range(taps))
        _close(out[at:at + n], want * torch.sigmoid(want))
        assert torch.equal(state[slot].view(taps - 1, channels), rows[-(taps - 1):].float())
        at += n


@pytest.mark.parametrize("wide_input", [False, True])
def test_silu_of_the_convolution(wide_input):
    """Every bfloat16 number, and 65536 32-bit ones, through the filter that hands its input on (one weight of 1): SiLU rounded to
    bfloat16 once (half a unit in the last place) behind an exponential and a division of two 32-bit units each and an addition
    (2^-20 of it in all), and to 2^-119 where e^-x leaves the range of the fast division."""
    bits = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.int16).view(BF)
    x = bits.view(64, 1024)
    if wide_input:
        x = torch.cat([x.float(), torch.linspace(-120, 120, 1024 * 64, device="cuda").view(64, 1024)])
    T, C = x.shape
    w = torch.zeros(C, 4, device="cuda")
    w[:, 3] = 1
    out, ctx = torch.empty(T, C, dtype=BF, device="cuda"), _ctx([1] * T)       # a token a sequence: no row meets another's zero weight
    ctx.seq_fresh.fill_(1)
    K.causal_conv(x, 0, C, w, None, torch.zeros(T + 1, 3 * C, device="cuda"), 0, ctx, out, silu=True)
    xd, got = x.double(), out.double()
    want = xd * torch.sigmoid(xd)
    fine = torch.isfinite(xd)
    half = torch.ldexp(torch.ones_like(want), torch.frexp(want).exponent - 9)
    assert bool(((got - want).abs()[fine] <= (half + 2.0 ** -20 * want.abs())[fine] + 2.0 ** -119).all())
    assert torch.equal(got[xd == float("inf")], xd[xd == float("inf")]) and bool(got[torch.isnan(xd)].isnan().all())
    assert bool(got[xd == -float("inf")].isnan().all())        # -inf / inf, as the division gives


@pytest.mark.parametrize("width,parts,shift", [(128, 1, 0), (512, 2, 0), (1024, 1, 8), (2048, 8, 0), (4096, 1, 0), (300, 3, 0),
                                               (1024, 1, 1), (16384, 1, 0)])
@pytest.mark.parametrize("first", [True, False])
def test_gated_norm(width, parts, shift, first):
    T = 37
    o, g, w = _rand(T, width), _rand(T, width + shift + 3 * (shift % 2), dtype=BF), 1 + 0.1 * _rand(width)
    y = torch.empty(T, width, dtype=BF, device="cuda")
    K.gated_rms_norm(o, (g, shift), w, 1e-5, y, parts, first)
    gd, od = g[:, shift:shift + width].double(), o.double()
    od = od * gd * torch.sigmoid(gd) if first else od
    n = od.view(T, parts, -1)
    n = (n / (n.square().mean(-1, keepdim=True) + 1e-5).sqrt()).reshape(T, width) * w.double()
    _close(y, n if first else n * torch.sigmoid(gd))


@pytest.mark.parametrize("heads,V,shift", [(4, 64, 0), (3, 128, 8), (5, 128, 1), (2, 96, 0), (1, 64, 0)])
@pytest.mark.parametrize("act", ["sigmoid", "silu"])
@pytest.mark.parametrize("gate_type", [BF, F32])
def test_norm_of_heads(heads, V, shift, act, gate_type):
    T, W = 61, heads * V
    o, g, w = _rand(T, W), _rand(T, W + shift, dtype=gate_type), 1 + 0.1 * _rand(V)
    y = torch.empty(T, W, dtype=BF, device="cuda")
    K.head_norm_gate(o, (g, shift), w, 1e-5, y, heads, V, act)
    gd, od = g[:, shift:].double(), o.double().view(T, heads, V)
    n = (od / (od.square().mean(-1, keepdim=True) + 1e-5).sqrt() * w.double()).reshape(T, W)
    _close(y, n * torch.sigmoid(gd) * (gd if act == "silu" else 1))


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("heads,dim", [(4, 64), (3, 128), (5, 24)])
def test_mix_and_output_of_wkv(lens, heads, dim):
    ctx, T, W = _ctx(lens), sum(lens), heads * dim
    x, mu, state = _rand(T, W, dtype=BF), _rand(5, W), _rand(len(lens) + 1, W)
    mixes = torch.empty(5, T, W, dtype=BF, device="cuda")
    K.wkv_shift_mix(x, mu, state, 0, ctx, mixes)
    prev = torch.cat([x[:1].double(), x[:-1].double()])
    for i in range(len(lens)):
        prev[int(ctx.cu_q[i])] = state[len(lens) - i].double() * (0 if i % 2 else 1)
    _close(mixes, x.double() + (prev - x.double()) * mu.double()[:, None])
    o, g, w = _rand(T, W, seed=1), _rand(T, W, dtype=BF, seed=2), 1 + 0.1 * _rand(W)
    y = torch.empty(T, W, dtype=BF, device="cuda")
    K.wkv_out(o, g, w, 1e-5, y, heads, dim)
    od, gd = o.double().view(T, heads, dim), g.double()
    n = (od / (od.square().mean(-1, keepdim=True) + 1e-5).sqrt()).reshape(T, W) * w.double()
    _close(y, n * gd * torch.sigmoid(gd))


@pytest.mark.parametrize("T,heads,vdim,shift,per_head", [(33, 4, 128, 0, False), (5, 3, 64, 8, False), (17, 3, 64, 1, False),
                                                         (9, 5, 20, 0, False), (33, 4, 128, 0, True)])
def test_gate_of_latent_attention(T, heads, vdim, shift, per_head):
    n = heads if per_head else heads * vdim
    val, g = _rand(heads, T, vdim, dtype=BF), _rand(T, n + shift, dtype=BF)[:, shift:]
    y = torch.empty(T, heads * vdim, dtype=BF, device="cuda")
    K.latent_gate(val, g, y, heads, vdim, per_head)
    gate = torch.sigmoid(g.double())
    gate = gate.repeat_interleave(vdim, 1) if per_head else gate
    _close(y, val.double().transpose(0, 1).reshape(T, -1) * gate)


@pytest.mark.parametrize("kernel", ["gated_norm", "gated_norm_behind", "head_norm_sigmoid", "head_norm_silu", "wkv_out", "latent_gate", "swiglu"])
@pytest.mark.parametrize("W", [128, 100])
def test_gates_far_below_zero(kernel, W):
    """Gates down to where e^-z leaves 32 bits (z of -88.7): exponential and division are the 32-bit ones, so the result, a normal number, has
    all its bits; a reciprocal that flushes small numbers gives 0 from -87.3 on."""
    z = torch.linspace(-88.5, -80.0, 9 * W, device="cuda").to(BF).view(9, W)
    sig, x = torch.sigmoid(z.double()), 1e6 * (1.5 + torch.rand(9, W, device="cuda"))
    w, y, xd = torch.ones(W, device="cuda"), torch.empty(9, W, dtype=BF, device="cuda"), x.double()
    unit = xd / (xd.square().mean(-1, keepdim=True)).sqrt()
    if kernel == "gated_norm":                       # x silu(z) in front of the norm: the largest of a row has to count in its own size
        eps = 1e-30
        K.gated_rms_norm(x, (z, 0), w, eps, y, 1, True)
        v = xd * z.double() * sig
        want = v / (v.square().mean(-1, keepdim=True) + eps).sqrt()
    elif kernel == "gated_norm_behind":
        K.gated_rms_norm(x, (z, 0), 1e6 * w, 0.0, y, 1, False)
        want = 1e6 * unit * sig
    elif kernel.startswith("head_norm"):
        K.head_norm_gate(x, (z, 0), 1e6 * w, 0.0, y, 1, W, kernel[10:])
        want = 1e6 * unit * sig * (z.double() if kernel.endswith("silu") else 1)
    elif kernel == "wkv_out":
        K.wkv_out(x, z, 1e6 * w, 0.0, y, 1, W)
        want = 1e6 * unit * sig * z.double()
    elif kernel == "latent_gate":
        val = x.to(BF).view(1, 9, W)
        K.latent_gate(val, z, y, 1, W)
        want = val[0].double() * sig
    else:
        u = x.to(BF)
        K.silu_mul(torch.cat([z, u], 1), y)
        want = z.double() * sig * u.double()
    assert bool(((y.double() - want).abs() <= 2.0 ** -8 * want.abs()).all()) and bool((y != 0).all())


@pytest.mark.parametrize("H,dim,rot,rank,planes,shift", [(3, 16, 64, 200, 1, 0), (8, 128, 64, 512, 1, 8), (2, 24, 8, 8, 1, 0), (5, 16, 48, 264, 1, 0),
                                                         (3, 16, 64, 200, 2, 0), (2, 16, 72, 64, 1, 0), (2, 16, 64, 520, 1, 0), (3, 16, 64, 200, 1, 1)])
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("writes", [True, False])
def test_rows_of_latent_attention(H, dim, rot, rank, planes, shift, interleaved, writes):
    """Query and cache rows in the form with a warp a token and in the other (two planes, rotations of more than 64, ranks above 512, rows
    off a 16-byte boundary): ranks that fill no whole round of a warp, a page outside the pool, a layer that writes no rows."""
    T, d, block, blocks = 37, rank + rot, 8, 7
    q, dkv, q_abs = _rand(T, H * (dim + rot), dtype=BF), _rand(T, d + shift, dtype=BF, seed=1)[:, shift:], _rand(H, T, rank, dtype=BF, seed=2)
    w, freq = 1 + 0.1 * _rand(rank), 10000.0 ** (-torch.arange(rot // 2, dtype=F64, device="cuda") * 2 / rot)
    table = torch.tensor([[3, 1, 6], [2, blocks, 5]], dtype=torch.int32, device="cuda")      # the second sequence's second page is none
    ctx = SimpleNamespace(positions=torch.cat([torch.arange(2, 22), torch.arange(17)]).to(torch.int32).cuda(),
                          token_seq=torch.tensor([0] * 20 + [1] * 17, dtype=torch.int32, device="cuda"), status=torch.zeros(1, dtype=torch.int32, device="cuda"))
    pages, q_full = torch.full((blocks, planes, 1, block, d), 7.0, dtype=BF, device="cuda"), torch.empty(T, H * d, dtype=BF, device="cuda")
    K.latent_finish(q, dkv if writes else None, q_abs, w, 1e-6, freq, ctx, table, pages, q_full, H, dim, rot, rank, interleaved=interleaved)
    ang = ctx.positions.double()[:, None] * freq

    def turned(x):                                        # [T, n, rot]
        a, b = (x[..., 0::2], x[..., 1::2]) if interleaved else (x[..., :rot // 2], x[..., rot // 2:])
        cs, sn = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
        a, b = a * cs - b * sn, b * cs + a * sn
        return torch.stack([a, b], -1).flatten(-2) if interleaved else torch.cat([a, b], -1)
    qd = q.double().view(T, H, dim + rot)[..., dim:]
    _close(q_full.view(T, H, d), torch.cat([q_abs.double().transpose(0, 1), turned(qd)], -1))
    page = table[ctx.token_seq.long(), ctx.positions.long() // block].long()
    ok = page < blocks
    assert int(ctx.status) == (2 if writes else 0) and int(ok.sum()) == T - 8
    want = torch.full(pages.shape, 7.0, dtype=F64, device="cuda")
    if writes:
        x = dkv.double()
        c = x[:, :rank] / (x[:, :rank].square().mean(-1, keepdim=True) + 1e-6).sqrt() * w.double()
        at = (page[ok], 0, 0, ctx.positions.long()[ok] % block)
        want[at] = torch.cat([c, turned(x[:, None, rank:])[:, 0]], -1)[ok]
        if planes == 2:
            want[(page[ok], 1, 0, at[3])] = torch.cat([c, torch.zeros(T, rot, dtype=F64, device="cuda")], -1)[ok]
    _close(pages, want)


@pytest.mark.parametrize("T,W,top", [(9, 1024, 4), (3, 20, 1), (5, 2500, 8), (7, 1032, 9), (4, 30, 2)])
@pytest.mark.parametrize("form", ["plain", "shared", "weighted", "written"])
def test_sum_of_experts_rows(T, W, top, form):
    rows, wts, res, shared, z = _rand(T * top + 3, W), _rand(T, top), _rand(T, W, seed=1), _rand(T, W, seed=2), _rand(T, seed=3)
    row_of = torch.randperm(T * top + 3, device="cuda")[:T * top].to(torch.int32)
    want = (rows.double()[row_of.long()].view(T, top, W) * (1 if form == "weighted" else wts.double()[:, :, None])).sum(1)
    want = want + (shared.double() * torch.sigmoid(z.double())[:, None] if form != "plain" else 0)
    want = 0.5 * want + (0 if form == "written" else res.double())
    got = res.clone()
    K.moe_combine(got, rows, row_of, None if form == "weighted" else wts, None if form == "plain" else shared, 0.5, top=top,
                  shared_z=None if form == "plain" else z, overwrite=form == "written")
    # 32-bit sums of top + 2 terms
    assert bool(((got.double() - want).abs() <= 2.0 ** -23 * (top + 2) * rows.abs().max() * wts.abs().max().clamp(min=1) * 4).all())
