"""The scratch memory that the recurrences over prompts can do without (`Workspace.try_get`, `ops/kernels.py: _recurrence_scratch`):
what happens where the device refuses it, in a run that sizes the buffers and in the capture behind it, and that the engine leaves
room for it."""
from types import SimpleNamespace

import pytest
import torch

from firefly_b200.config.base import PartSpec
from firefly_b200.engine.context import Workspace
from firefly_b200.engine.engine import Engine, EngineOptions
from firefly_b200.engine.graphs import DecodeGraphs
from firefly_b200.models.decoder import DecoderModel
from firefly_b200.ops import kernels as K
from firefly_b200.parts.base import Runtime, build_part


class _Small(Workspace):
    """A device that holds `room` numbers in one buffer."""

    def __init__(self, room, device="cpu"):
        super().__init__(device)
        self.room, self.asked = room, []

    def _allocate(self, n, dtype):
        self.asked.append(n)
        if n > self.room:
            raise torch.OutOfMemoryError("no memory left")
        return torch.empty(n, dtype=dtype)


def _scratch(ws, monkeypatch, numbers):
    monkeypatch.setattr(K, "_recurrence_scratch_bytes", lambda *a: 4 * numbers)
    _, p, size = K._recurrence_scratch(SimpleNamespace(workspace=ws), "ssm", "ff_scan_scratch_bytes", 32, ())
    assert (p.value is None) == (size.value == 0)
    return size.value // 4


def test_a_refused_size_is_not_asked_for_again(monkeypatch):
    ws = _Small(100)
    assert _scratch(ws, monkeypatch, 200) == 0 and ws.asked == [200]
    assert _scratch(ws, monkeypatch, 200) == 0 and _scratch(ws, monkeypatch, 300) == 0 and ws.asked == [200]
    assert _scratch(ws, monkeypatch, 50) == 50 and _scratch(ws, monkeypatch, 80) == 80 and ws.asked == [200, 50, 80]
    assert _scratch(ws, monkeypatch, 200) == 0 and _scratch(ws, monkeypatch, 60) == 60 and len(ws.asked) == 3
    with pytest.raises(torch.OutOfMemoryError):             # what a step cannot do without is asked for and raises
        ws.get("scan.o", (500,), torch.float32)


def test_a_capture_takes_what_the_run_before_it_took(monkeypatch):
    """The run that sizes the buffers is refused one layer's records and gets another's; the capture behind it answers the same
    and allocates nothing, also when memory has become free in between."""
    capturing = [False]
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing[0])
    ws = _Small(100, "cuda")
    first = [_scratch(ws, monkeypatch, n) for n in (50, 200)]
    version, asked, capturing[0], ws.room = ws.version, len(ws.asked), True, 10 ** 6
    assert [_scratch(ws, monkeypatch, n) for n in (50, 200)] == first == [50, 0]
    assert _scratch(ws, monkeypatch, 70) == 0               # never seen before: not while a graph is captured
    assert ws.version == version and len(ws.asked) == asked
    capturing[0] = False
    assert _scratch(ws, monkeypatch, 70) == 70              # a capture is no refusal


def test_a_frozen_workspace_answers_none(monkeypatch):
    ws = _Small(100)
    assert _scratch(ws, monkeypatch, 50) == 50
    ws.frozen = True
    assert _scratch(ws, monkeypatch, 60) == 0 and _scratch(ws, monkeypatch, 50) == 50 and _scratch(ws, monkeypatch, 40) == 40
    assert ws.asked == [50]


def test_no_long_sequence_no_scratch_memory(monkeypatch):
    """What goes by chunks is counted from the host's copy of the lengths, once a step; a step without such a sequence asks for nothing."""
    monkeypatch.setattr(K, "_recurrence_scratch_bytes", lambda *a: 40)
    for lens, n_long in (([1, 1, 31], 0), ([1, 32, 500], 2), (None, -1)):
        ws = _Small(100)
        ctx = SimpleNamespace(workspace=ws, q_lens=lens, memo={})
        for _ in range(2):
            n, p, size = K._recurrence_scratch(ctx, "ssm", "ff_scan_scratch_bytes", 32, ())
            assert n.value == n_long and size.value == (0 if n_long == 0 else 40) and len(ws.asked) == (n_long != 0)
            assert lens is None or ctx.memo[("long_seqs", 32)] == n_long


class _Holder:
    def __init__(self, *parts):
        self._parts = parts

    def parts(self):
        return list(self._parts)


def test_the_engine_leaves_room_for_the_records():
    """The largest of a model's parts counts, wherever it stands, for the longest step and for the longest captured one."""
    mixer = lambda scale: SimpleNamespace(step_scratch_bytes=lambda tokens, n: scale * (tokens + n))  # noqa: E731
    model = SimpleNamespace(blocks=[_Holder(object(), mixer(3)), _Holder(_Holder(mixer(7)), mixer(5)), object()],
                            spec=SimpleNamespace(hidden_size=16, vocab_size=100))
    model.step_scratch_bytes = lambda tokens, n: DecoderModel.step_scratch_bytes(model, tokens, n)
    plain = SimpleNamespace(spec=model.spec)
    opts = EngineOptions(max_num_batched_tokens=8000, max_batch_size_limit=10)
    estimate = lambda m, o: Engine._scratch_estimate(SimpleNamespace(model=m), o)  # noqa: E731
    assert estimate(model, opts) - estimate(plain, opts) == 7 * 8010 + 7 * (DecodeGraphs.SHAPE_MAX_TOKENS + 10)
    opts.use_cuda_graphs = False
    assert estimate(model, opts) - estimate(plain, opts) == 7 * 8010


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["wkv", "state_space", "channel_delta", "gated_linear_attention", "linear_attention"])
def test_a_mixer_says_what_its_recurrence_takes(kind):
    H, N, lens = 4, 64, [300, 1, 70]
    T, n, bf = sum(lens), len(lens), torch.bfloat16
    params = dict(hidden_size=256, eps=1e-6, heads=H, dim=N)
    params.update({"wkv": dict(decay_rank=8), "state_space": dict(vdim=N, state=N, conv=4), "linear_attention": dict(decay=[0.9] * H),
                   "gated_linear_attention": dict(decay_rank=8, tau=16.0), "channel_delta": dict(kv_heads=H, vdim=N, conv=4)}[kind])
    part = build_part("mixer", PartSpec(kind, params), Runtime(torch.device("cuda"), bf))
    x = torch.randn(T, 4 * H * N, device="cuda").to(bf)
    f = lambda *s: torch.randn(*s, device="cuda")  # noqa: E731
    cu = torch.tensor([0, 300, 301, 371], dtype=torch.int32, device="cuda")
    ctx = SimpleNamespace(cu_q=cu, num_seqs=n, q_lens=lens, workspace=Workspace("cuda"), memo={},
                          state_slots=torch.arange(1, n + 1, dtype=torch.int32, device="cuda"), seq_fresh=torch.ones(n, dtype=torch.int32, device="cuda"))
    state, o, q, k, v = f(n + 1, H * N * N + 256), f(T, H * N), (x, 0), (x, H * N), (x, 2 * H * N)
    if kind == "wkv":
        K.wkv_scan(x.view(T, 4, H * N).transpose(0, 1).contiguous(), f(T, H * N), f(H * N), f(H * N), state, H * N * N, x[:, :256].contiguous(), ctx, o, H, N)
    elif kind == "channel_delta":
        K.delta_rule_scan(q, k, v, (x, 0), (f(T, H * N), 0), f(H * N), f(H), state, 0, ctx, o, H, N, N)
    else:
        kw = {"state_space": dict(step=(x, 0), step_bias=f(H), a_log=f(H), heads_per_group=H), "linear_attention": dict(decay=f(H), silu_inputs=True),
              "gated_linear_attention": dict(channel_decay=(torch.rand(T, H * N, device="cuda"), 0))}[kind]
        K.scalar_decay_scan(q, k, v, state, 0, ctx, o, H, N, N, **kw)
    assert part.step_scratch_bytes(T, n) == ctx.workspace.bytes() and (ctx.workspace.bytes() > 0) == (kind != "linear_attention")
