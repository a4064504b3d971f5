"""The scratch memory that the recurrences over prompts can do without (`Workspace.try_get`, `ops/kernels.py: _recurrence_scratch`):
what happens where the device refuses it, in a run that sizes the buffers and in the capture behind it."""
from types import SimpleNamespace

import pytest
import torch

from firefly_b200.engine.context import Workspace
from firefly_b200.ops import kernels as K


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
    _, p, size = K._recurrence_scratch(SimpleNamespace(workspace=ws), "ssm", "ff_scan_scratch_bytes", 32)
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
            n, p, size = K._recurrence_scratch(ctx, "ssm", "ff_scan_scratch_bytes", 32)
            assert n.value == n_long and size.value == (0 if n_long == 0 else 40) and len(ws.asked) == (n_long != 0)
            assert lens is None or ctx.memo[("long_seqs", 32)] == n_long
