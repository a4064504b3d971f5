"""What a layer of a mixed step asks of the attention kernels' libraries, and in which order: the single tokens' kernel waits for nothing when the
portions' kernel is the launch right in front of it, so nothing may come between the two; and every call costs host time."""
from types import SimpleNamespace

import pytest
import torch

from firefly_b200.ops import kernels as K


class _Library:
    def __init__(self, calls):
        self.calls = calls

    def __getattr__(self, name):
        return lambda *args: (self.calls.append((name, [getattr(a, "value", a) for a in args])), 0)[1]


@pytest.fixture
def calls(monkeypatch):
    seen = []
    for name in ("_attn_lib", "_attn_tc_lib"):
        monkeypatch.setattr(K, name, lambda *a, **k: _Library(seen))
    monkeypatch.setattr(K, "_need_cuda", lambda *a: None)
    monkeypatch.setattr(K, "_stream", lambda: K.c_void_p(0))
    monkeypatch.setattr(K, "sm_count", lambda: 148)
    monkeypatch.setattr(K, "_decode_places_per_kv_head", lambda nkv, d: 55)
    return seen


def _step(q_lens, before, by_length=False):
    from firefly_b200.engine.context import Workspace
    n, n_dec, nq, nkv, d, block = len(q_lens), q_lens.count(1), 16, 8, 128, 16
    ints = lambda x: torch.tensor(x, dtype=torch.int32)
    per = -(-max(a + b for a, b in zip(q_lens, before)) // block)
    ctx = SimpleNamespace(cu_q=ints([sum(q_lens[:i]) for i in range(n + 1)]), ctx_lens=ints(before), num_seqs=n, q_lens=q_lens, ctx_lens_host=before,
                          num_decode_seqs=n_dec, max_kv_len=per * block, ranges_by_length=by_length, workspace=Workspace(torch.device("cpu")),
                          captured=False, memo={}, status=ints([0]))
    T = sum(q_lens)
    pages, table = torch.zeros(2, 2, nkv, block, d, dtype=torch.bfloat16), torch.zeros(n, per, dtype=torch.int32)
    before_count = K.LAUNCHES
    K.paged_attention(torch.zeros(T, (nq + 2 * nkv) * d, dtype=torch.bfloat16), (nq + 2 * nkv) * d, pages, table, ctx,
                      torch.zeros(T, nq * d, dtype=torch.bfloat16), nq, nkv, d, 0.1, 0)
    return K.LAUNCHES - before_count


@pytest.mark.parametrize("by_length", [False, True])
def test_portions_that_fill_the_gpu_take_two_calls(calls, by_length):
    launches = _step([1] * 8 + [2048, 600], [500] * 7 + [3000, 0, 64], by_length)
    assert [c[0] for c in calls] == ["ff_attn_tc", "ff_attn_decode_units" if by_length else "ff_attn_decode"]
    assert launches == 3                                         # two attentions, and the join of the single tokens' ranges


def test_portions_whose_keys_are_shared_out_take_a_third_call_behind_both(calls):
    launches = _step([1] * 8 + [65], [300] * 8 + [1500])
    assert [c[0] for c in calls] == ["ff_attn_tc", "ff_attn_decode", "ff_attn_tc_join"]
    assert calls[0][1][-2] == 0                                  # no join in the first one: it would stand between the two
    assert launches == 4


def test_portions_without_a_token_leave_nothing_to_run_beside(calls):
    _step([1, 1, 0], [100, 30, 5])
    assert [c[0] for c in calls] == ["ff_attn_tc", "ff_attn_decode"] and calls[1][1][-3] == 0


@pytest.mark.parametrize("q_lens,before", [([1] * 8 + [65], [300] * 8 + [1500]), ([1] * 8 + [2048], [300] * 8 + [0])])
def test_single_tokens_run_beside_the_portions_kernel_right_in_front_of_them(calls, q_lens, before):
    _step(q_lens, before)
    at = [c[0] for c in calls].index("ff_attn_decode")
    assert calls[at][1][-3] == 1 and calls[at - 1][0] == "ff_attn_tc"
