"""Decode attention whose blocks are more than the GPU holds at once: the sequences are taken longest first, whatever their order."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", [0, 40])
@pytest.mark.parametrize("n", [56, 127, 128, 129])            # three ranges each: from here on more than a round; up to 300 tokens: in their own order
def test_longest_first_gives_what_single_sequences_give(n, window):
    from firefly_b200.engine.context import Workspace
    from firefly_b200.ops import kernels as K
    nq, nkv, d, block, dev = 8, 4, 64, 16, "cuda"
    lens = [(37 * i) % 300 if i % 5 else 90 for i in range(n)]    # many ties
    per = -(-301 // block)
    g = torch.Generator(device=dev).manual_seed(n)
    pages = torch.randn(n * per + 1, 2, nkv, block, d, generator=g, device=dev).to(torch.bfloat16)
    table = torch.arange(n * per, dtype=torch.int32, device=dev).view(n, per) + 1
    q = torch.randn(n, nq * d, generator=g, device=dev).to(torch.bfloat16)
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    ws, status = Workspace(torch.device(dev)), ints([0])
    splits = 3

    def run(rows):
        m = len(rows)
        out = torch.full((m, nq * d), 7.0, dtype=torch.bfloat16, device=dev)
        part = ws.get("o", (m * nq * splits * d,), torch.float32), ws.get("ml", (m * nq * splits * 2,), torch.float32)
        K.attn_decode(q[rows].contiguous(), nq * d, pages, table[rows].contiguous(), ints(list(range(m + 1))), ints([lens[r] for r in rows]), m, out, *part,
                      nq, nkv, d, d ** -0.5, window, splits, status)
        return out
    together = run(list(range(n)))
    for i in range(0, n, 8):                                     # few at a time: in order
        rows = list(range(i, min(n, i + 8)))
        assert torch.equal(together[rows], run(rows)), i
    assert int(status) == 0


def _long_lens(n):
    """Many ties, the longest behind the shortest, lengths on tile borders, and equal ones at last: up to 1500 tokens, so that spread and longest are large
    enough for the order to be taken."""
    return [(151 * i) % 1500 if i % 4 else 64 * (i % 7) for i in range(n - 3)] + [1500, 0, 1500]


@pytest.mark.parametrize("form", ["plain", "sink", "temperature"])
@pytest.mark.parametrize("n", [56, 64, 127, 128, 129])
def test_longest_first_with_heads_finished_in_the_kernel(n, form):
    """The newest key and value go into the pages of the sequence that the order gave the block: outputs and pages bit for bit those of a few sequences at
    a time, which stay in order."""
    from firefly_b200.engine.context import Workspace
    from firefly_b200.ops import kernels as K
    nq, nkv, d, block, dev, splits = 8, 4, 64, 16, "cuda", 3
    lens = _long_lens(n)
    per = -(-1501 // block)
    g = torch.Generator(device=dev).manual_seed(n)
    pages0 = torch.randn(n * per + 1, 2, nkv, block, d, generator=g, device=dev).to(torch.bfloat16)
    table = torch.randperm(n * per, generator=g, device=dev).to(torch.int32).view(n, per) + 1
    qkv = torch.randn(n, (nq + 2 * nkv) * d, generator=g, device=dev).to(torch.bfloat16)
    norm = [1 + 0.1 * torch.randn(d, generator=g, device=dev) for _ in range(2)]
    cos_sin = torch.randn(1600, d, generator=g, device=dev)
    sink = torch.randn(nq, generator=g, device=dev) if form == "sink" else None
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    ws = Workspace(torch.device(dev))

    def run(rows, pages):
        m, out, status = len(rows), torch.full((len(rows), nq * d), 7.0, dtype=torch.bfloat16, device=dev), ints([0])
        ctx = SimpleNamespace(num_seqs=m, cu_q=ints(list(range(m + 1))), ctx_lens=ints([lens[r] for r in rows]), max_kv_len=1501, workspace=ws, status=status,
                              ranges_by_length=False)
        K.attn_decode_heads(qkv[rows].contiguous(), pages, table[rows].contiguous(), ctx, out, nq, nkv, d, d ** -0.5, 0, *norm, 1e-6, cos_sin, splits,
                            sink=sink, q_temp=(0.1, 256) if form == "temperature" else None)
        assert int(status) == 0
        return out
    pages = pages0.clone()
    together = run(list(range(n)), pages)
    few = pages0.clone()
    for i in range(0, n, 8):
        rows = list(range(i, min(n, i + 8)))
        assert torch.equal(together[rows], run(rows, few)), i
    assert torch.equal(pages, few) and not torch.equal(pages, pages0)


@pytest.mark.parametrize("lens", [[1500 - 10 * i for i in range(64)], [703] + [0] * 63, [0] * 63 + [704], [1500] * 63 + [1310], [1500] * 63 + [1343]],
                         ids=["falling", "below_12_tiles", "12_tiles", "more_than_an_eighth", "an_eighth"])
def test_borders_of_where_the_order_is_taken(lens):
    from firefly_b200.engine.context import Workspace
    from firefly_b200.ops import kernels as K
    nq, nkv, d, block, dev, splits, n = 4, 4, 64, 16, "cuda", 3, len(lens)
    per = -(-1501 // block)
    g = torch.Generator(device=dev).manual_seed(lens[-1])
    pages = torch.randn(n * per + 1, 2, nkv, block, d, generator=g, device=dev).to(torch.bfloat16)
    table = torch.arange(n * per, dtype=torch.int32, device=dev).view(n, per) + 1
    q = torch.randn(n, nq * d, generator=g, device=dev).to(torch.bfloat16)
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    ws, status = Workspace(torch.device(dev)), ints([0])

    def run(rows):
        m, out = len(rows), torch.full((len(rows), nq * d), 7.0, dtype=torch.bfloat16, device=dev)
        part = ws.get("o", (m * nq * splits * d,), torch.float32), ws.get("ml", (m * nq * splits * 2,), torch.float32)
        K.attn_decode(q[rows].contiguous(), nq * d, pages, table[rows].contiguous(), ints(list(range(m + 1))), ints([lens[r] for r in rows]), m, out, *part,
                      nq, nkv, d, d ** -0.5, 0, splits, status)
        return out
    together = run(list(range(n)))
    for i in range(0, n, 8):
        rows = list(range(i, i + 8))
        assert torch.equal(together[rows], run(rows)), i
    assert int(status) == 0
