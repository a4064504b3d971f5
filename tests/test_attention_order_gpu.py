"""Decode attention whose blocks are more than the GPU holds at once: the sequences are taken longest first, whatever their order."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", [0, 40])
@pytest.mark.parametrize("n", [56, 127, 128, 129])            # three ranges each: from here on more than a round; a block ranks up to 128 sequences
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
