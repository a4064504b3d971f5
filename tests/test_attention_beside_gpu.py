"""The attention of single tokens beside that of portions in the same step: bit for bit what the two give one after the other."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# portions: many row tiles (two a block), few (keys shared out over blocks), shorter than a tile; single tokens in fixed ranges and by length
@pytest.mark.parametrize("q_lens,before", [([1] * 24 + [256, 256], [60 * i for i in range(24)] + [1536, 1500]), ([1, 2048], [0, 0]),
                                           ([1, 1, 3], [2000, 5, 700]), ([1] * 64 + [1500, 2], [31 * i for i in range(64)] + [0, 64]),
                                           ([1, 1, 0], [100, 30, 5])])            # a portion without a token: nothing to run beside
@pytest.mark.parametrize("d,by_length", [(128, False), (128, True), (64, False)])
def test_single_tokens_beside_portions(q_lens, before, d, by_length):
    from firefly_b200.engine.context import Workspace
    from firefly_b200.ops import kernels as K
    nq, nkv, block, dev, bf = 16, 4, 16, "cuda", torch.bfloat16
    n, T, n_dec = len(q_lens), sum(q_lens), q_lens.count(1)
    per = -(-max(a + b for a, b in zip(q_lens, before)) // block)
    g = torch.Generator(device=dev).manual_seed(d + n)
    pages = torch.randn(n * per + 1, 2, nkv, block, d, generator=g, device=dev).to(bf)
    table = (torch.arange(n * per, dtype=torch.int32, device=dev).view(n, per) + 1).contiguous()
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    ctx = SimpleNamespace(cu_q=ints([0] + list(np.cumsum(q_lens))), ctx_lens=ints(before), num_seqs=n, q_lens=q_lens, ctx_lens_host=before,
                          token_seq=ints(np.repeat(np.arange(n), q_lens).tolist()), positions=ints([c + i for c, ql in zip(before, q_lens) for i in range(ql)]),
                          num_decode_seqs=n_dec, max_kv_len=max(a + b for a, b in zip(q_lens, before)), ranges_by_length=by_length,
                          workspace=Workspace(torch.device(dev)), captured=False, memo={}, key_share_level=0, status=ints([0]))
    width = (nq + 2 * nkv) * d
    one = torch.ones(d, device=dev)
    out, want = torch.zeros(T, nq * d, dtype=bf, device=dev), torch.zeros(T, nq * d, dtype=bf, device=dev)
    rows = [torch.randn(T, width, generator=g, device=dev).to(bf) for _ in range(4)]
    qkv = torch.empty_like(rows[0])
    for it in range(12):
        qkv.copy_(rows[it % 4])
        # what both attentions read comes from the kernel in front of them
        K.qk_norm_rope_store(qkv, nq, nkv, d, one, one, 1e-6, None, 0, ctx.positions, ctx.token_seq, table, pages, ctx.status)
        K.paged_attention(qkv, width, pages, table, ctx, out, nq, nkv, d, d ** -0.5, 0)
        torch.cuda.synchronize()
        alone = SimpleNamespace(**dict(vars(ctx), num_seqs=n_dec, memo={}))
        K.paged_attention(qkv, width, pages, table, alone, want, nq, nkv, d, d ** -0.5, 0)
        tail = SimpleNamespace(**dict(vars(ctx), num_seqs=n - n_dec, num_decode_seqs=0, q_lens=q_lens[n_dec:], ctx_lens_host=before[n_dec:],
                                      cu_q=ctx.cu_q[n_dec:], ctx_lens=ctx.ctx_lens[n_dec:], memo={}))
        # (the rows of portions lie behind the single tokens': their first row is what the step says it is)
        tiles = sum(-(-(ql * nq // nkv) // 128) for ql in tail.q_lens)
        key_tiles = max(-(-(c + ql) // 64) for c, ql in zip(tail.ctx_lens_host, tail.q_lens))
        count = K.attn_tc_shares(tiles, nkv, key_tiles)
        cells = T * nq * count
        shares = (count, torch.empty(cells * d, device=dev), torch.empty(cells * 2, device=dev), n_dec, T - n_dec) if count > 1 else None
        K.attn_tc(qkv, width, pages, table[n_dec:], tail.cu_q, tail.ctx_lens, n - n_dec, tiles, want, nq, nkv, d, d ** -0.5, 0, ctx.status, shares=shares,
                  two_tiles=count == 1 and K.attn_tc_two_tiles(tail.q_lens, tail.ctx_lens_host, nq // nkv, nkv))
        torch.cuda.synchronize()
        assert torch.equal(out, want) and int(ctx.status) == 0, it
