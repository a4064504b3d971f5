"""The first and the last kernel of a step: rows out of the embedding, and the sampled tokens with the status word behind them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,shift,dtype", [(8, 0, torch.bfloat16), (12, 0, torch.bfloat16), (4104, 0, torch.bfloat16), (1024, 1, torch.bfloat16),
                                           (4, 0, torch.float32), (2052, 0, torch.float32), (64, 1, torch.float32), (20000, 0, torch.bfloat16)])
def test_embedding_rows_by_16_bytes_and_one_by_one(H, shift, dtype):
    from firefly_b200.ops import kernels as K
    V, T = 33, 9
    flat = torch.randn(V * H + shift, device="cuda").to(dtype)
    table = flat[shift:].view(V, H)                              # shift 1: not on a 16-byte border
    ids = torch.randint(0, V, (T,), dtype=torch.int32, device="cuda")
    out, status = torch.full((T, H), 7.0, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    K.embedding(ids, table, out, status)
    assert torch.equal(out, table[ids.long()].float()) and int(status) == 0
    ids[3] = -1
    K.embedding(ids, table, out, status)
    assert int(status) == 1


@pytest.mark.parametrize("rows,V", [(1, 300), (5, 300), (1, 151936), (64, 32768)])
def test_status_word_behind_the_tokens(rows, V):
    from firefly_b200.ops import kernels as K
    logits = torch.randn(rows, V, device="cuda")
    out, status = torch.full((rows + 2,), -7, dtype=torch.int32, device="cuda"), torch.full((1,), 42, dtype=torch.int32, device="cuda")
    K.sample(logits, out, status=status)
    assert out[:rows].tolist() == logits.argmax(-1).tolist() and out[rows:].tolist() == [42, -7]
