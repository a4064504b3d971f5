"""Rules that choose a kernel by a step's sizes, on the host."""
from firefly_b200.ops import kernels as K


def test_which_steps_take_two_row_tiles_a_block(monkeypatch):
    """Long walks do, many short portions do not (they would leave half of every block idle), nor what leaves SMs without a block."""
    monkeypatch.setattr(K, "sm_count", lambda device=None: 148)
    two = lambda lens, before=0, G=4, nkv=8, window=0: K.attn_tc_two_tiles(lens, [before] * len(lens), G, nkv, window)  # noqa: E731
    assert two([8191]) and two([2048]) and two([3000] * 4) and two([512] * 8, 1024) and two([64] * 64, 2000)
    assert not two([1024]) and not two([32] * 40) and not two([1] * 128, G=32) and not two([256] * 64) and not two([512] * 16)
    assert not two([20] * 100, 2000) and not two([8191], window=128) and two([8191], window=4096)
