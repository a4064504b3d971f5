"""Decays from a low-rank projection: borders of tiles, ranks and channels, rows of weights on and off 16 bytes, both forms of the softplus."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tau", [1.0, 15.9, 16.0, 64.0])
@pytest.mark.parametrize("T,C,R,shift,dtype", [(1, 128, 16, 0, torch.bfloat16), (5, 129, 8, 0, torch.bfloat16), (777, 1024, 16, 0, torch.bfloat16),
                                               (4143, 256, 24, 0, torch.bfloat16), (33, 130, 17, 0, torch.bfloat16), (64, 64, 16, 1, torch.bfloat16),
                                               (31, 100, 20, 0, torch.float32), (4143, 1024, 900, 0, torch.bfloat16), (6, 40, 7, 0, torch.float32)])
def test_low_rank_decay(T, C, R, shift, dtype, tau):
    from firefly_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(T + C)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    low, flat, bias = rn(T, R + 3).to(dtype), rn(C * R + shift).to(dtype), 3 * rn(C)
    w = flat[shift:].view(C, R)
    alpha = torch.empty(T, C, device="cuda")
    K.low_rank_decay((low, 2), w, bias, tau, alpha)
    z = low[:, 2:2 + R].double() @ w.double().T + bias.double()
    want = torch.sigmoid(z) ** (1 / tau)
    size = low[:, 2:2 + R].double().abs() @ w.double().abs().T + bias.double().abs()
    # a sum of R + 1 products in 32-bit (which covers the exponent's own rounding, as |z| <= size), the softplus to 4.2e-7, the result to two
    # units; results below the smallest normal number (z of -88 and less) have fewer bits or none
    bound = want * (((R + 2) * 2.0 ** -24 * size + 4.2e-7) / tau + 2.0 ** -22) + 2.0 ** -126
    assert bool(((alpha.double() - want).abs() <= bound).all())
