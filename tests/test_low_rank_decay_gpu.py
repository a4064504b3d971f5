"""Decays from a low-rank projection: borders of tiles, ranks and channels, rows of weights on and off 16 bytes, and the softplus with all its bits."""
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
    # a sum of R + 1 products in 32-bit (which covers the exponent's own rounding, as |z| <= size); the softplus to 2.4e-7: an exponential of at most 1
    # to two units (1.2e-7), an addition to 1 and a logarithm of at most 0.7 (6e-8 each); the result to two units; results below the
    # smallest normal number (z of -88 and less) have fewer bits or none
    bound = want * (((R + 2) * 2.0 ** -24 * size + 2.4e-7) / tau + 2.0 ** -22) + 2.0 ** -126
    assert bool(((alpha.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("tau", [1.0, 16.0, 64.0])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_decays_have_all_their_bits(tau, dtype):
    """Decays of thousands of tokens are multiplied, so an error that no single one shows still counts: the exponential and logarithm are the 32-bit
    ones at every tau.  With z a number of the input's own (one weight of 1, no bias) nothing else rounds, and the same formula in 32 bits gives the
    same number but where another build of the two functions rounds another way (under 1 in 100; the fast ones change one in twenty and more)."""
    from firefly_b200.ops import kernels as K
    T, C = 4096, 64
    z = torch.linspace(-10, 14, T, device="cuda").to(dtype)[:, None].contiguous()
    alpha = torch.empty(T, C, device="cuda")
    K.low_rank_decay((z, 0), torch.ones(C, 1, dtype=dtype, device="cuda"), torch.zeros(C, device="cuda"), tau, alpha)
    z = z.float()
    inv_tau = (torch.ones((), device="cuda") / torch.tensor(tau, device="cuda"))
    want = torch.exp(-(torch.relu(-z) + torch.log(1 + torch.exp(-z.abs()))) * inv_tau).expand(T, C)
    assert float((alpha != want).float().mean()) < 0.01
    assert bool(((alpha - want).abs() <= 2.0 ** -22 * want).all())
