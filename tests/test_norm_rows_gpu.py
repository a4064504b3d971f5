"""Residual add and norm with the row in registers: widths around its limits, selected rows, no delta, and rows of many blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [4, 508, 512, 516, 4100, 16384, 16388])
@pytest.mark.parametrize("ddt,odt", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.float32, torch.bfloat16)])
def test_add_rms_norm_rows(H, ddt, odt):
    from firefly_b200.ops import kernels as K
    rows, eps = 300, 1e-6
    g = torch.Generator(device="cuda").manual_seed(H)
    res, w = 3 * torch.randn(rows, H, generator=g, device="cuda"), 1 + 0.1 * torch.randn(H, generator=g, device="cuda")
    delta = torch.randn(rows, H, generator=g, device="cuda").to(ddt)
    pick = torch.tensor([299, 0, 7, 7], dtype=torch.int32, device="cuda")
    for d in (delta, None):
        for idx in (None, pick):
            r, out = res.clone(), torch.empty(rows if idx is None else 4, H, dtype=odt, device="cuda")
            K.add_rms_norm(r, d, w, eps, out, idx) if idx is not None else K.add_rms_norm(r, d, w, eps, out)
            x = res if d is None else res + d.float()
            assert torch.equal(r, x if idx is None else res)
            x = (x if idx is None else x[pick.long()]).double()
            want = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()
            # the root of a 32-bit sum over the row, two products; then the result's own rounding
            tol = 2.0 ** -20 + (2.0 ** -8 if odt == torch.bfloat16 else 0.0)
            assert bool(((out.double() - want).abs() <= tol * want.abs() + 1e-30).all()), (H, d is None, idx is None)
