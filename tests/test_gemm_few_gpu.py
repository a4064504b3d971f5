"""The product of a few tokens with a small matrix (csrc/gemm_few.cu) against the products in 64-bit: every epilogue, sizes around its tiles and limits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# K: one step of a warp, less than a step for some, a ring that wraps, the longest; N: parts of a block, both numbers of warps
SIZES = [(16, 32), (7, 96), (33, 288), (1000, 1024), (2368, 2080), (2369, 512), (4096, 1024), (640, 3584),
         # eight warps a block with long rows: three and two blocks an SM, and a second round of blocks that is half full
         (4200, 2048), (4736, 3328), (7104, 2560)]


def _K():
    from firefly_b200.ops import kernels as K
    return K


def _rand(seed):
    g = torch.Generator().manual_seed(seed)
    return lambda *s: torch.randn(*s, generator=g)


@pytest.mark.parametrize("T", [1, 3, 8])
@pytest.mark.parametrize("N,Kd", SIZES)
def test_epilogues(T, N, Kd):
    """Sums of K products in 32 bits, in any order: within K / 2 units in the last place of the sum of their sizes, 16-bit results within half of one."""
    K = _K()
    rn = _rand(N + Kd + T)
    x, w, base = rn(T, Kd).to(torch.bfloat16), (rn(N, Kd) / Kd ** 0.5).to(torch.bfloat16), rn(T, N)
    assert K.gemm_few_usable(T, N, Kd)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    tol32 = size * Kd * 2.0 ** -25 + 1e-30
    xd, wd = x.cuda(), w.cuda()
    torch.cuda.synchronize()         # the weights are asked for in front of whatever runs before
    out = base.cuda()
    K.gemm_few(xd, wd, out, K.EPI_RESIDUAL_ADD)
    assert ((out.cpu().double() - base.double() - want).abs() <= tol32 + 2.0 ** -23 * (base.double().abs() + want.abs())).all()
    out = torch.full((T, N), float("nan"), device="cuda")
    K.gemm_few(xd, wd, out, K.EPI_F32)
    assert ((out.cpu().double() - want).abs() <= tol32).all()
    for epi, ref in ((K.EPI_BF16, want), (K.EPI_RELU2, want.clamp(min=0) ** 2)):
        out = torch.full((T, N), float("nan"), dtype=torch.bfloat16, device="cuda")
        K.gemm_few(xd, wd, out, epi)
        slack = tol32 * (1 if epi == K.EPI_BF16 else 2 * want.abs() + tol32)
        assert ((out.cpu().double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1.01 * slack).all()
    if N % 32 == 0:
        gate, up = want[:, : N // 2], want[:, N // 2:]
        out = torch.full((T, N // 2), float("nan"), dtype=torch.bfloat16, device="cuda")
        K.gemm_few(xd, K.interleave_gate_up(wd[: N // 2], wd[N // 2:]), out, K.EPI_SWIGLU)
        ref = gate * torch.sigmoid(gate) * up
        slack = 1.1 * tol32[:, : N // 2] * up.abs() + tol32[:, N // 2:] * gate.abs() + 2.0 ** -20 * ref.abs()
        assert ((out.cpu().double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1.1 * slack).all()


@pytest.mark.parametrize("T", [1, 5, 8])
@pytest.mark.parametrize("H", [72, 1024, 2400, 3520])
def test_rms_norm_folded_into_two_products(T, H):
    """Few and many rows of sums of squares, and sums handed to and taken from `gemm_tc`."""
    K = _K()
    rn = _rand(T + H)
    Ka, Nb, eps = 512, 320, 1e-5
    res0, xa, nw = 2 * rn(T, H), rn(T, Ka).to(torch.bfloat16), 1 + 0.1 * rn(H)
    wa, wb = (rn(H, Ka) / Ka ** 0.5).to(torch.bfloat16), (rn(Nb, H) / H ** 0.5).to(torch.bfloat16)
    wa_d, wb_d, nw_d, xa_d = wa.cuda(), wb.cuda(), nw.cuda(), xa.cuda()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    res_want = res0.double() + xa.double() @ wa.double().T
    xn = res_want * torch.rsqrt((res_want ** 2).mean(-1, keepdim=True) + eps) * nw.double()
    want = xn @ wb.double().T
    for rows, first in ((K.gemm_few_rows(), lambda *a, **k: K.gemm_few(*a, **k)), (128, lambda x, w, o, e, **k: K.gemm_tc(x, w, o, e, 1, status, **k))):
        res, xw = res0.cuda(), torch.zeros(T, H, dtype=torch.bfloat16, device="cuda")
        ssq = torch.full((-(-H // rows), T), float("nan"), device="cuda")
        first(xa_d, wa_d, res, K.EPI_RESIDUAL_ADD, norm_out=(xw, nw_d, ssq))
        assert torch.allclose(ssq.sum(0).cpu().double(), (res.cpu().double() ** 2).sum(-1), rtol=1e-5)
        assert torch.equal(xw, (res * nw_d).to(torch.bfloat16))
        for second in (lambda o: K.gemm_few(xw, wb_d, o, K.EPI_F32, norm_in=(ssq, H, eps)) if H % 32 == 0 else None,
                       lambda o: K.gemm_tc(xw, wb_d, o, K.EPI_F32, 1, status, norm_in=(ssq, H, eps))):
            out = torch.full((T, Nb), float("nan"), device="cuda")
            if second(out) is None and torch.isnan(out).any():
                assert H % 32
                continue
            assert float((out.cpu().double() - want).norm() / want.norm()) < 2.0 ** -8      # xw is rounded to 16 bits
    assert int(status) == 0


def test_limits():
    """Sizes that it does not take go to `gemm_tc`."""
    K = _K()
    assert not K.gemm_few_usable(9, 512, 512) and not K.gemm_few_usable(1, 512, 72) and not K.gemm_few_usable(1, 512, 4096)
    # the rows of all blocks on the GPU at once, whatever K: 4, 3, 2 and 1 blocks of 16 rows an SM; a second round where the rows are short or it is half full
    row = 16 * K.sm_count()
    for Kd, most in ((1536, 4 * row), (1568, 4 * row), (2304, 4 * row), (2816, 2 * row), (3328, 2 * row), (3552, row), (3584, row)):
        assert K.gemm_few_usable(1, most, Kd) and not K.gemm_few_usable(1, most + 1, Kd), Kd
    assert K.gemm_few_usable(8, 3 * row, 3072) and not K.gemm_few_usable(8, 3 * row - 16, 3072) and not K.gemm_few_usable(1, 3 * row, 3104)
    x, w = torch.zeros(9, 64, dtype=torch.bfloat16, device="cuda"), torch.zeros(16, 64, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(K.KernelError, match="bad argument"):
        K.gemm_few(x, w, torch.zeros(9, 16, device="cuda"), K.EPI_F32)
