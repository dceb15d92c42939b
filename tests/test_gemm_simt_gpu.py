"""The fp32 contraction kernel's three tiles at their edges: remainders in every direction, rows that do not start on
16-byte boundaries, K slices, against float64.  Bound: every product and sum is rounded to fp32 once, so an output is
within (K + 8) 2^-24 of sum |a||b|, whatever the order of the sum."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from pipedream_b200 import functional as pf      # noqa: E402


def _mat(rows, cols, ld, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(rows, ld, generator=g).cuda()[:, :cols]


def _check(got, a, b, k):
    a, b = a.double(), b.double()
    ref, mag = a @ b, a.abs() @ b.abs()
    assert ((got.double() - ref).abs() <= (k + 8) * 2.0 ** -24 * mag + 1e-30).all()


# 64x64 tile; 128x64 (many rows, narrow); 128x128; odd leading dimensions; K below, at and past a chunk of 16
@pytest.mark.parametrize("M,N,K,odd", [(1, 8, 1, False), (63, 65, 15, True), (64, 64, 16, False), (130, 129, 17, False),
                                       (40001, 64, 33, False), (40001, 61, 9, True), (5003, 1030, 48, False),
                                       (5003, 1029, 31, True), (7, 1000, 2048, False), (8, 34, 132, False), (1, 66, 4, False), (8, 4096, 516, False)])
def test_tiles(M, N, K, odd):
    ld = lambda n: n + 3 if odd else (n + 3) // 4 * 4
    a, b = _mat(M, K, ld(K), 1), _mat(N, K, ld(K), 2)
    _check(pf.gemm_nt(a, b), a, b.t(), K)
    c = _mat(K, N, ld(N), 3)
    _check(pf.gemm_nn(a, c), a, c, K)
    at = _mat(K, M, ld(M), 4)
    out = torch.zeros(M, N, device="cuda")
    for split in (0, 1, 3):
        _check(pf.gemm_tn(at, c, out, accumulate=False, split_k=split), at.t(), c, K)


@pytest.mark.parametrize("N,H,Cin,Cout", [(1, 7, 64, 8), (2, 14, 64, 192), (1, 30, 128, 64)])
def test_convolution_passes(N, H, Cin, Cout):
    g = torch.Generator().manual_seed(5)
    x, w = torch.randn(N, Cin, H, H, generator=g).cuda(), torch.randn(Cout, Cin, 3, 3, generator=g).cuda()
    dy = torch.randn(N, Cout, H, H, generator=g).cuda()
    wl = w.contiguous(memory_format=torch.channels_last)
    xp, dyp = pf.pack_pnhwc(x), pf.pack_pnhwc(dy)
    inner = lambda t: t[:, 1:-1, 1:-1].permute(0, 3, 1, 2)
    conv = lambda u, v: torch.nn.functional.conv2d(u.double(), v.double(), padding=1)
    back = lambda u, v: torch.nn.functional.conv_transpose2d(u.double(), v.double(), padding=1)
    eps = 2.0 ** -24
    y = pf.conv2d_fwd(xp, wl, wl.stride(0), Cout, None, False)
    assert ((inner(y) - conv(x, w)).abs() <= (9 * Cin + 8) * eps * conv(x.abs(), w.abs())).all()
    assert y[:, 0].abs().max() == 0 and y[:, :, -1].abs().max() == 0
    dx = pf.conv2d_dgrad(dyp, wl, wl.stride(0), Cin)
    assert ((inner(dx) - back(dy, w)).abs() <= (9 * Cout + 8) * eps * back(dy.abs(), w.abs())).all()
    dw = torch.zeros_like(wl)
    ref = lambda u, v: torch.nn.grad.conv2d_weight(u.double(), w.shape, v.double(), padding=1)
    for split in (0, 1):
        pf.conv2d_wgrad(xp, dyp, dw, dw.stride(0), accumulate=False, split_k=split)
        assert ((dw - ref(x, dy)).abs() <= (N * (H + 2) ** 2 + 8) * eps * ref(x.abs(), dy.abs())).all()


# the last output tile and the last chunk of 64 k partly filled; operands whose rows are not on 16 bytes
@pytest.mark.parametrize("M,N,K", [(2051, 1029, 1000), (1920, 1160, 4608), (2048, 1024, 71)])
@pytest.mark.parametrize("form", ["nt", "nn", "tn"])
def test_tensor_core_parts_against_float64(form, M, N, K):
    """Products large enough for the three-part tile.  Bound: a chunk of 64 k rounds (towards zero) at most six times at
    the size of its sum, the K/64 chunk sums round to nearest once each, and those roundings are independent."""
    g = torch.Generator().manual_seed(M + K)
    a, b = torch.randn(M, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda()
    ref = a.double() @ b.double().t()
    if form == "nt":
        out = pf.gemm_nt(a, b)
    elif form == "nn":
        out = pf.gemm_nn(a, b.t().contiguous())
    else:
        out = torch.zeros(M, N, device="cuda")
        pf.gemm_tn(a.t().contiguous(), b.t().contiguous(), out)
    rel = ((out.double() - ref).norm() / ref.norm()).item()
    assert rel <= 2.0 ** -24 * (6 + (K / 64) ** 0.5), rel
    assert pf.gemm_poll_error() == 0


def test_tensor_core_parts_keep_infinities():
    """Values whose parts would multiply to NaN (infinities, and what rounds up to one) give what fp32 gives."""
    g = torch.Generator().manual_seed(5)
    a, b = torch.randn(1920, 512, generator=g).cuda(), torch.randn(1160, 512, generator=g).cuda()
    a[3, 7], a[200, 1], b[5, 2], a[900, 500] = float("inf"), -float("inf"), float("nan"), 3.4e38
    a[1500], b[1100] = 1e-41, 1e-30                      # subnormal inputs and products
    out, ref = pf.gemm_nt(a, b), a.double() @ b.double().t()
    want = ref.float()
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isinf(), want.isinf())
    assert torch.equal(out[out.isinf()], want[want.isinf()])
    fine = want.isfinite()
    # relative to a row's products, not to their sum; a part below bf16's smallest step (2^-133) is lost whole, which
    # shows where a row has subnormal values only
    A, B = a.double().abs(), b.double().abs()
    bound = 2.0 ** -20 * (A @ B.t()) + 2.0 ** -133 * (A.sum(1, keepdim=True) + B.sum(1))
    assert ((out.double() - ref).abs() <= bound)[fine].all()
