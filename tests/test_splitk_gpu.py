"""Products with few output tiles and a long contraction, which are cut along K: data gradients, and Linear layers of up to
128 rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from pipedream_b200 import functional as pf  # noqa: E402


# the first row count past the small-batch rule, a partial last K block, the largest tile count and one more, a width
# that the vector form of the second kernel does not take
@pytest.mark.parametrize("M,N,K", [(129, 1024, 2048), (400, 1024, 4104), (768, 1024, 2112), (769, 1024, 2048),
                                   (200, 1028, 2048), (33, 264, 4096)])
def test_long_contractions_against_float64(M, N, K):
    """fp32 sums in any order, rounded to bf16 once."""
    g = torch.Generator().manual_seed(M)
    a = torch.randn(M, K, generator=g).cuda().bfloat16()
    w = (torch.randn(N, K, generator=g) * 0.05).cuda().bfloat16()
    bias = torch.randn(N, generator=g).cuda().bfloat16()
    ref, mag = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()

    def check(got, want):
        assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + K * 2.0 ** -23 * mag).all()
    check(pf.gemm_nt(a, w, bias, relu=True), (ref + bias.double()).clamp_min(0))
    if N % 8 == 0:
        check(pf.gemm_nn(a, w.t().contiguous()), ref)
    prev = pf.set_deterministic(True)
    try:
        assert torch.equal(pf.gemm_nt(a, w), pf.gemm_nt(a, w))
    finally:
        pf.set_deterministic(prev)
    assert pf.gemm_poll_error() == 0
