"""The tiled layout kernels and the masked batch-norm passes at the sizes where they can go wrong."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

from pipedream_b200 import functional as pf  # noqa: E402

DTYPES = [torch.float32, torch.bfloat16]


def rnd(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).cuda()


def padded(x, dtype):
    return F.pad(x.to(dtype), (1, 1, 1, 1)).permute(0, 2, 3, 1).contiguous()


# one pixel, a tile of 64 pixels exactly and one more, channels beside multiples of the 64-channel tile, many images
SHAPES = [(1, 8, 1, 1), (2, 64, 8, 8), (3, 72, 5, 13), (1, 2048, 7, 7), (2, 136, 1, 65), (33, 16, 3, 3)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("src", DTYPES, ids=["f32", "bf16"])
@pytest.mark.parametrize("dst", DTYPES, ids=["f32", "bf16"])
def test_pack_unpack_tiles(shape, src, dst):
    """Values only move or round once: bit-equal to torch for every order and stride of the source."""
    N, C, H, W = shape
    x = rnd(*shape, seed=1).to(src)
    wide = rnd(N, C, 2 * H, 2 * W, seed=2).to(src)
    odd = torch.empty(x.numel() + 1, dtype=src, device="cuda")[1:].view(N, H, W, C)      # channels last, off 16 bytes
    odd.copy_(x.permute(0, 2, 3, 1))
    sources = [x, x.contiguous(memory_format=torch.channels_last), odd.permute(0, 3, 1, 2), wide[:, :, ::2, ::2],
               wide.contiguous(memory_format=torch.channels_last)[:, :, 1::2, 1::2],
               wide.transpose(2, 3).contiguous().transpose(2, 3)[:, :, :H, :W], x[:1].expand(N, C, H, W)]
    for s in sources:
        assert torch.equal(pf.pack_pnhwc(s, dst), padded(s, dst))
    pad = padded(x, src)
    assert torch.equal(pf.unpack_pnhwc(pad, dst), x.to(dst))


@pytest.mark.parametrize("dtype", DTYPES, ids=["f32", "bf16"])
@pytest.mark.parametrize("res", [False, True], ids=["plain", "residual"])
@pytest.mark.parametrize("shape", [(1, 8, 1, 2), (5, 64, 9, 7), (2, 2048, 3, 3), (9, 256, 28, 28)], ids=str)
def test_batchnorm_mask(dtype, res, shape):
    """The mask says y > 0, and the backward pass gives the same from it as from y."""
    N, C, H, W = shape
    x, dy = padded(rnd(*shape, seed=3), dtype), padded(rnd(*shape, seed=4), dtype)
    sc = padded(rnd(*shape, seed=5), dtype) if res else None
    gamma, beta = (rnd(C, seed=6) * 0.2 + 1).to(dtype), rnd(C, seed=7).to(dtype)
    y, mean, invstd, mask = pf.bn_fwd(x, gamma, beta, 1e-5, 0.1, True, None, None, sc, want_mask=True)
    bits = (mask.view(-1, 1) >> torch.arange(8, device="cuda", dtype=torch.uint8)) & 1
    assert torch.equal(bits.view(y.shape).bool(), y > 0)
    got = []
    for kw in ({"mask": mask}, {}):
        dg, db = torch.empty(C, device="cuda"), torch.empty(C, device="cuda")
        got.append(pf.bn_bwd(x, dy, y, gamma, mean, invstd, dg, db, False, want_dres=True, **kw) + (dg, db))
    for a, b in zip(*got):
        assert torch.equal(a, b)


def test_batchnorm_from_variance():
    x, gamma, beta = padded(rnd(3, 64, 5, 5, seed=8), torch.bfloat16), rnd(64, seed=9).bfloat16(), rnd(64, seed=10).bfloat16()
    mean, var = rnd(64, seed=11), rnd(64, seed=12).square()
    want = pf.bn_apply(x, gamma, beta, mean, torch.rsqrt(var + 1e-5), True)
    assert torch.equal(pf.bn_apply_var(x, gamma, beta, mean, var, 1e-5, True), want)
