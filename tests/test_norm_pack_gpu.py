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
