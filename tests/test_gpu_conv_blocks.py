"""Convolutions whose pixels arrive by blocks of 32 or 16 channels, against the gathering producer, bit for bit.

Both walk K in the same order, 16 elements per MMA; a number of blocks that does not fill the last slab leaves part of it out.
"""
import pytest
import torch

from helix_b200 import ops
from helix_b200._lib import OP_CONV_F16

pytestmark = pytest.mark.gpu


# 27, 125, 27, 12 and 9 blocks of 32 channels, 27, 25 and 52 of 16; more images than one tile, a cut last tile, pixels beyond the image, infinities where
# the absent half would be read
@pytest.mark.parametrize("geom", [(9, 96, 14, 14, 72, 3, 1, 1), (3, 160, 17, 19, 136, 5, 2, 2), (40, 96, 9, 7, 200, 3, 2, 0),
                                  (5, 96, 21, 16, 64, 2, 1, 0), (7, 32, 25, 24, 40, 3, 1, 1), (3, 48, 30, 31, 136, 3, 2, 1),
                                  (11, 16, 20, 22, 200, 5, 1, 2), (2, 208, 19, 19, 72, 2, 1, 1)])
@pytest.mark.parametrize("bn,swap", [(64, 0), (128, 0), (192, 0), (256, 0), (64, 1), (192, 1), (256, 1), (0, 0)])
def test_blocks_of_channels_equal_the_gathered_convolution(geom, bn, swap):
    nb, c, h, w, ko, r, stride, pad = geom
    if swap and ko <= 64 and c != 96:
        pytest.skip("swapped tiles of up to 64 output channels run M = 64 MMAs, which take no blocks")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(c + ko)
    x = torch.empty((nb, h, w, c), dtype=torch.float16, device="cuda").normal_(0, 1, generator=gen)
    if nb * h * w * c * 2 < 131072:        # smaller inputs do not go through the tensor map
        x = x.repeat(131072 // (nb * h * w * c * 2) + 1, 1, 1, 1)
    f = torch.empty((ko, r, r, c), dtype=torch.float16, device="cuda").normal_(0, 0.05, generator=gen)
    x[0, -1, -1, -1] = float("inf")
    cfg = ops.make_cfg(OP_CONV_F16, 128, bn, 64, swap_ab=swap) if bn else None
    got = ops.conv2d_f16_nhwc(x, f, stride, pad, cfg=cfg)
    ref = ops.conv2d_f16_nhwc(x, f, stride, pad, cfg=ops.make_cfg(OP_CONV_F16, 128, 64, 64, conv_gather=1))
    torch.cuda.synchronize()
    ops.check_status()
    exact = torch.nn.functional.conv2d(x[1:].double().permute(0, 3, 1, 2), f.double().permute(0, 3, 1, 2), stride=stride,
                                       padding=pad).permute(0, 2, 3, 1)
    # one rounding to half on top of fp32 sums
    assert float((got[1:].double() - exact).norm() / exact.norm()) < 2.0 ** -11
    if bn:      # the library's own choice may cut K
        assert torch.equal(torch.nan_to_num(got, nan=1e4), torch.nan_to_num(ref, nan=1e4))
