"""The timeline of a launch is that of the schedule which runs without it."""
import numpy as np
import pytest
import torch

from helix_b200 import ops
from helix_b200._lib import OP_CONV_F16

pytestmark = pytest.mark.gpu
TILES, SLABS = 20, 32      # kTraceTiles and kTraceSlabs of csrc/kernels.h


# 12 blocks of 32 channels in 6 slabs (8 when filled up to 64), 36 of 16 in 9, 4 of 32 in 2, four slabs of 64
@pytest.mark.parametrize("c,ko,r,bn,swap,slabs", [(96, 72, 2, 128, 0, 6), (96, 136, 2, 64, 1, 6), (144, 136, 2, 256, 1, 9), (32, 136, 2, 192, 1, 2),
                                                  (64, 136, 2, 128, 0, 4)])
def test_timeline_of_a_convolution(c, ko, r, bn, swap, slabs):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(c)
    x = torch.empty((8, 33, 33, c), device="cuda", dtype=torch.float16).normal_(0, 1, generator=gen)
    w = torch.empty((ko, r, r, c), device="cuda", dtype=torch.float16).normal_(0, 0.1, generator=gen)
    y = torch.empty((8, 32, 32, ko), device="cuda", dtype=torch.float16)
    l = ops.launch_conv2d_f16(x, w, y, 1, 0, ops.make_cfg(OP_CONV_F16, 128, bn, 64, swap_ab=swap))
    ops.run(l)
    plain = y.clone()
    y.zero_()
    stamps = ops.capture_timeline(l, warm=0)
    assert torch.equal(y, plain)
    rows, cols = (ko, 8192) if swap else (8192, ko)
    tiles = -(-rows // 128) * -(-cols // bn)
    ran = stamps[:, 0] != 0
    ctas = int(ran.sum())
    assert ctas == min(tiles, ops.device_info().sm_count)
    consumed = (stamps[ran, 8 + 6 * TILES + SLABS:8 + 6 * TILES + 2 * SLABS] != 0).sum(axis=1)
    assert (consumed == np.array([-(-(tiles - i) // ctas) * slabs for i in range(ctas)])).all()
