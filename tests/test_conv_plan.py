"""How a convolution's pixels are fetched, as the library plans it, and the name of the kernel that does it (no GPU needed)."""
import pytest

from helix_b200 import ops
from helix_b200._lib import HelixError, OP_CONV_F16, OP_GEMM_F16


def _launch(geom, y=0, **cfg):
    l = ops.Launch()
    l.op, l.c = OP_CONV_F16, y
    for i, v in enumerate(geom):
        l.conv[i] = v
    if cfg:
        l.cfg = ops.make_cfg(OP_CONV_F16, **cfg)
    return l


# N H W C KO R S stride pad
C96 = (20, 26, 26, 96, 256, 5, 5, 1, 2)
C32 = (32, 56, 56, 32, 64, 3, 3, 1, 1)
C144 = (16, 26, 26, 144, 136, 3, 3, 1, 1)
C160 = (32, 14, 14, 160, 256, 3, 3, 1, 1)


@pytest.mark.parametrize("launch,channels", [
    (_launch(C96), 32), (_launch(C96, tile_n=256, swap_ab=1), 32), (_launch(C96, y=4098), 64), (_launch(C96, tile_n=128, stream_k=1), 64),
    (_launch(C96, tile_n=128, split_k=2), 64), (_launch(C96, tile_n=32), 64), (_launch(C96, tile_n=128, probe=1), 64),
    (_launch(C96, tile_n=128, conv_gather=1), 0), (_launch(C96, tile_n=64), 32), (_launch(C160, tile_n=64), 64),
    (_launch(C160, tile_n=128), 32), (_launch(C144, tile_n=128), 16), (_launch(C32, tile_n=128), 32), (_launch(C32, y=4098, tile_n=128), 0),
    (_launch(C32, tile_n=128, stream_k=1), 0), (_launch(C32, tile_n=128, swap_ab=1), 0), (_launch((1, 8, 8, 32, 64, 3, 3, 1, 1)), 0),
    (_launch((32, 28, 28, 128, 128, 3, 3, 1, 1)), 64)])
def test_channels_per_pixel_and_the_kernels_name(launch, channels):
    assert ops.conv_pixel_channels(launch) == channels
    assert ops.kernel_name(launch).endswith(",%d>" % (channels == 0))


def test_convolutions_without_such_a_fetch():
    for geom, cfg, name in (((32, 28, 28, 128, 128, 1, 1, 1, 0), {}, "gemm_f16_tc"), ((8, 224, 224, 4, 64, 7, 7, 2, 3), {}, "conv_f16_stem_kernel"),
                            ((32, 56, 56, 64, 64, 3, 3, 1, 1), {"conv_gather": 4}, "conv_f16_rows_kernel"),
                            ((32, 28, 28, 128, 128, 3, 3, 1, 1), {"tile_n": 64, "conv_gather": 3}, "conv_f16_win_kernel")):
        l = _launch(geom, **cfg)
        assert ops.kernel_name(l).startswith(name)
        with pytest.raises(HelixError):
            ops.conv_pixel_channels(l)
    l = ops.Launch()
    l.op = OP_GEMM_F16
    with pytest.raises(HelixError):
        ops.conv_pixel_channels(l)
