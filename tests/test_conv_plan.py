"""How a convolution's pixels are fetched, as the library plans it, and what the names and the cost model make of it (no GPU needed)."""
import pytest

from helix_b200 import costmodel, harness, ops
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


def _dictionary():
    slab = {256: 0.45e-6, 128: 0.31e-6, 64: 0.27e-6, 32: 0.26e-6, 16: 0.25e-6}
    d = {("sm_count",): 148, ("dram_gbs_per_sm",): 40.0, ("hbm_gbs",): 6000.0}
    for key in costmodel.gemm_keys():
        d[key] = (4e-6, slab[key[2]] if key[3] == 1 else 0.41e-6)
    for bn in (256, 128, 64):
        d[("conv_slab_swap", bn)] = slab[bn]
    return d


def test_the_cost_model_walks_the_channels_that_exist(monkeypatch):
    d = _dictionary()
    walks = harness.conv_block_walks(d, 20, 96, 26, 26, 256, 5, 5, 1, 2)
    assert set(walks.values()) == {25 * 96} and all(k[2] >= 64 and k[3] == 1 and k[5] == 0 for k in walks) and len(walks) == 6
    assert not harness.conv_block_walks(d, 32, 128, 28, 28, 128, 3, 3, 1, 1)
    # 16 channels of a 5 x 5 filter: swapped tiles are open, which a gathering layer's are not
    walks = harness.conv_block_walks(d, 14, 16, 20, 22, 200, 5, 5, 1, 2)
    assert (6, 128, 128, 1, 1, 0) in walks
    M, N, K = 20 * 26 * 26, 256, 25 * 128
    for key in harness.conv_block_walks(d, 20, 96, 26, 26, 256, 5, 5, 1, 2):
        full = costmodel.gemm_time(d, key, M, N, K, 1, "im2col")
        assert costmodel.gemm_time(d, key, M, N, 25 * 96, 1, "im2col") < full
        assert costmodel.cost_model({**{k: v for k, v in d.items() if len(k) == 1 or len(k) == 2}, key: d[key]}, M, N, K, 1, "im2col",
                                    walks={key: 25 * 96}) == key
    seen = {}
    monkeypatch.setattr(harness, "require_gpu", lambda: None)
    monkeypatch.setattr(harness, "time_conv_f16", lambda *a, **k: 1e-5)
    monkeypatch.setattr(harness.costmodel, "cost_model", lambda *a, **k: seen.update(k))
    harness.conv_f16_result(d, 20, 96, 26, 26, 256, 5, 5, 1, 2)
    assert seen["walks"][(4, 128, 256, 1, 1, 0)] == 25 * 96


def test_swapped_whole_tiles_are_open_to_the_cost_model_where_the_library_takes_them():
    d = _dictionary()
    inf = float("inf")
    key, narrow, cut = (4, 128, 256, 1, 1, 0), (8, 128, 64, 1, 1, 0), (4, 128, 256, 1, 1, 1)
    assert costmodel.gemm_time(d, key, 25088, 128, 512) < inf
    assert costmodel.gemm_time(d, narrow, 25088, 128, 512) == inf and costmodel.gemm_time(d, cut, 25088, 128, 512) == inf
    assert costmodel.gemm_time(d, key, 25088, 132, 512) == inf      # rows of C that TMA cannot store
    assert costmodel.gemm_time(d, key, 25088, 64, 512) == inf and costmodel.gemm_time(d, key, 128, 4096, 512) == inf
