"""Swapped-operand tiles: the transposed TMA store against the direct 2-byte stores, bit for bit.

Both run the same MMAs; a C whose leading dimension is no multiple of 8 halves takes the direct stores, so the two results
must agree in every bit and nothing beyond the matrix may be written.
"""
import pytest
import torch

from helix_b200 import ops
from helix_b200._lib import OP_CONV_F16, OP_GEMM_F16

pytestmark = pytest.mark.gpu


# N = 136 and 200: the last 128-row block has 8 and 72 rows, so one or both of its 64-row boxes are cut; M: fewer pixels than
# one 64-column box, a cut box, several tiles
@pytest.mark.parametrize("bn", [64, 128, 192, 256])
@pytest.mark.parametrize("m,n,k,batch", [(40, 72, 64, 1), (200, 136, 200, 1), (777, 200, 136, 1), (513, 512, 64, 3),
                                         (25000, 128, 72, 1)])
def test_transposed_store_equals_direct_stores(bn, m, n, k, batch):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(bn + m)
    a = torch.empty((batch, m, k), dtype=torch.float16, device="cuda").normal_(0, 1, generator=gen)
    b = torch.empty((batch, n, k), dtype=torch.float16, device="cuda").normal_(0, 0.1, generator=gen)
    cfg = ops.make_cfg(OP_GEMM_F16, 128, bn, 64, swap_ab=1)
    fast = torch.full((batch, m + 3, n + 8), 7.0, dtype=torch.float16, device="cuda")
    slow = torch.full((batch, m + 3, n + 9), 7.0, dtype=torch.float16, device="cuda")
    for c in (fast, slow):
        ops.run(ops.launch_gemm_f16(a, b, c[:, :m, :n], cfg))
    torch.cuda.synchronize()
    ops.check_status()
    assert torch.equal(fast[:, :m, :n], slow[:, :m, :n])
    for c in (fast, slow):
        assert bool((c[:, m:] == 7.0).all()) and bool((c[:, :m, n:] == 7.0).all())
    ref = torch.matmul(a.double(), b.double().transpose(1, 2))
    # one rounding to half (2^-11 relative) on top of fp32 sums of k products
    assert float((fast[:, :m, :n].double() - ref).norm() / ref.norm()) < 2.0 ** -11


@pytest.mark.parametrize("bn", [64, 192, 256])
@pytest.mark.parametrize("geom", [(3, 128, 14, 14, 72, 3, 1, 1), (2, 96, 26, 26, 200, 5, 1, 2), (5, 64, 9, 11, 136, 3, 2, 1)])
def test_convolution_pixels_on_the_wide_axis(bn, geom):
    nb, c, h, w, ko, r, stride, pad = geom
    gen = torch.Generator(device="cuda")
    gen.manual_seed(bn)
    x = torch.empty((nb, h, w, c), dtype=torch.float16, device="cuda").normal_(0, 1, generator=gen)
    f = torch.empty((ko, r, r, c), dtype=torch.float16, device="cuda").normal_(0, 0.05, generator=gen)
    if nb * h * w * c * 2 < 131072:     # the im2col map is used from 128 KiB on
        x = x.repeat(131072 // (nb * h * w * c * 2) + 1, 1, 1, 1)
    got = ops.conv2d_f16_nhwc(x, f, stride, pad, cfg=ops.make_cfg(OP_CONV_F16, 128, bn, 64, swap_ab=1))
    torch.cuda.synchronize()
    ops.check_status()
    ref = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), f.double().permute(0, 3, 1, 2), stride=stride,
                                     padding=pad).permute(0, 2, 3, 1)
    assert float((got.double() - ref).norm() / ref.norm()) < 2.0 ** -11


@pytest.mark.parametrize("m,n,k,swapped", [(25088, 128, 512, 1), (25000, 136, 264, 0), (6468, 1024, 256, 1), (12544, 128, 512, 0),
                                           (3291, 5648, 232, 1)])
def test_library_choice_of_swapped_tiles(m, n, k, swapped):
    """Both sides of the choice, and the same shapes with a C that only plain stores can write."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(m)
    a = torch.empty((m, k), dtype=torch.float16, device="cuda").normal_(0, 1, generator=gen)
    b = torch.empty((n, k), dtype=torch.float16, device="cuda").normal_(0, 0.1, generator=gen)
    ref = torch.matmul(a.float(), b.float().t())
    for pad in (0, 3):
        c = torch.full((m, n + pad), 7.0, dtype=torch.float16, device="cuda")
        l = ops.launch_gemm_f16(a, b, c[:, :n])
        if ops.device_info().sm_count == 148:
            assert ops.default_config(l).swap_ab == (swapped if pad == 0 else 0)     # the choice follows the real C
        ops.run(l)
        torch.cuda.synchronize()
        ops.check_status()
        assert bool((c[:, n:] == 7.0).all())
        # one rounding to half, and fp32 sums of k products on both sides
        assert float((c[:, :n].float() - ref).norm() / ref.norm()) < 2.0 ** -11
