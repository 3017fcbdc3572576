"""What a flagged launch may start beside: only the launch queued just before it, whatever kernel that one runs."""
import pytest
import torch

from helix_b200 import ops
from helix_b200._lib import LAUNCH_INDEPENDENT, LAUNCH_STATIC_A, OP_CONV_F16, OP_GEMM_F16, OP_GEMV_F16

pytestmark = pytest.mark.gpu
H = torch.float16


def _rand(*shape, dtype=H):
    return torch.randn(shape, device="cuda", dtype=dtype) * 0.1


def _gemv(rows, k, m, cfg=None, flags=0):
    l = ops.launch_gemv_f16(_rand(rows, k), _rand(m, k), torch.empty((m, rows), device="cuda", dtype=H), cfg)
    l.flags = flags
    return l


def _gemm(m, n, k, flags=0, **cfg):
    l = ops.launch_gemm_f16(_rand(m, k), _rand(n, k), torch.empty((m, n), device="cuda", dtype=H),
                            ops.make_cfg(OP_GEMM_F16, **cfg) if cfg else None)
    l.flags = flags
    return l


def _conv(b, hw, c, ko, r, stride, pad, **cfg):
    o = ops.conv_out_hw(hw, hw, r, r, stride, pad)[0]
    return ops.launch_conv2d_f16(_rand(b, hw, hw, c), _rand(ko, r, r, c), torch.empty((b, o, o, ko), device="cuda", dtype=H),
                                 stride, pad, ops.make_cfg(OP_CONV_F16, **cfg) if cfg else None)


MIDDLE = {
    "fp32 GEMV": lambda: ops.launch_gemv_f32(_rand(2000, 1024, dtype=torch.float32), _rand(1, 1024, dtype=torch.float32),
                                             torch.empty((1, 2000), device="cuda")),
    "streaming GEMV": lambda: _gemv(2048, 1024, 1),
    # the library counts these as launches with a workspace: their own flag does not let the next launch past them
    "few long rows, static weights": lambda: _gemv(700, 4096, 1, flags=LAUNCH_STATIC_A),
    "few long rows, independent": lambda: _gemv(700, 4096, 2, flags=LAUNCH_INDEPENDENT),
    "skinny GEMM, independent": lambda: _gemm(8, 2048, 512, flags=LAUNCH_INDEPENDENT),
    "matrix GEMV": lambda: _gemv(2048, 512, 4),
    "plain GEMV": lambda: _gemv(256, 512, 1),
    "split-K GEMV": lambda: _gemv(256, 4096, 1, ops.make_cfg(OP_GEMV_F16, tile_m=1, tile_n=2, tile_k=256, split_k=4)),
    "skinny GEMM": lambda: _gemm(8, 2048, 512),
    "stream-K GEMM with its fix-up": lambda: _gemm(17, 1024, 2048),
    "one-CTA GEMM": lambda: _gemm(128, 128, 64, tile_n=128),
    "pair GEMM": lambda: _gemm(256, 256, 128, tile_n=256, cta_group=2),
    "fp32 GEMM": lambda: ops.launch_gemm_f32(_rand(96, 64, dtype=torch.float32), _rand(64, 96, dtype=torch.float32),
                                             torch.empty((96, 96), device="cuda")),
    "im2col convolution": lambda: _conv(2, 24, 64, 32, 3, 1, 1),
    "gathering convolution": lambda: _conv(1, 12, 24, 32, 3, 1, 1),
    "first layer": lambda: _conv(1, 64, 4, 64, 7, 2, 3),
    "row-pair convolution": lambda: _conv(1, 48, 64, 64, 3, 1, 1, tile_n=64, conv_gather=4),
    "window convolution": lambda: _conv(1, 28, 64, 64, 3, 1, 1, tile_n=64, conv_gather=3),
}


@pytest.mark.parametrize("middle", sorted(MIDDLE))
def test_a_flagged_launch_sees_what_was_queued_before_its_predecessor(middle):
    """A (long, on four SMs, ordered) -> B (short, unrelated buffers, ordered or with a workspace) -> C (flagged, reads
    A's output).  The flag vouches for B alone, so A must be complete when C starts."""
    a, b = _rand(512, 8192), _rand(1024, 8192)
    w = torch.zeros((512, 1024), device="cuda", dtype=H)                 # A's output, C's operand
    cfg = ops.make_cfg(OP_GEMM_F16, tile_n=128)
    cfg.max_ctas = 4
    la = ops.launch_gemm_f16(a, b, w, cfg)
    lb = MIDDLE[middle]()
    outs = [torch.empty((1, 512), device="cuda", dtype=H), torch.empty((1, 512), device="cuda", dtype=H),
            torch.empty((128, 512), device="cuda", dtype=H)]
    lcs = [ops.launch_gemv_f16(w, _rand(1, 1024), outs[0]), ops.launch_gemv_f16(w, _rand(1, 1024), outs[1]),
           ops.launch_gemm_f16(_rand(128, 1024), w, outs[2], ops.make_cfg(OP_GEMM_F16, tile_n=64))]
    for l, flags in zip(lcs, (LAUNCH_STATIC_A, LAUNCH_INDEPENDENT, LAUNCH_INDEPENDENT)):
        l.flags = flags
    ops.run(la)
    torch.cuda.synchronize()
    for lc in lcs:
        ops.run(lc)
        torch.cuda.synchronize()
    want = [o.clone() for o in outs]
    assert all(float(o.abs().max()) > 0 for o in want)
    for trial in range(2):
        for i, lc in enumerate(lcs):
            w.zero_()
            outs[i].zero_()
            torch.cuda.synchronize()
            for l in (la, lb, lc):
                ops.run(l)
            torch.cuda.synchronize()
            assert torch.equal(outs[i], want[i]), (middle, i, trial)
    ops.check_status()
