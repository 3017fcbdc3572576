"""An ordered launch behind a kernel that runs for longer than the bounded waits allow: nothing is wrong, so nothing may time out.

The predecessor is a flagged product on two SMs, which lets its successor in at once and leaves it room, so that the successor's
warps are all resident while it runs.
"""
import pytest
import torch

from helix_b200 import ops
from helix_b200._lib import LAUNCH_INDEPENDENT, OP_CONV_F16, OP_GEMM_F16

pytestmark = pytest.mark.gpu
H = torch.float16
LIMIT_MS = 2000.0      # kWaitLimitNs of csrc/common.cuh


def _rand(*shape):
    return torch.randn(shape, device="cuda", dtype=H) * 0.1


def _gemm(m, n, k, **cfg):
    l = ops.launch_gemm_f16(_rand(m, k), _rand(n, k), torch.zeros((m, n), device="cuda", dtype=H),
                            ops.make_cfg(OP_GEMM_F16, **cfg) if cfg else None)
    return l, l._refs[2]


def _conv(b, hw, c, ko, **cfg):
    l = ops.launch_conv2d_f16(_rand(b, hw, hw, c), _rand(ko, 3, 3, c), torch.zeros((b, hw, hw, ko), device="cuda", dtype=H), 1, 1,
                              ops.make_cfg(OP_CONV_F16, **cfg) if cfg else None)
    return l, l._refs[2]


# one issuing warp, two of them, stream-K with its fix-up, CTA pairs with two issuers and with a watcher, warps that gather
SUCCESSORS = {
    "whole tiles": lambda: _gemm(512, 512, 512, tile_n=128),
    "two issuing warps": lambda: _gemm(512, 512, 512, tile_n=128, probe=0x80),
    "stream-K": lambda: _gemm(24, 1024, 2048),
    "pairs": lambda: _gemm(512, 512, 512, tile_n=256, cta_group=2),
    "pairs, one issuer": lambda: _gemm(512, 512, 512, tile_n=128, cta_group=2, probe=0x200),
    "gathering convolution": lambda: _conv(4, 14, 24, 64),
}


@pytest.fixture(scope="module")
def long_launch():
    """A launch of some 2.6 s, made by the length of its K."""
    def make(k):
        cfg = ops.make_cfg(OP_GEMM_F16, tile_n=16)
        cfg.max_ctas = 2
        l = ops.launch_gemm_f16(torch.zeros((16384, k), device="cuda", dtype=H), torch.zeros((16384, k), device="cuda", dtype=H),
                                torch.empty((16384, 16384), device="cuda", dtype=H), cfg)
        l.flags = LAUNCH_INDEPENDENT
        return l

    def ms(l):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record()
        ops.run(l)
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1)

    short, twice = make(512), make(1024)
    ms(short)
    return make(int(512 * 1.3 * LIMIT_MS / (ms(twice) - ms(short))) // 64 * 64)


@pytest.mark.parametrize("name", list(SUCCESSORS))
def test_the_clock_of_a_wait_does_not_run_while_the_predecessor_does(long_launch, name):
    l, out = SUCCESSORS[name]()
    ops.run(l)
    torch.cuda.synchronize()
    ops.check_status()
    ref = out.clone()
    out.zero_()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    ops.run(long_launch)
    ops.run(l)
    e1.record()
    torch.cuda.synchronize()
    ops.check_status()
    assert e0.elapsed_time(e1) > 1.05 * LIMIT_MS
    assert torch.equal(out, ref)
