"""Weights that the predecessor writes: an ordered launch asks the L2 for them ahead of its wait and must read what was written."""
import pytest
import torch

from helix_b200 import ops
from helix_b200._lib import OP_GEMM_F16

pytestmark = pytest.mark.gpu


# streaming GEMV, deep GEMV (blocks of 32 rows and, with few rows, of J = 4), skinny product, swapped tiles of 32 columns
SIZES = [(2048, 2048, 1), (3000, 4104, 2), (2560, 4096, 8), (1024, 8192, 3), (4096, 4096, 16), (2048, 2056, 13), (2048, 2048, 24),
         (1100, 4096, 32)]


@pytest.mark.parametrize("dtype,rows,k,m", [(torch.float16, *s) for s in SIZES] + [(torch.float32, *s) for s in SIZES if s[2] <= 8])
def test_weights_written_by_the_predecessor(dtype, rows, k, m):
    w = torch.zeros((rows, k), device="cuda", dtype=dtype)
    x = torch.randn((m, k), device="cuda", dtype=dtype)
    out = torch.empty((m, rows), device="cuda", dtype=dtype)
    if dtype == torch.float16:
        lb = ops.launch_gemv_f16(w, x, out) if m <= 8 else ops.launch_gemm_f16(x, w, out)
    else:
        lb = ops.launch_gemv_f32(w, x, out)
    for _ in range(3):
        a, b = (torch.randn((n, 64), device="cuda", dtype=dtype) * 0.1 for n in (rows, k))
        if dtype == torch.float16:
            cfg = ops.make_cfg(OP_GEMM_F16, tile_n=128)
            cfg.max_ctas = 8                                # long beside what it is followed by
            la = ops.launch_gemm_f16(a, b, w, cfg)
        else:
            la = ops.launch_gemm_f32(a, b.t().contiguous(), w)
        torch.cuda.synchronize()
        ops.run(la)
        ops.run(lb)                                         # queued while la runs
        torch.cuda.synchronize()
        got = out.clone()
        ops.run(lb)
        torch.cuda.synchronize()
        assert torch.equal(got, out) and torch.isfinite(out).all()
        ref = x.double() @ w.double().t()
        assert (out.double() - ref).norm() <= 1e-3 * ref.norm()     # fp16 rounding is 2^-11 at most
