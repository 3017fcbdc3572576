"""The deep streaming kernel (long streams, three to sixteen right-hand sides) at the edges of its blocks and pieces of K."""
import pytest
import torch

from helix_b200 import ops
from helix_b200._lib import LAUNCH_INDEPENDENT

pytestmark = pytest.mark.gpu


# rows per CTA of 148: 1-2, 8, 16-17 (the first sizes with shorter pieces of K), 33 (blocks of 64 for nine and more vectors), 38 (one
# block of 64 for up to eight), 49 and 97 (several blocks); K: whole pieces, one element over, short of a whole turn of the warps
@pytest.mark.parametrize("rows,K,m", [(150, 32776, 6), (1100, 4104, 3), (2399, 4608, 16), (2400, 4616, 8), (4884, 4104, 9),
                                      (5600, 4352, 8), (7252, 4128, 3), (14300, 1032, 16), (14300, 1048, 5), (1024, 8192, 11)])
def test_deep_streams(rows, K, m):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows + m)
    w = torch.full((rows, K + 8), float("nan"), dtype=torch.float16, device="cuda")[:, :K]
    x = torch.full((m, K + 16), float("nan"), dtype=torch.float16, device="cuda")[:, :K]
    w.copy_(torch.empty((rows, K), device="cuda").normal_(0, 0.05, generator=gen))
    x.copy_(torch.empty((m, K), device="cuda").normal_(0, 1, generator=gen))
    ref = torch.matmul(x.double(), w.double().t())
    results = []
    for flag, ctas, transposed in ((0, 0, False), (1, 0, False), (2, 0, False), (0, 37, False), (0, 0, True)):
        out = torch.full((rows, m + 1) if transposed else (m, rows + 3), 7.0, dtype=torch.float16, device="cuda")
        if m <= 8:
            y = out[:, :m].t() if transposed else out[:, :rows]
            l = ops.launch_gemv_f16(w, x, out[:, :m] if transposed else y, out_transposed=transposed)
        elif flag == 1 or transposed:
            continue
        else:
            y = out[:, :rows]
            l = ops.launch_gemm_f16(x, w, y)
        if ctas:
            ops.limit_ctas(l, ctas)
        l.flags = flag
        ops.run(l)
        torch.cuda.synchronize()
        # one rounding to half (2^-11) on top of fp32 sums
        assert float((y.double() - ref).norm() / ref.norm()) < 2.0 ** -11
        assert bool((out[:, m:] == 7.0).all()) if transposed else bool((out[:, rows:] == 7.0).all())
        if not ctas or m <= 8:     # a product of more rows may go to the tiles on a share of the machine
            results.append(y.clone())
    assert all(torch.equal(results[0], r) for r in results[1:])


# flagged products of nine and more rows, with the workspace (the library then holds the next launch back) and without it, which is
# the only way to two CTAs on an SM; few rows (J = 4) and more, one block and several per CTA
@pytest.mark.parametrize("rows,K,m", [(2400, 4608, 16), (1024, 8192, 11), (4884, 4112, 9), (14300, 1040, 16), (2400, 4368, 9)])
def test_deep_streams_of_flagged_products(rows, K, m):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows + m)
    w = torch.empty((rows, K), dtype=torch.float16, device="cuda").normal_(0, 0.05, generator=gen)
    x = torch.empty((m, K), dtype=torch.float16, device="cuda").normal_(0, 1, generator=gen)
    ref = torch.matmul(x.double(), w.double().t())
    results = []
    for flag, scratch in ((0, True), (0, False), (LAUNCH_INDEPENDENT, True), (LAUNCH_INDEPENDENT, False)):
        out = torch.full((m, rows + 3), 7.0, dtype=torch.float16, device="cuda")
        l = ops.launch_gemm_f16(x, w, out[:, :rows])
        assert l.ws and l.ws_bytes
        if not scratch:
            l.ws, l.ws_bytes = None, 0
        l.flags = flag
        torch.cuda.synchronize()
        ops.run(l)
        torch.cuda.synchronize()
        # one rounding to half (2^-11) on top of fp32 sums
        assert float((out[:, :rows].double() - ref).norm() / ref.norm()) < 2.0 ** -11
        assert bool((out[:, rows:] == 7.0).all())
        results.append(out)
    assert all(torch.equal(results[0], r) for r in results[1:])
