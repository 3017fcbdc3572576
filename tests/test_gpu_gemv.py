"""GPU parity: fp16 GEMV (1..8 right-hand sides) through the C ABI vs the CPU oracle."""
import numpy as np
import pytest
import torch

from helix_b200 import datagen, ops
from helix_b200._lib import OP_GEMV_F16
from tests import util

pytestmark = pytest.mark.gpu


def _run(w, x, cfg=None, transposed=False):
    wd, xd = torch.from_numpy(w).cuda(), torch.from_numpy(x).cuda()
    if transposed:
        out = torch.full((w.shape[0], x.shape[0]), float("nan"), dtype=torch.float16, device="cuda")
        ops.run(ops.launch_gemv_f16(wd, xd, out, cfg, out_transposed=True))
        res = out.t()
    else:
        out = torch.full((x.shape[0], w.shape[0]), float("nan"), dtype=torch.float16, device="cuda")
        ops.run(ops.launch_gemv_f16(wd, xd, out, cfg))
        res = out
    torch.cuda.synchronize()
    ops.check_status()
    return res.cpu().numpy()


@pytest.mark.parametrize("rows,K,m", [(4096, 4096, 1), (1000, 1024, 1), (7, 8, 1), (1, 256, 1), (129, 264, 2),
                                      (513, 2048, 3), (300, 4096, 4), (64, 512, 8), (4096, 4096, 8), (33, 40, 5)])
def test_gemv_matches_oracle(oracle, rows, K, m):
    w, x = datagen.c2_gemv(rows, K, m, seed=1)
    got = _run(w, x)
    _, ref32 = oracle.hgemm_naive(x, w)  # [m, rows]
    util.assert_f16_close(got, ref32, f"gemv {rows}x{K} m={m}")


@pytest.mark.parametrize("split", [2, 4, 16])
def test_gemv_split_k_is_deterministic_and_close(oracle, split):
    w, x = datagen.c2_gemv(96, 8192, 2, seed=7)
    cfg = ops.make_cfg(OP_GEMV_F16, tile_m=1, tile_n=2, tile_k=256, split_k=split)
    a = _run(w, x, cfg)
    b = _run(w, x, cfg)
    assert np.array_equal(a.view(np.uint16), b.view(np.uint16))
    _, ref32 = oracle.hgemm_naive(x, w)
    util.assert_f16_close(a, ref32, f"gemv split_k={split}")


def test_gemv_transposed_output_layout(oracle):
    """N <= 8 case of the reference sweep, e.g. (7680, 2, 2560): C[M, N] with the matrix on M."""
    w, x = datagen.c2_gemv(640, 2560, 2, seed=3)
    got = _run(w, x, transposed=True)
    _, ref32 = oracle.hgemm_naive(x, w)
    util.assert_f16_close(got, ref32, "gemv transposed")


def test_gemv_known_answer_ones():
    w = np.ones((50, 1024), np.float16)
    x = np.ones((1, 1024), np.float16)
    assert np.all(_run(w, x) == 1024.0)


def test_gemv_rejects_bad_arguments():
    w = torch.zeros((8, 20), dtype=torch.float16, device="cuda")   # K not a multiple of 8
    x = torch.zeros((1, 20), dtype=torch.float16, device="cuda")
    out = torch.zeros((1, 8), dtype=torch.float16, device="cuda")
    with pytest.raises(Exception) as e:
        ops.run(ops.launch_gemv_f16(w, x, out))
    assert "-2" in str(e.value)
    x9 = torch.zeros((9, 24), dtype=torch.float16, device="cuda")
    w24 = torch.zeros((8, 24), dtype=torch.float16, device="cuda")
    with pytest.raises(Exception):
        ops.run(ops.launch_gemv_f16(w24, x9, torch.zeros((9, 8), dtype=torch.float16, device="cuda")))


@pytest.mark.parametrize("flag", [1, 2])
def test_gemv_launch_ordering_flags_do_not_change_results(oracle, flag):
    """INDEPENDENT (1) and STATIC_A (2) only move the wait for the preceding kernel; a chain of launches on
    distinct outputs must give bit-identical results to fully ordered launches."""
    w, x = datagen.c2_gemv(2048, 4096, 1, seed=5)
    wd, xd = torch.from_numpy(w).cuda(), torch.from_numpy(x).cuda()
    outs = [torch.full((1, 2048), float("nan"), dtype=torch.float16, device="cuda") for _ in range(6)]
    ref = ops.gemv_f16(wd, xd)
    for o in outs:
        l = ops.launch_gemv_f16(wd, xd, o)
        l.flags = flag
        ops.run(l)
    torch.cuda.synchronize()
    for o in outs:
        assert torch.equal(o, ref)
    _, ref32 = oracle.hgemm_naive(x, w)
    util.assert_f16_close(ref.cpu().numpy(), ref32, "gemv flags")


@pytest.mark.parametrize("rows,K,m", [(149, 16392, 1), (2048, 1032, 2), (1185, 2056, 1), (9473, 296, 2), (5, 72, 3),
                                      (4885, 520, 8), (300, 4104, 5), (148, 64, 4), (2100, 504, 7)])
def test_streaming_gemv_at_the_edges_of_its_row_and_k_blocks(oracle, rows, K, m):
    """One row more than SMs, K that leaves part of a chunk, a stretch or a warp's share, blocks of fewer rows than a
    fragment; every right-hand-side count class; plain, static and independent launches bit-identical."""
    w, x = datagen.c2_gemv(rows, K, m, seed=rows + K)
    got = _run(w, x)
    _, ref32 = oracle.hgemm_naive(x, w)
    util.assert_f16_close(got, ref32, f"streaming gemv {rows}x{K} m={m}")
    assert np.array_equal(_run(w, x, transposed=True), got)
    wd, xd = torch.from_numpy(w).cuda(), torch.from_numpy(x).cuda()
    for flag in (1, 2):
        out = torch.full((m, rows), float("nan"), dtype=torch.float16, device="cuda")
        l = ops.launch_gemv_f16(wd, xd, out)
        l.flags = flag
        ops.run(l)
        assert np.array_equal(out.cpu().numpy(), got)


@pytest.mark.parametrize("M,N,K", [(1, 1024, 512), (2, 1025, 520), (3, 1191, 1000), (9, 1024, 520), (16, 5003, 536)])
def test_skinny_gemm_through_the_streaming_kernel(oracle, M, N, K):
    """Up to 16 rows of A: strided operands and output, odd N, a K that is no multiple of 64; unaligned rows keep failing."""
    w, x = datagen.c2_gemv(N, K, M, seed=M + N)
    a = torch.full((M, K + 8), float("nan"), dtype=torch.float16, device="cuda")
    b = torch.full((N, K + 16), float("nan"), dtype=torch.float16, device="cuda")
    out = torch.full((M, N + 3), 7.0, dtype=torch.float16, device="cuda")
    a[:, :K], b[:, :K] = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    ops.run(ops.launch_gemm_f16(a[:, :K], b[:, :K], out[:, :N]))
    torch.cuda.synchronize()
    _, ref32 = oracle.hgemm_naive(x, w)
    util.assert_f16_close(out[:, :N].cpu().numpy(), ref32, f"skinny gemm {M}x{N}x{K}")
    assert torch.all(out[:, N:] == 7.0)
    with pytest.raises(Exception) as e:
        ops.run(ops.launch_gemm_f16(a[:, 1:K - 7], b[:, :K - 8], out[:, :N]))
    assert "-2" in str(e.value)


@pytest.mark.parametrize("rows,K,m,launches", [(64, 65536, 3, 2), (64, 16384, 8, 2), (148, 32768, 4, 2), (512, 8192, 3, 2),
                                               (700, 8192, 3, 1), (296, 16384, 8, 1), (40, 4096, 4, 1)])
def test_few_long_rows_are_cut_over_ctas_where_that_is_faster(oracle, rows, K, m, launches):
    """Three and more right-hand sides: split over CTAs (a kernel and the sum of its slices) or shared by the warps of one."""
    w, x = datagen.c2_gemv(rows, K, m, seed=rows + m)
    wd, xd = torch.from_numpy(w).cuda(), torch.from_numpy(x).cuda()
    out = torch.empty((m, rows), dtype=torch.float16, device="cuda")
    l = ops.launch_gemv_f16(wd, xd, out)
    before = ops.launch_count()
    ops.run(l)
    assert ops.launch_count() - before == launches
    _, ref32 = oracle.hgemm_naive(x, w)
    util.assert_f16_close(out.cpu().numpy(), ref32, f"gemv {rows}x{K} m={m}")
    l.ws, l.ws_bytes = None, 0             # without room for partial sums: one launch
    out.zero_()
    ops.run(l)
    assert ops.launch_count() - before == launches + 1
    util.assert_f16_close(out.cpu().numpy(), ref32, f"gemv {rows}x{K} m={m} without scratch")


@pytest.mark.parametrize("rows,K,m", [(8192, 3072, 1), (8192, 3080, 1), (4096, 2048, 1), (6000, 1536, 1), (256, 256, 3),
                                      (512, 2048, 4), (777, 2048, 8), (2048, 1024, 4), (4096, 4104, 8), (4104, 4096, 3)])
@pytest.mark.parametrize("flag", [0, 1, 2])
def test_gemv_on_both_sides_of_its_kernel_choice(oracle, rows, K, m, flag):
    w, x = datagen.c2_gemv(rows, K, m, seed=rows + K + m)
    wd, xd = torch.from_numpy(w).cuda(), torch.from_numpy(x).cuda()
    _, ref32 = oracle.hgemm_naive(x, w)
    for transposed in (False, True):
        out = torch.full((rows, m) if transposed else (m, rows), float("nan"), dtype=torch.float16, device="cuda")
        l = ops.launch_gemv_f16(wd, xd, out, out_transposed=transposed)
        l.flags = flag
        ops.run(l)
        got = out.cpu().numpy()
        util.assert_f16_close(got.T if transposed else got, ref32, f"gemv {rows}x{K} m={m} flag={flag}")


@pytest.mark.parametrize("M,N,K,launches", [(8, 1024, 10240, 1), (8, 1024, 10248, 2), (16, 2048, 8192, 1), (9, 2048, 8200, 2),
                                            (3, 3552, 10248, 1), (16, 24584, 512, 2), (2, 1024, 32768, 1)])
def test_skinny_gemm_leaves_long_k_of_few_rows_to_the_tiles(oracle, M, N, K, launches):
    w, x = datagen.c2_gemv(N, K, M, seed=M + K)
    a, b = torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda()
    out = torch.empty((M, N), dtype=torch.float16, device="cuda")
    l = ops.launch_gemm_f16(a, b, out)
    before = ops.launch_count()
    ops.run(l)
    assert ops.launch_count() - before == launches
    _, ref32 = oracle.hgemm_fast(x, w)
    util.assert_f16_close(out.cpu().numpy(), ref32, f"skinny {M}x{N}x{K}")
    l.ws, l.ws_bytes = None, 0
    out.zero_()
    ops.run(l)
    assert ops.launch_count() - before == launches + 1
    util.assert_f16_close(out.cpu().numpy(), ref32, f"skinny {M}x{N}x{K} without scratch")
