"""GPU parity: true-fp32 SIMT GEMM through the C ABI vs the CPU oracle (bit-exact vs an fmaf chain)."""
import os

import numpy as np
import pytest
import torch

from helix_b200 import datagen, ops
from helix_b200._lib import OP_GEMM_F32
from tests import util

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")


def _run(a, b, trans_a=False, cfg=None):
    ad, bd = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    M = a.shape[1] if trans_a else a.shape[0]
    out = torch.full((M, b.shape[1]), float("nan"), dtype=torch.float32, device="cuda")
    ops.run(ops.launch_gemm_f32(ad, bd, out, trans_a, cfg))
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("cfg_idx", range(10))
@pytest.mark.parametrize("shape", [(128, 128, 64), (257, 131, 67), (1, 1, 1), (64, 300, 1000), (5, 1024, 16),
                                   (260, 392, 8), (132, 136, 200)])
def test_sgemm_bit_exact_vs_fma_chain(oracle, shape, cfg_idx):
    M, N, K = shape
    a, b = datagen.c1_fp32_gemm(M, N, K, seed=10 + cfg_idx)
    cfg = ops.configs(OP_GEMM_F32)[cfg_idx]
    got = _run(a, b, cfg=cfg)
    want = oracle.sgemm_naive(a, b, fma=True)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (shape, cfg.key())


def test_sgemm_config1_1024_cubed(oracle):
    """FP32 GEMM 1024^3, U[-1,1], seed 0: within 1e-5 of the reference-style loop, bit-equal to the FMA chain."""
    a, b = datagen.c1_fp32_gemm()
    got = _run(a, b)
    assert np.array_equal(got, oracle.sgemm_naive(a, b, fma=True))
    util.assert_f32_close(got, oracle.sgemm_parallel(a, b), "vs parallel template (mul+add)")
    util.assert_f32_close(got, oracle.sgemm_f64acc(a, b), "vs fp64 accumulate")


@pytest.mark.parametrize("trans_a", [False, True])
@pytest.mark.parametrize("cfg_idx", range(5))
def test_sgemm_pipelined_kernel_ragged_sizes_inside_aligned_leading_dimensions(oracle, cfg_idx, trans_a):
    """16-byte-aligned rows but M, N, K that are not multiples of 4: the cp.async ring zero-fills partial
    chunks at the K and N tails and whole chunks outside M; the result stays the fmaf chain, bit for bit."""
    cfg = ops.configs(OP_GEMM_F32)[cfg_idx]
    assert cfg.stages >= 3
    M, N, K = 203, 262, 150 + cfg_idx
    a, b = datagen.c1_fp32_gemm(M, N, K, seed=30 + cfg_idx)
    want = oracle.sgemm_naive(a, b, fma=True)
    big_a = torch.full((K + 3, 208) if trans_a else (M + 1, 160), float("nan"), device="cuda")
    big_b = torch.full((K + 2, 264), float("nan"), device="cuda")
    big_c = torch.full((M + 1, 272), -7.0, device="cuda")
    av = big_a[:K, :M] if trans_a else big_a[:M, :K]
    av.copy_(torch.from_numpy(np.ascontiguousarray(a.T) if trans_a else a))
    big_b[:K, :N].copy_(torch.from_numpy(b))
    ops.run(ops.launch_gemm_f32(av, big_b[:K, :N], big_c[:M, :N], trans_a, cfg))
    torch.cuda.synchronize()
    ops.check_status()
    got = big_c.cpu().numpy()
    assert np.array_equal(got[:M, :N].view(np.uint32), want.view(np.uint32))
    assert np.all(got[M:] == -7.0) and np.all(got[:, N:] == -7.0)       # nothing written outside C


def test_sgemm_transposed_a_layout(oracle):
    a, b = datagen.c1_fp32_gemm(200, 96, 130, seed=4)
    got = _run(np.ascontiguousarray(a.T), b, trans_a=True)
    assert np.array_equal(got, oracle.sgemm_naive(a, b, fma=True))


def test_sgemm_unaligned_leading_dimensions(oracle):
    a, b = datagen.c1_fp32_gemm(70, 33, 45, seed=5)   # N, K not multiples of 4: scalar path
    got = _run(a, b)
    assert np.array_equal(got, oracle.sgemm_naive(a, b, fma=True))


def test_sgemm_golden_vectors_from_reference_loop():
    g = np.load(os.path.join(GOLD, "sgemm_ref.npz"))
    for n in sorted({k[:-2] for k in g.files}):
        got = _run(g[n + "_a"], g[n + "_b"])
        util.assert_f32_close(got, g[n + "_c"], n)
    assert np.all(_run(g["s_one_a"], g["s_one_b"]) == 1000.0)
    assert np.array_equal(_run(g["s_id_a"], g["s_id_b"]), g["s_id_a"])


@pytest.mark.parametrize("trans_a", [False, True])
@pytest.mark.parametrize("cfg_idx", [0, 2, 10, 11, 12])
@pytest.mark.parametrize("shape", [(33, 65, 4), (129, 131, 67), (31, 36, 40), (64, 64, 33), (200, 68, 100)])
def test_sgemm_ring_tiles_take_any_alignment_and_stay_the_fmaf_chain(oracle, shape, cfg_idx, trans_a):
    """The tiles the library chooses from: aligned operands (16-byte copies), unaligned ones (4-byte copies), K that ends
    inside a slab, inside a 16-byte chunk, and before the ring is full."""
    M, N, K = shape
    a, b = datagen.c1_fp32_gemm(M, N, K, seed=50 + cfg_idx)
    cfg = ops.configs(OP_GEMM_F32)[cfg_idx]
    assert cfg.stages >= 3
    got = _run(np.ascontiguousarray(a.T) if trans_a else a, b, trans_a, cfg)
    want = oracle.sgemm_naive(a, b, fma=True)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    # the same matrices behind rows of 16-byte-aligned and of odd lengths
    for pad in (4 - (N % 4), 5):
        big = torch.full((K, N + pad), float("nan"), device="cuda")
        big[:, :N] = torch.from_numpy(b).cuda()
        ad = torch.from_numpy(np.ascontiguousarray(a.T) if trans_a else a).cuda()
        out = torch.empty((M, N), device="cuda")
        ops.run(ops.launch_gemm_f32(ad, big[:, :N], out, trans_a, cfg))
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32)), pad


@pytest.mark.parametrize("cfg_idx", [None, 0, 1, 2, 3, 4, 10, 11, 12])
@pytest.mark.parametrize("M,N,K,lda,ldb", [(70, 36, 21, 24, 36), (33, 130, 50, 53, 132), (129, 67, 7, 8, 68)])
def test_sgemm_ring_with_a_base_of_its_own_alignment(oracle, M, N, K, lda, ldb, cfg_idx):
    """A starts 4 bytes behind a 16-byte boundary while B's rows start on one: columns and k that do not exist are copies of
    nothing whose source must be aligned all the same."""
    a, b = datagen.c1_fp32_gemm(M, N, K, seed=M)
    ad = torch.as_strided(torch.full((M * lda + 4,), float("nan"), device="cuda"), (M, K), (lda, 1), 1)
    bd = torch.full((K, ldb), float("nan"), device="cuda")
    ad.copy_(torch.from_numpy(a))
    bd[:, :N] = torch.from_numpy(b).cuda()
    assert ad.data_ptr() % 16 == 4 and bd.data_ptr() % 16 == 0
    out = torch.empty((M, N), device="cuda")
    cfg = None if cfg_idx is None else ops.configs(OP_GEMM_F32)[cfg_idx]
    ops.run(ops.launch_gemm_f32(ad, bd[:, :N], out, cfg=cfg))
    want = oracle.sgemm_naive(a, b, fma=True)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("cfg_idx", [None, 0, 2, 10, 11, 12])
@pytest.mark.parametrize("M,N,K", [(130, 132, 60), (145, 96, 12), (33, 68, 16), (257, 40, 32)])
def test_sgemm_tiles_that_end_inside_the_rows(oracle, M, N, K, cfg_idx):
    """Tiles that end one or two rows into A, a K of less than a slab, of whole slabs and with a tail: nothing behind A's last
    row is read or written, and the result stays the fmaf chain."""
    a, b = datagen.c1_fp32_gemm(M, N, K, seed=M + K)
    store = torch.full(((M + 128) * K,), float("nan"), device="cuda")
    store[:M * K] = torch.from_numpy(a).cuda().flatten()
    out = torch.full((M + 4, N), -3.0, device="cuda")
    cfg = None if cfg_idx is None else ops.configs(OP_GEMM_F32)[cfg_idx]
    ops.run(ops.launch_gemm_f32(store[:M * K].view(M, K), torch.from_numpy(b).cuda(), out[:M], cfg=cfg))
    got = out.cpu().numpy()
    want = oracle.sgemm_naive(a, b, fma=True)
    assert np.array_equal(got[:M].view(np.uint32), want.view(np.uint32)) and np.all(got[M:] == -3.0)


@pytest.mark.parametrize("tile", [(32, 32, 16, 2), (32, 32, 16, 4), (32, 32, 32, 2), (32, 32, 8, 3)])
@pytest.mark.parametrize("n", [64, 66])
def test_sgemm_refuses_a_32x32_tile_that_is_not_the_rings(tile, n):
    cfg = ops.make_cfg(OP_GEMM_F32, tile_m=tile[0], tile_n=tile[1], tile_k=tile[2], stages=tile[3])
    with pytest.raises(Exception) as e:
        ops.gemm_f32(torch.zeros((64, 64), device="cuda"), torch.zeros((64, n), device="cuda"), cfg=cfg)
    assert "-6" in str(e.value)
