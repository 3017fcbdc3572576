// True-fp32 SIMT GEMM: C[M,N] = A * B with FFMA only (no TF32, no tensor cores).
//
// Counterpart of the reference's mySgemmCPAsyncTemplate (src_template/Ampere_FP32/sgemm.cu
// :97-350).  B is K x N row-major; A is M x K row-major (the x86 template's layout,
// scripts/x86_CPU/profile_x86_CPU.py:27-29) or K x M when trans_a is set (what the reference
// kernel is handed, sgemm.cu:138).  Every output element accumulates k = 0, 1, 2, ... in one
// fp32 register with one fused multiply-add per step, so the result is bit-identical to an
// fmaf() chain on the host.
//
// CTA tile BM x BN x BK, (BM/TM)*(BN/TN) threads, each thread a TM x TN register block split
// into 4-wide quads that are strided across the tile (conflict-free float4 reads from shared
// memory).  A is staged K-major ([BK][BM]) so both operands are read as float4 along the
// output dimension.  Global loads of slab k+1 are issued into registers before the FFMA loop
// of slab k and written to the other shared buffer afterwards (one __syncthreads per slab).
//
// That is the register-staged kernel below, which remains for explicit two-buffer configurations and for rows 2^23 or more
// floats apart; everything else runs the cp.async ring kernel of sgemm_f32_ring.cuh.
#include "sgemm_f32_ring.cuh"

namespace helix {

template <int BM, int BN, int BK, int TM, int TN>
struct SgemmTraits {
  static constexpr int kThreadsM = BM / TM;
  static constexpr int kThreadsN = BN / TN;
  static constexpr int kThreads = kThreadsM * kThreadsN;
  static constexpr int kAElems = BM * BK / kThreads;  // floats of A per thread per slab
  static constexpr int kBElems = BN * BK / kThreads;
  static_assert(TM % 4 == 0 && TN % 4 == 0, "register block is made of 4-wide quads");
  static_assert(kAElems % 4 == 0 && kBElems % 4 == 0, "whole float4s per thread");
  static_assert(kThreadsM % 4 == 0 && kThreadsN % 8 == 0, "a warp covers 4 x 8 threads of the grid");
};

template <int BM, int BN, int BK, int TM, int TN, bool TRANS_A, bool VEC>
__global__ void __launch_bounds__(SgemmTraits<BM, BN, BK, TM, TN>::kThreads)
sgemm_f32_kernel(const float* __restrict__ A, int64_t lda, const float* __restrict__ B, int64_t ldb,
                 float* __restrict__ C, int64_t ldc, int M, int N, int K) {
  using T = SgemmTraits<BM, BN, BK, TM, TN>;
  constexpr int NT = T::kThreads;
  constexpr int A4 = T::kAElems / 4;
  constexpr int B4 = T::kBElems / 4;
  __shared__ __align__(16) float sA[2][BK][BM + 4];
  __shared__ __align__(16) float sB[2][BK][BN + 4];

  // a warp covers 4 x 8 threads of the kThreadsM x kThreadsN grid, a half-warp 4 x 4: a 128-bit shared
  // load is served half-warp by half-warp, and 4 distinct float4 per half cost one pass instead of two
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  constexpr int kWarpsN = T::kThreadsN / 8;
  const int tn = (warp % kWarpsN) * 8 + (lane & 3) + 4 * (lane >> 4);
  const int tm = (warp / kWarpsN) * 4 + ((lane >> 2) & 3);
  const int m0 = blockIdx.y * BM;
  const int n0 = blockIdx.x * BN;

  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

  float4 ra[A4], rb[B4];
  auto a_swz = [](int kk) { return ((kk >> 2) & 3) << 2; };   // column XOR of sA row kk (multiple of 4)

  // ---- global -> registers for slab starting at k0 (zero fill outside the matrix)
  auto load_global = [&](int k0) {
#pragma unroll
    for (int v = 0; v < A4; ++v) {
      const int f = (v * NT + tid);  // float4 index inside the slab
      float4 val = make_float4(0.f, 0.f, 0.f, 0.f);
      if (TRANS_A) {
        // A is K x M: a float4 runs along M
        const int kk = f / (BM / 4), mm = (f % (BM / 4)) * 4;
        const int gk = k0 + kk, gm = m0 + mm;
        if (gk < K) {
          const float* p = A + (int64_t)gk * lda + gm;
          if (VEC && gm + 3 < M) val = *reinterpret_cast<const float4*>(p);
          else {
            if (gm + 0 < M) val.x = p[0];
            if (gm + 1 < M) val.y = p[1];
            if (gm + 2 < M) val.z = p[2];
            if (gm + 3 < M) val.w = p[3];
          }
        }
      } else {
        // A is M x K: a float4 runs along K
        const int mm = f / (BK / 4), kk = (f % (BK / 4)) * 4;
        const int gk = k0 + kk, gm = m0 + mm;
        if (gm < M) {
          const float* p = A + (int64_t)gm * lda + gk;
          if (VEC && gk + 3 < K) val = *reinterpret_cast<const float4*>(p);
          else {
            if (gk + 0 < K) val.x = p[0];
            if (gk + 1 < K) val.y = p[1];
            if (gk + 2 < K) val.z = p[2];
            if (gk + 3 < K) val.w = p[3];
          }
        }
      }
      ra[v] = val;
    }
#pragma unroll
    for (int v = 0; v < B4; ++v) {
      const int f = (v * NT + tid);
      const int kk = f / (BN / 4), nn = (f % (BN / 4)) * 4;
      const int gk = k0 + kk, gn = n0 + nn;
      float4 val = make_float4(0.f, 0.f, 0.f, 0.f);
      if (gk < K) {
        const float* p = B + (int64_t)gk * ldb + gn;
        if (VEC && gn + 3 < N) val = *reinterpret_cast<const float4*>(p);
        else {
          if (gn + 0 < N) val.x = p[0];
          if (gn + 1 < N) val.y = p[1];
          if (gn + 2 < N) val.z = p[2];
          if (gn + 3 < N) val.w = p[3];
        }
      }
      rb[v] = val;
    }
  };
  // ---- registers -> shared buffer `buf`
  auto store_shared = [&](int buf) {
#pragma unroll
    for (int v = 0; v < A4; ++v) {
      const int f = (v * NT + tid);
      if (TRANS_A) {
        const int kk = f / (BM / 4), mm = (f % (BM / 4)) * 4;
        *reinterpret_cast<float4*>(&sA[buf][kk][mm ^ a_swz(kk)]) = ra[v];
      } else {
        // the four k values of a float4 go to four rows; rows kk, kk+4, kk+8, kk+12 of one warp's
        // stores would share banks pairwise, so the column is XOR-ed with a multiple of 4 that
        // depends on kk / 4 (whole float4 groups move, the later float4 reads stay aligned)
        const int mm = f / (BK / 4), kk = (f % (BK / 4)) * 4;
        const int col = mm ^ a_swz(kk);
        sA[buf][kk + 0][col] = ra[v].x;
        sA[buf][kk + 1][col] = ra[v].y;
        sA[buf][kk + 2][col] = ra[v].z;
        sA[buf][kk + 3][col] = ra[v].w;
      }
    }
#pragma unroll
    for (int v = 0; v < B4; ++v) {
      const int f = (v * NT + tid);
      const int kk = f / (BN / 4), nn = (f % (BN / 4)) * 4;
      *reinterpret_cast<float4*>(&sB[buf][kk][nn]) = rb[v];
    }
  };

  const int num_slabs = (K + BK - 1) / BK;
  if (num_slabs > 0) {
    load_global(0);
    store_shared(0);
  }
  __syncthreads();

  for (int s = 0; s < num_slabs; ++s) {
    const int buf = s & 1;
    if (s + 1 < num_slabs) load_global((s + 1) * BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float av[TM], bv[TN];
#pragma unroll
      for (int q = 0; q < TM / 4; ++q) {
        const float4 t = *reinterpret_cast<const float4*>(&sA[buf][kk][((q * T::kThreadsM + tm) * 4) ^ a_swz(kk)]);
        av[q * 4 + 0] = t.x; av[q * 4 + 1] = t.y; av[q * 4 + 2] = t.z; av[q * 4 + 3] = t.w;
      }
#pragma unroll
      for (int q = 0; q < TN / 4; ++q) {
        const float4 t = *reinterpret_cast<const float4*>(&sB[buf][kk][(q * T::kThreadsN + tn) * 4]);
        bv[q * 4 + 0] = t.x; bv[q * 4 + 1] = t.y; bv[q * 4 + 2] = t.z; bv[q * 4 + 3] = t.w;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    if (s + 1 < num_slabs) store_shared(buf ^ 1);
    __syncthreads();
  }

  // ---- epilogue: quads are strided across the tile
#pragma unroll
  for (int qi = 0; qi < TM / 4; ++qi)
#pragma unroll
    for (int ii = 0; ii < 4; ++ii) {
      const int gm = m0 + (qi * T::kThreadsM + tm) * 4 + ii;
      if (gm >= M) continue;
#pragma unroll
      for (int qj = 0; qj < TN / 4; ++qj) {
        const int gn = n0 + (qj * T::kThreadsN + tn) * 4;
        float* p = C + (int64_t)gm * ldc + gn;
        const float* a = &acc[qi * 4 + ii][qj * 4];
        if (VEC && gn + 3 < N) *reinterpret_cast<float4*>(p) = make_float4(a[0], a[1], a[2], a[3]);
        else {
          if (gn + 0 < N) p[0] = a[0];
          if (gn + 1 < N) p[1] = a[1];
          if (gn + 2 < N) p[2] = a[2];
          if (gn + 3 < N) p[3] = a[3];
        }
      }
    }
}

// stages == 2: register-staged double buffer (any alignment); stages >= 3: the cp.async ring kernel.  Of the ring
// configurations, those the library itself chooses from (kSgemmTiles) take any alignment, the others need 16-byte-aligned
// operands and fall back to the register-staged kernel of the same tile.
struct SgemmCfg { int bm, bn, bk, tm, tn, stages; };
static const SgemmCfg kSgemmCfgs[] = {
    {128, 128, 16, 8, 8, 4}, {128, 128, 32, 8, 8, 3}, {128, 64, 16, 8, 8, 4}, {128, 64, 32, 8, 8, 3},
    {64, 128, 16, 8, 8, 4},
    {128, 128, 16, 8, 8, 2}, {128, 64, 16, 8, 4, 2}, {64, 128, 16, 4, 8, 2}, {64, 64, 16, 4, 4, 2}, {32, 64, 16, 4, 4, 2},
    {64, 64, 16, 4, 8, 4}, {32, 64, 16, 4, 4, 6}, {32, 32, 32, 2, 4, 4},
};
constexpr int kNumSgemmCfgs = sizeof(kSgemmCfgs) / sizeof(kSgemmCfgs[0]);

int sgemm_f32_num_configs() { return kNumSgemmCfgs; }
void sgemm_f32_get_config(int idx, helix_cfg_t* out) {
  *out = helix_cfg_t{};
  out->op = HELIX_OP_GEMM_F32;
  out->tile_m = kSgemmCfgs[idx].bm;
  out->tile_n = kSgemmCfgs[idx].bn;
  out->tile_k = kSgemmCfgs[idx].bk;
  out->thread_m = kSgemmCfgs[idx].tm;
  out->thread_n = kSgemmCfgs[idx].tn;
  out->stages = kSgemmCfgs[idx].stages;
  out->cta_group = 1;
  out->split_k = 1;
}

// Time of one step of k on the busiest SM: `alone` cycles for a CTA that has the SM to itself (its chain of fragment
// loads and multiply-adds), at least `busy` cycles per CTA when several share it.  Measured at 1.92 GHz on 1024^3, 2048^3,
// 4096^3 and on grids of less than one tile per SM; a 128 x 64 tile would need 64 cycles for its multiply-adds alone: with
// one warp per scheduler the two cycles of every packed instruction and the fragment loads between them add up, with many
// the shared-memory passes of the fragment loads (88 % of the pipe at 64 x 64) come close to the FMA pipe's time.
struct SgemmTile { int cfg, ctas_per_sm; double alone, busy; };
static const SgemmTile kSgemmTiles[] = {
    {0, 2, 187, 165}, {2, 3, 106, 82}, {10, 4, 62, 46}, {11, 4, 41, 25}, {12, 4, 20.5, 15},
};

// The configuration with the least work on the busiest SM; a wave holds ctas_per_sm tiles on every SM.  (K counts where a slab
// is longer than K: 145 x 2412 x 12 on 32 x 32 tiles with slabs of 32 took 3.1 us, 2.8 on 32 x 64 ones with slabs of 16.)
void sgemm_f32_default_config(int M, int N, int K, int sm_count, helix_cfg_t* out) {
  int pick = 0;
  double best = 1e300;
  for (const SgemmTile& tl : kSgemmTiles) {
    const SgemmCfg& c = kSgemmCfgs[tl.cfg];
    const int64_t tiles = (int64_t)((M + c.bm - 1) / c.bm) * ((N + c.bn - 1) / c.bn);
    const int64_t slots = (int64_t)sm_count * tl.ctas_per_sm;
    const int64_t full = (tiles - 1) / slots;                              // full waves before the last one
    const int64_t last = (tiles - full * slots + sm_count - 1) / sm_count; // tiles of the last wave on the busiest SM
    const double steps = K > 0 ? (double)(((int64_t)K + c.bk - 1) / c.bk * c.bk) : 1.0;   // whole slabs of k are walked
    const double t = steps * (full * std::max(tl.alone, tl.ctas_per_sm * tl.busy) + std::max(tl.alone, last * tl.busy));
    if (t < best) { best = t; pick = tl.cfg; }
  }
  sgemm_f32_get_config(pick, out);
}

template <int BM, int BN, int BK, int TM, int TN>
static void launch_sgemm(const float* A, int64_t lda, bool trans_a, const float* B, int64_t ldb, float* C,
                         int64_t ldc, int M, int N, int K, bool vec, cudaStream_t stream) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  constexpr int NT = SgemmTraits<BM, BN, BK, TM, TN>::kThreads;
  if (trans_a) {
    if (vec) sgemm_f32_kernel<BM, BN, BK, TM, TN, true, true><<<grid, NT, 0, stream>>>(A, lda, B, ldb, C, ldc, M, N, K);
    else sgemm_f32_kernel<BM, BN, BK, TM, TN, true, false><<<grid, NT, 0, stream>>>(A, lda, B, ldb, C, ldc, M, N, K);
  } else {
    if (vec) sgemm_f32_kernel<BM, BN, BK, TM, TN, false, true><<<grid, NT, 0, stream>>>(A, lda, B, ldb, C, ldc, M, N, K);
    else sgemm_f32_kernel<BM, BN, BK, TM, TN, false, false><<<grid, NT, 0, stream>>>(A, lda, B, ldb, C, ldc, M, N, K);
  }
}

template <typename T>
static int launch_vec(const RingParams& p, bool trans_a, cudaStream_t stream) {
  return trans_a ? launch_ring<T, kCols16, kCols16>(p, stream) : launch_ring<T, kRows4, kCols16>(p, stream);
}
template <typename T>
static int launch_any(const RingParams& p, bool trans_a, bool a16, bool b16, cudaStream_t stream) {
  if (trans_a) return a16 && b16 ? launch_ring<T, kCols16, kCols16>(p, stream) : launch_ring<T, kCols4, kCols4>(p, stream);
  // 128 x 128: two fragments of four k are more registers than two CTAs per SM leave, so A stays K-major there
  constexpr int kWide = T::BM * T::BN > 8192 ? kRows4 : kRows16;
  if (b16) return a16 ? launch_ring<T, kWide, kCols16>(p, stream) : launch_ring<T, kRows4, kCols16>(p, stream);
  return launch_ring<T, kRows4, kCols4>(p, stream);
}

int sgemm_f32_launch(const helix_cfg_t* cfg, const float* A, int64_t lda, int trans_a, const float* B, int64_t ldb,
                     float* C, int64_t ldc, int M, int N, int K, int sm_count, cudaStream_t stream,
                     int64_t* launches) {
  if (!A || !B || !C || M <= 0 || N <= 0 || K < 0) return HELIX_ERR_INVALID;
  if (lda == 0) lda = trans_a ? M : K;
  if (ldb == 0) ldb = N;
  if (ldc == 0) ldc = N;
  const bool vec = ((lda & 3) == 0) && ((ldb & 3) == 0) && ((ldc & 3) == 0) &&
                   ((reinterpret_cast<uintptr_t>(A) & 15) == 0) && ((reinterpret_cast<uintptr_t>(B) & 15) == 0) &&
                   ((reinterpret_cast<uintptr_t>(C) & 15) == 0);
  int bm, bn, bk, stages;
  if (cfg && cfg->tile_m != 0) {
    bm = cfg->tile_m;
    bn = cfg->tile_n;
    bk = cfg->tile_k ? cfg->tile_k : 16;
    stages = cfg->stages ? cfg->stages : 2;
  } else {
    helix_cfg_t def{};
    sgemm_f32_default_config(M, N, K, sm_count, &def);
    bm = def.tile_m;
    bn = def.tile_n;
    bk = def.tile_k;
    stages = def.stages;
  }
  const bool ta = trans_a != 0;
  if (bm == 32 && bn == 32 && !(stages >= 3 && bk == 32)) return HELIX_ERR_UNSUPPORTED;   // a ring tile only
  // the ring kernel addresses the rows of a tile with 32-bit offsets
  if (stages >= 3 && lda < (1 << 23) && ldb < (1 << 23)) {
    RingParams p{};
    p.A = A; p.B = B; p.C = C;
    p.lda = lda; p.ldb = ldb; p.ldc = ldc;
    p.M = M; p.N = N; p.K = K;
    p.vec_c = (ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
    const bool a16 = (lda & 3) == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
    const bool b16 = (ldb & 3) == 0 && (reinterpret_cast<uintptr_t>(B) & 15) == 0;
    p.none = b16 ? B : A;      // columns of B go by 16 bytes with b16, rows and columns of A only where B's do too
    int rc = HELIX_ERR_UNSUPPORTED;
    if (bm == 128 && bn == 128 && bk == 16) rc = launch_any<RingTile128x128>(p, ta, a16, b16, stream);
    else if (bm == 128 && bn == 64 && bk == 16) rc = launch_any<RingTile128x64>(p, ta, a16, b16, stream);
    else if (bm == 64 && bn == 64 && bk == 16) rc = launch_any<RingTile64x64>(p, ta, a16, b16, stream);
    else if (bm == 32 && bn == 64 && bk == 16) rc = launch_any<RingTile32x64>(p, ta, a16, b16, stream);
    else if (bm == 32 && bn == 32 && bk == 32) rc = launch_any<RingTile32x32>(p, ta, a16, b16, stream);
    else if (b16 && (!ta || a16)) {
      if (bm == 128 && bn == 128 && bk == 8 && stages == 4) rc = launch_vec<RingTile<128, 128, 8, 8, 8, 4, 2>>(p, ta, stream);
      else if (bm == 128 && bn == 128 && bk == 8) rc = launch_vec<RingTile<128, 128, 8, 8, 8, 3, 2>>(p, ta, stream);
      else if (bm == 128 && bn == 128 && bk == 32) rc = launch_vec<RingTile<128, 128, 32, 8, 8, 3, 2>>(p, ta, stream);
      else if (bm == 128 && bn == 64 && bk == 32) rc = launch_vec<RingTile<128, 64, 32, 8, 8, 3, 2>>(p, ta, stream);
      else if (bm == 64 && bn == 128 && bk == 16) rc = launch_vec<RingTile<64, 128, 16, 8, 8, 4, 3>>(p, ta, stream);
    }
    if (rc == HELIX_OK) ++*launches;
    if (rc != HELIX_ERR_UNSUPPORTED || vec) return rc;
  }
  if (bm == 32 && bn == 32) bn = 64;   // the ring's smallest tile, rows too far apart for it
  if (bm == 128 && bn == 128) launch_sgemm<128, 128, 16, 8, 8>(A, lda, ta, B, ldb, C, ldc, M, N, K, vec, stream);
  else if (bm == 128 && bn == 64) launch_sgemm<128, 64, 16, 8, 4>(A, lda, ta, B, ldb, C, ldc, M, N, K, vec, stream);
  else if (bm == 64 && bn == 128) launch_sgemm<64, 128, 16, 4, 8>(A, lda, ta, B, ldb, C, ldc, M, N, K, vec, stream);
  else if (bm == 64 && bn == 64) launch_sgemm<64, 64, 16, 4, 4>(A, lda, ta, B, ldb, C, ldc, M, N, K, vec, stream);
  else if (bm == 32 && bn == 64) launch_sgemm<32, 64, 16, 4, 4>(A, lda, ta, B, ldb, C, ldc, M, N, K, vec, stream);
  else return HELIX_ERR_UNSUPPORTED;
  ++*launches;
  return cudaGetLastError() == cudaSuccess ? HELIX_OK : HELIX_ERR_CUDA;
}

}  // namespace helix
