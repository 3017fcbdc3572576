// Tile kernel of the true-fp32 GEMM and convolution: C[M,N] = A * B with fused multiply-adds only.
//
// Every output element accumulates k = 0, 1, 2, ... in one fp32 register, so the result is bit-identical to an fmaf()
// chain on the host whatever the tile.  What bounds it is the FMA pipe, and before that the issue slots: one scalar FFMA per
// warp and clock is the whole fp32 rate, which leaves no slot for fragment loads and address work (52.5 of 74.4 TFLOP/s
// at 4096^3).  fma.rn.f32x2 does two of them, each rounded as usual, in one instruction of twice the pipe time: a thread
// keeps its accumulators as pairs of neighbouring columns, B fragments come from shared memory as pairs, A values are
// doubled in registers.  Both operands are staged K-major ([BK][rows + 4]) by cp.async through a ring of STAGES slabs; the
// fragments of step k + 1 are fetched while step k computes, across slab borders too (the barrier of the next slab
// comes before the last step of the current one).
//
// Operands reach the ring in one of these ways: columns along k (K x N B; K x M A) by 16-byte copies, or 4-byte ones
// where the operand is not 16-byte aligned; rows along k (the filters of a convolution; an unaligned M x K A) transposed by
// 4-byte copies; an aligned M x K A by 16-byte copies into [rows][BK] as it is -- a thread then fetches four k of a row with
// one shared load, the same number of loads as K-major, but a transposing copy instruction takes four shared-memory
// wavefronts for 32 elements where a 16-byte one takes four for 128 (3 x 3, 128 -> 128
// channels, 28 x 28 x 32, implicit: 180 -> 172 us; 1500 x 800 x 640: 50 -> 40 us); and the
// windows of an NHWC image, a row of the column matrix gathered on the fly, in either of the two row layouts.
#pragma once
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace helix {

enum RingSource { kRows4, kCols16, kCols4, kWindow4, kRows16, kWindow16 };
__host__ __device__ constexpr bool ring_row_major(int src) { return src == kRows16 || src == kWindow16; }

struct RingParams {
  const float* A;
  const float* B;
  float* C;
  int64_t lda, ldb, ldc;
  // Source of copies of nothing (an absent row, column or k): these too need a source aligned to their size.  A or B, one
  // that starts on 16 bytes where a loader copies 16.
  const float* none;
  int M, N, K, tiles_n;
  int vec_c;                         // rows of C may be written 16 bytes at a time
  // kWindow4, kWindow16: A is x[N][H][W][C]
  int H, W, Cin, S, stride, pad, R;
  FastDiv fd_c, fd_s, fd_wo, fd_ho;
};

template <int BM_, int BN_, int BK_, int TM_, int TN_, int STAGES_, int MIN_CTAS_>
struct RingTile {
  static constexpr int BM = BM_, BN = BN_, BK = BK_, TM = TM_, TN = TN_, STAGES = STAGES_, MIN_CTAS = MIN_CTAS_;
  static constexpr int kThreadsM = BM / TM, kThreadsN = BN / TN, kThreads = kThreadsM * kThreadsN;
  static constexpr int QM = TM < 4 ? TM : 4;                    // consecutive rows of a thread
  static constexpr int kAPitch = BM + 4, kBPitch = BN + 4;      // floats per k
  static constexpr int kStage = BK * (kAPitch + kBPitch);
  static constexpr int kSmemBytes = STAGES * kStage * 4;
  static_assert(kThreadsM % 4 == 0 && kThreadsN % 8 == 0, "a warp covers 4 x 8 threads of the grid");
  static_assert(TN % 4 == 0 && TM % QM == 0 && BK % 8 == 0, "whole quads");
};

__device__ __forceinline__ void ring_cp4(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ring_cp4(uint32_t dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void ring_cp16(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ring_cp16(uint32_t dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Row r of the tile at r0, relative to r0.  Rows that do not exist are read from the tile before: their results are not
// stored.  Not from the last row, but in the only tile: every column tile reading that up to 31 times at once is a hot spot of
// the L2 (130 x 3000 x 60 took 7.2 us, now 3.9; 140 x 2140 x 60: 6.9, now 3.6).
template <int ROWS>
__device__ __forceinline__ int ring_row(int r0, int r, int rows) {
  const int absent = r0 > 0 ? r - ROWS : rows - 1;
  return r0 + r < rows ? r : absent;
}

// ROWS rows of the operand from r0 on; slabs are asked for in order, one issue() per slab.
template <int SRC, int ROWS, int BK, int NT, int PITCH>
struct RingLoader;

template <int ROWS, int BK, int NT, int PITCH>
struct RingLoader<kRows4, ROWS, BK, NT, PITCH> {
  static constexpr int kPassRows = NT / 8, kPasses = ROWS / kPassRows;
  static_assert(ROWS % kPassRows == 0, "whole passes");
  const float* run;
  int off[kPasses];
  uint32_t dst;
  int kk;
  __device__ __forceinline__ void init(const RingParams&, const float* p, int64_t ld, int r0, int rows, uint32_t smem) {
    const int r = threadIdx.x / 8;
    kk = threadIdx.x % 8;
    run = p + r0 * ld + kk;
#pragma unroll
    for (int i = 0; i < kPasses; ++i) off[i] = static_cast<int>(ring_row<ROWS>(r0, r + i * kPassRows, rows) * ld);
    dst = smem + (kk * PITCH + r) * 4;
  }
  __device__ __forceinline__ void issue(const RingParams& p, int k0, uint32_t stage_off) {
    if (k0 + BK <= p.K) {
#pragma unroll
      for (int i = 0; i < kPasses; ++i)
#pragma unroll
        for (int o = 0; o < BK / 8; ++o)
          ring_cp4(dst + stage_off + (o * 8 * PITCH + i * kPassRows) * 4, run + off[i] + o * 8);
    } else {
#pragma unroll
      for (int i = 0; i < kPasses; ++i)
#pragma unroll
        for (int o = 0; o < BK / 8; ++o) {
          const bool in = k0 + o * 8 + kk < p.K;
          ring_cp4(dst + stage_off + (o * 8 * PITCH + i * kPassRows) * 4, in ? run + off[i] + o * 8 : p.none, in ? 4 : 0);
        }
    }
    run += BK;
  }
};

template <int ROWS, int BK, int NT, int PITCH>
struct RingLoader<kCols16, ROWS, BK, NT, PITCH> {
  static constexpr int kPassK = NT / (ROWS / 4), kPasses = BK / kPassK;
  static_assert(NT % (ROWS / 4) == 0 && BK % kPassK == 0, "whole passes");
  const float* run;
  int64_t ld;
  uint32_t dst;
  int kr, bytes;
  __device__ __forceinline__ void init(const RingParams&, const float* ptr, int64_t ld_, int r0, int rows, uint32_t smem) {
    const int c = threadIdx.x % (ROWS / 4) * 4;
    kr = threadIdx.x / (ROWS / 4);
    ld = ld_;
    bytes = max(0, min(4, rows - (r0 + c))) * 4;
    run = bytes ? ptr + kr * ld + r0 + c : nullptr;
    dst = smem + (kr * PITCH + c) * 4;
  }
  __device__ __forceinline__ void issue(const RingParams& p, int k0, uint32_t stage_off) {
    if (bytes == 16 && k0 + BK <= p.K) {
#pragma unroll
      for (int i = 0; i < kPasses; ++i) ring_cp16(dst + stage_off + i * kPassK * PITCH * 4, run + i * kPassK * ld);
    } else {
#pragma unroll
      for (int i = 0; i < kPasses; ++i) {
        const int b = k0 + kr + i * kPassK < p.K ? bytes : 0;
        ring_cp16(dst + stage_off + i * kPassK * PITCH * 4, b ? run + i * kPassK * ld : p.none, b);
      }
    }
    if (bytes) run += BK * ld;
  }
};

template <int ROWS, int BK, int NT, int PITCH>
struct RingLoader<kCols4, ROWS, BK, NT, PITCH> {
  static constexpr int kPassK = NT / ROWS, kPasses = BK / kPassK;
  static_assert(NT % ROWS == 0 && BK % kPassK == 0, "whole passes");
  const float* run;
  int64_t ld;
  uint32_t dst;
  int kr;
  bool in;
  __device__ __forceinline__ void init(const RingParams&, const float* ptr, int64_t ld_, int r0, int rows, uint32_t smem) {
    const int c = threadIdx.x % ROWS;
    kr = threadIdx.x / ROWS;
    ld = ld_;
    in = r0 + c < rows;
    run = ptr + kr * ld + min(r0 + c, rows - 1);
    dst = smem + (kr * PITCH + c) * 4;
  }
  __device__ __forceinline__ void issue(const RingParams& p, int k0, uint32_t stage_off) {
#pragma unroll
    for (int i = 0; i < kPasses; ++i) {
      const bool ok = in && k0 + kr + i * kPassK < p.K;
      ring_cp4(dst + stage_off + i * kPassK * PITCH * 4, ok ? run + i * kPassK * ld : p.none, ok ? 4 : 0);
    }
    run += BK * ld;
  }
};

// A row of the column matrix: output pixel m, k ordered (r, s, c).  A thread keeps, per row, the offset of the window's
// origin and one bit per filter tap that says whether the tap lies inside the image (R * S <= 32).
__device__ __forceinline__ void ring_window(const RingParams& p, int m, int rows, int& off, uint32_t& taps) {
  int t, wo, n, ho;
  fast_divmod(m, p.fd_wo, t, wo);
  fast_divmod(t, p.fd_ho, n, ho);
  const int h = ho * p.stride - p.pad, w = wo * p.stride - p.pad;
  off = ((n * p.H + h) * p.W + w) * p.Cin;
  const int s_lo = max(0, -w), s_hi = min(p.S, p.W - w);
  const uint32_t cols = s_hi > s_lo ? static_cast<uint32_t>((1ull << s_hi) - (1ull << s_lo)) : 0u;
  taps = 0;
  if (m >= rows) return;                   // a pixel that does not exist
  for (int q = max(0, -h); q < min(p.R, p.H - h); ++q) taps |= cols << (q * p.S);
}
template <int ROWS, int BK, int NT, int PITCH>
struct RingLoader<kWindow4, ROWS, BK, NT, PITCH> {
  static constexpr int kPassRows = NT / 8, kPasses = ROWS / kPassRows;
  static_assert(ROWS % kPassRows == 0, "whole passes");
  int off[kPasses];
  uint32_t taps[kPasses];
  uint32_t dst;
  int kk;
  __device__ __forceinline__ void init(const RingParams& p, const float*, int64_t, int r0, int rows, uint32_t smem) {
    const int r = threadIdx.x / 8;
    kk = threadIdx.x % 8;
#pragma unroll
    for (int i = 0; i < kPasses; ++i) ring_window(p, r0 + r + i * kPassRows, rows, off[i], taps[i]);
    dst = smem + (kk * PITCH + r) * 4;
  }
  __device__ __forceinline__ void issue(const RingParams& p, int k0, uint32_t stage_off) {
#pragma unroll
    for (int o = 0; o < BK / 8; ++o) {
      const int k = k0 + o * 8 + kk;
      int tap, c, fr, fs;
      fast_divmod(k, p.fd_c, tap, c);
      fast_divmod(tap, p.fd_s, fr, fs);
      const uint32_t bit = k < p.K ? 1u << tap : 0u;
      const int tap_off = (fr * p.W + fs) * p.Cin + c;
#pragma unroll
      for (int i = 0; i < kPasses; ++i) {
        const bool in = (taps[i] & bit) != 0;
        ring_cp4(dst + stage_off + (o * 8 * PITCH + i * kPassRows) * 4, p.A + (in ? off[i] + tap_off : 0), in ? 4 : 0);
      }
    }
  }
};

// [rows][BK] as in memory: 16-byte chunks of four k.  The chunks of a row are exchanged so that neither the copies (whole
// rows of 64 or 128 bytes) nor the fragment loads (the same chunk of four consecutive rows) meet in a bank.
template <int BK>
__device__ __forceinline__ int ring_swizzle(int row) {
  return BK == 16 ? (row >> 1) & 3 : row & 7;
}

template <int ROWS, int BK, int NT, int PITCH>
struct RingLoader<kRows16, ROWS, BK, NT, PITCH> {
  static constexpr int kChunks = BK / 4, kPassRows = NT / kChunks, kPasses = ROWS / kPassRows;
  static_assert((BK == 16 || BK == 32) && ROWS % kPassRows == 0 && kPassRows % 8 == 0, "whole passes, one swizzle");
  const float* run;
  int off[kPasses];
  uint32_t dst;
  int kk;
  __device__ __forceinline__ void init(const RingParams&, const float* p, int64_t ld, int r0, int rows, uint32_t smem) {
    const int r = threadIdx.x / kChunks, ch = threadIdx.x % kChunks;
    kk = ch * 4;
    run = p + r0 * ld + kk;
#pragma unroll
    for (int i = 0; i < kPasses; ++i) off[i] = static_cast<int>(ring_row<ROWS>(r0, r + i * kPassRows, rows) * ld);
    dst = smem + (r * BK + (ch ^ ring_swizzle<BK>(r)) * 4) * 4;
  }
  __device__ __forceinline__ void issue(const RingParams& p, int k0, uint32_t stage_off) {
    if (k0 + BK <= p.K) {
#pragma unroll
      for (int i = 0; i < kPasses; ++i) ring_cp16(dst + stage_off + i * kPassRows * BK * 4, run + off[i]);
    } else {
      const int bytes = max(0, min(4, p.K - (k0 + kk))) * 4;
#pragma unroll
      for (int i = 0; i < kPasses; ++i)
        ring_cp16(dst + stage_off + i * kPassRows * BK * 4, bytes ? run + off[i] : p.none, bytes);
    }
    run += BK;
  }
};

template <int ROWS, int BK, int NT, int PITCH>
struct RingLoader<kWindow16, ROWS, BK, NT, PITCH> {     // channels a multiple of 4: a chunk belongs to one tap
  static constexpr int kChunks = BK / 4, kPassRows = NT / kChunks, kPasses = ROWS / kPassRows;
  static_assert((BK == 16 || BK == 32) && ROWS % kPassRows == 0 && kPassRows % 8 == 0, "whole passes, one swizzle");
  int off[kPasses];
  uint32_t taps[kPasses];
  uint32_t dst;
  int kk;
  __device__ __forceinline__ void init(const RingParams& p, const float*, int64_t, int r0, int rows, uint32_t smem) {
    const int r = threadIdx.x / kChunks, ch = threadIdx.x % kChunks;
    kk = ch * 4;
#pragma unroll
    for (int i = 0; i < kPasses; ++i) ring_window(p, r0 + r + i * kPassRows, rows, off[i], taps[i]);
    dst = smem + (r * BK + (ch ^ ring_swizzle<BK>(r)) * 4) * 4;
  }
  __device__ __forceinline__ void issue(const RingParams& p, int k0, uint32_t stage_off) {
    const int k = k0 + kk;
    int tap, c, fr, fs;
    fast_divmod(k, p.fd_c, tap, c);
    fast_divmod(tap, p.fd_s, fr, fs);
    const uint32_t bit = k < p.K ? 1u << tap : 0u;
    const int tap_off = (fr * p.W + fs) * p.Cin + c;
#pragma unroll
    for (int i = 0; i < kPasses; ++i) {
      const bool in = (taps[i] & bit) != 0;
      ring_cp16(dst + stage_off + i * kPassRows * BK * 4, p.A + (in ? off[i] + tap_off : 0), in ? 16 : 0);
    }
  }
};

__device__ __forceinline__ uint64_t ring_dup(float v) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
  return d;
}
__device__ __forceinline__ uint64_t ring_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

template <typename T, int ASRC, int BSRC>
__global__ void __launch_bounds__(T::kThreads, T::MIN_CTAS) sgemm_f32_ring_kernel(const RingParams p) {
  constexpr int BM = T::BM, BN = T::BN, BK = T::BK, TM = T::TM, TN = T::TN, STAGES = T::STAGES, QM = T::QM;
  extern __shared__ __align__(16) float ring_smem[];
  const uint32_t smem = smem_u32(ring_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // A warp covers 4 x 8 threads of the grid.  A 16-byte shared load takes one pass per half-warp where lanes that differ in
  // bit 0, or lanes that differ in bit 1, read the same address, and two otherwise (counted: 2 against 4 wavefronts per
  // load); A addresses leave out bit 0 and B addresses bit 1.
  constexpr int kWarpsN = T::kThreadsN / 8;
  const int tn = (warp % kWarpsN) * 8 + (lane & 1) + ((lane >> 1) & 2) + ((lane >> 2) & 4);
  const int tm = (warp / kWarpsN) * 4 + ((lane >> 1) & 1) + ((lane >> 2) & 2);
  const int mt = blockIdx.x / p.tiles_n;
  const int m0 = mt * BM, n0 = (blockIdx.x - mt * p.tiles_n) * BN;

  RingLoader<ASRC, BM, BK, T::kThreads, T::kAPitch> la;
  RingLoader<BSRC, BN, BK, T::kThreads, T::kBPitch> lb;
  la.init(p, p.A, p.lda, m0, p.M, smem);
  lb.init(p, p.B, p.ldb, n0, p.N, smem + BK * T::kAPitch * 4);

  uint64_t acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0;

  const int num_slabs = (p.K + BK - 1) / BK;
  int k_issue = 0;
  uint32_t w_stage = 0, r_stage = 0;       // byte offsets of the ring stage that is filled / read
  auto issue = [&]() {
    if (k_issue < p.K) {
      la.issue(p, k_issue, w_stage);
      lb.issue(p, k_issue, w_stage);
      k_issue += BK;
    }
    cp_async_commit();
    w_stage = w_stage == (STAGES - 1) * T::kStage * 4 ? 0 : w_stage + T::kStage * 4;
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) issue();

  constexpr bool kInner = ring_row_major(ASRC);           // A in shared memory: [rows][BK], else [BK][rows]
  constexpr int kAvK = kInner ? 4 : 1;
  // row of the tile that accumulator row i belongs to: consecutive rows for one thread (K-major fragments are read along
  // them), or consecutive rows for neighbouring threads
  auto row_of = [&](int i) { return kInner ? i * T::kThreadsM + tm : ((i / QM) * T::kThreadsM + tm) * QM + i % QM; };
  float av[2][TM][kAvK];
  uint64_t bv[2][TN / 2];
  const uint32_t a_row = smem + tm * BK * 4;
  const int a_swz = ring_swizzle<BK>(tm);
  static_assert(!kInner || T::kThreadsM % 8 == 0, "one swizzle for all rows of a thread");
  auto fetch_chunk = [&](int c, int h) {                  // kInner: k = 4 c ... 4 c + 3
#pragma unroll
    for (int i = 0; i < TM; ++i)
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(av[h][i][0]), "=f"(av[h][i][1 % kAvK]), "=f"(av[h][i][2 % kAvK]), "=f"(av[h][i][3 % kAvK])
                   : "r"(a_row + r_stage + i * T::kThreadsM * BK * 4 + ((c ^ a_swz) << 4)) : "memory");
  };
  const uint32_t a_src = smem + tm * QM * 4, b_src = smem + (BK * T::kAPitch + tn * 4) * 4;
  auto fetch = [&](int kk, int h) {
#pragma unroll
    for (int q = 0; q < (kInner ? 0 : TM / QM); ++q) {
      const uint32_t src = a_src + r_stage + (kk * T::kAPitch + q * T::kThreadsM * QM) * 4;
      if constexpr (QM == 4)
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(av[h][q * 4][0]), "=f"(av[h][q * 4 + 1][0]), "=f"(av[h][q * 4 + 2][0]), "=f"(av[h][q * 4 + 3][0])
                     : "r"(src) : "memory");
      else
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(av[h][q * 2][0]), "=f"(av[h][q * 2 + 1][0]) : "r"(src) : "memory");
    }
#pragma unroll
    for (int q = 0; q < TN / 4; ++q)
      asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];"
                   : "=l"(bv[h][q * 2]), "=l"(bv[h][q * 2 + 1])
                   : "r"(b_src + r_stage + (kk * T::kBPitch + q * T::kThreadsN * 4) * 4) : "memory");
  };
  if (num_slabs > 0) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    if constexpr (kInner) fetch_chunk(0, 0);
    fetch(0, 0);
  }
  for (int s = 0; s < num_slabs; ++s) {
    issue();                               // into the stage that was read at s - 1
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      if (kInner && kk % 4 == 0 && kk + 4 < BK) fetch_chunk(kk / 4 + 1, (kk / 4 + 1) & 1);
      if (kk + 1 < BK) {
        fetch(kk + 1, (kk + 1) & 1);
      } else if (s + 1 < num_slabs) {
        cp_async_wait<STAGES - 2>();       // slab s + 1 has landed, this thread's copies ...
        __syncthreads();                   // ... and everyone's; nobody reads slab s any more
        r_stage = r_stage == (STAGES - 1) * T::kStage * 4 ? 0 : r_stage + T::kStage * 4;
        if constexpr (kInner) fetch_chunk(0, 0);
        fetch(0, 0);
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const uint64_t a2 = ring_dup(kInner ? av[(kk / 4) & 1][i][kk % kAvK] : av[kk & 1][i][0]);
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = ring_fma2(a2, bv[kk & 1][j], acc[i][j]);
      }
    }
  }
  cp_async_wait<0>();

#pragma unroll
  for (int i = 0; i < TM; ++i) {
      const int gm = m0 + row_of(i);
      if (gm >= p.M) continue;
#pragma unroll
      for (int qj = 0; qj < TN / 4; ++qj) {
        const int gn = n0 + (qj * T::kThreadsN + tn) * 4;
        float* dst = p.C + gm * p.ldc + gn;
        const uint64_t lo = acc[i][qj * 2], hi = acc[i][qj * 2 + 1];
        float v[4];
        asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(lo));
        asm("mov.b64 {%0, %1}, %2;" : "=f"(v[2]), "=f"(v[3]) : "l"(hi));
        if (p.vec_c && gn + 3 < p.N) {
          *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (gn + e < p.N) dst[e] = v[e];
        }
      }
    }
}

template <typename T, int ASRC, int BSRC>
int launch_ring(RingParams p, cudaStream_t stream) {
  auto kern = sgemm_f32_ring_kernel<T, ASRC, BSRC>;
  static thread_local int attr_dev = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (attr_dev != dev) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmemBytes) != cudaSuccess)
      return HELIX_ERR_CUDA;
    attr_dev = dev;
  }
  p.tiles_n = (p.N + T::BN - 1) / T::BN;
  const int64_t tiles = (int64_t)((p.M + T::BM - 1) / T::BM) * p.tiles_n;
  if (tiles > 0x7fffffff) return HELIX_ERR_INVALID;
  // A plain launch on purpose: with programmatic overlap the next launch's CTAs take the free slots of SMs that happen to
  // hold fewer of this one's and end up three to an SM beside SMs with one (1024^3 in a chain: 54 -> 78 us).
  kern<<<(unsigned)tiles, T::kThreads, T::kSmemBytes, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? HELIX_OK : HELIX_ERR_CUDA;
}

// The tiles the library chooses from (sgemm_f32_default_config); smaller ones for problems that would leave SMs idle.
using RingTile128x128 = RingTile<128, 128, 16, 8, 8, 4, 2>;
using RingTile128x64 = RingTile<128, 64, 16, 8, 8, 4, 3>;
using RingTile64x64 = RingTile<64, 64, 16, 4, 8, 4, 4>;
using RingTile32x64 = RingTile<32, 64, 16, 4, 4, 6, 4>;
using RingTile32x32 = RingTile<32, 32, 32, 2, 4, 4, 4>;

}  // namespace helix
