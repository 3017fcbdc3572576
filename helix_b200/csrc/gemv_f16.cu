// Memory-bound fp16 GEMV for 1..8 right-hand sides, and products of up to 16 rows: a plain kernel (explicit configurations, split
// K, small problems), and streaming kernels, with scalar multiply-adds up to two right-hand sides and mma.sync beyond (one kernel for
// short streams, with X in shared memory, a deeper one for long ones).
//
//   Y[i, r] = sum_k W[r, k] * X[i, k]        W: rows x K (row-major, the HBM stream)
//                                              X: m x K, m <= 8 (stays in L1/L2)
// fp32 accumulate, one rounding to half at the end.  Counterpart of the reference's
// mySGemvKernel_Stage4 (src_template/Ampere_FP16/gemv.cu:151-216) and its split-K twin
// (gemv_splitK.cu:153-221); unlike those it accumulates in fp32, takes any row count and any
// K that is a multiple of 8, and reduces split-K partials deterministically.
//
// Mapping of the plain kernel: one warp owns RPW consecutive rows; lane l reads the 16-byte chunk l of each
// 512-byte row segment, UNROLL segments in flight per row, so a thread keeps RPW*UNROLL
// independent 128-bit streaming loads outstanding.  Lanes are reduced with a shuffle tree.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace helix {

template <int MRHS, int RPW, int UNROLL>
__global__ void __launch_bounds__(256)
gemv_f16_kernel(const __half* __restrict__ W, int64_t ldw, const __half* __restrict__ X, int64_t ldx,
                __half* __restrict__ Y, int64_t ldy, int64_t ldy_inner, float* __restrict__ partial,
                int rows, int K, int m, int split_k, int k_per_split, int order_mode) {
  // Let the next kernel on the stream be scheduled while this one drains.  How this launch orders
  // itself after the kernel queued before it (order_mode):
  //   0  wait for it before touching global memory (safe default);
  //   1  W is not written by it (weights): the first batch of W loads is issued, THEN the kernel
  //      waits, then reads X and later writes Y -- launch latency and ramp-up hide behind the
  //      predecessor's tail while X may still be its output;
  //   2  nothing is shared with it: no wait before the work.
  // In modes 1 and 2 every thread that has not waited yet does so just before it exits, after its last
  // store: this kernel then cannot complete before its predecessor has, so a later kernel that waits
  // for this one is still ordered after everything queued earlier.  The next kernel may start after the wait in mode
  // 0, at once in modes 1 and 2 (common.cuh).
  bool waited = order_mode == 0;
  if (order_mode == 0) griddep_wait();
  griddep_launch_dependents();
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int warps_per_block = blockDim.x >> 5;
  const int row_groups = (rows + RPW - 1) / RPW;
  const int ks = blockIdx.y;
  const int k_begin = ks * k_per_split;
  const int k_end = min(K, k_begin + k_per_split);

  for (int g = blockIdx.x * warps_per_block + warp; g < row_groups; g += gridDim.x * warps_per_block) {
    const int r0 = g * RPW;
    float acc[RPW][MRHS];
#pragma unroll
    for (int r = 0; r < RPW; ++r)
#pragma unroll
      for (int i = 0; i < MRHS; ++i) acc[r][i] = 0.0f;

    const __half* wrow[RPW];
#pragma unroll
    for (int r = 0; r < RPW; ++r) wrow[r] = W + (int64_t)min(r0 + r, rows - 1) * ldw;

    for (int k0 = k_begin + lane * 8; k0 < k_end; k0 += 256 * UNROLL) {
      uint4 wv[UNROLL][RPW];
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const int k = k0 + u * 256;
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
          if (k < k_end) wv[u][r] = ldg_stream_16(wrow[r] + k);
          else wv[u][r] = make_uint4(0u, 0u, 0u, 0u);
        }
      }
      if (!waited && order_mode == 1) {   // warp-uniform
        griddep_wait();
        waited = true;
      }
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const int k = k0 + u * 256;
        if (k < k_end) {
#pragma unroll
          for (int i = 0; i < MRHS; ++i) {
            if (i < m) {
              const uint4 xv = __ldg(reinterpret_cast<const uint4*>(X + (int64_t)i * ldx + k));
              const __half2* xh = reinterpret_cast<const __half2*>(&xv);
#pragma unroll
              for (int r = 0; r < RPW; ++r) {
                const __half2* wh = reinterpret_cast<const __half2*>(&wv[u][r]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float2 wf = __half22float2(wh[j]);
                  const float2 xf = __half22float2(xh[j]);
                  acc[r][i] = fmaf(wf.x, xf.x, acc[r][i]);
                  acc[r][i] = fmaf(wf.y, xf.y, acc[r][i]);
                }
              }
            }
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < RPW; ++r)
#pragma unroll
      for (int i = 0; i < MRHS; ++i) {
        float v = acc[r][i];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        acc[r][i] = v;
      }
    if (!waited && order_mode == 1) {   // empty K range: still order the stores after the predecessor
      griddep_wait();
      waited = true;
    }
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < RPW; ++r) {
        if (r0 + r < rows) {
#pragma unroll
          for (int i = 0; i < MRHS; ++i) {
            if (i < m) {
              if (split_k == 1) Y[(int64_t)i * ldy + (int64_t)(r0 + r) * ldy_inner] = __float2half_rn(acc[r][i]);
              else partial[((int64_t)ks * m + i) * rows + r0 + r] = acc[r][i];
            }
          }
        }
      }
    }
  }
  if (!waited) griddep_wait();
}

// ---------------------------------------------------------------------------------------------
// Streaming kernels: one persistent CTA per SM, an equal share of the rows each.
//
// What bounds a GEMV is HBM, and what keeps it from HBM's rate is not the arithmetic but the shape of the grid
// and the bursts of the loads: with a warp per two rows, 4096 rows are 256 CTAs on 148 SMs (two on some, one
// on others), and a warp that has issued its batch of loads computes before it issues the next.  Here the
// rows are cut into sm_count contiguous ranges that differ by at most one row, the 16 warps of a CTA split K (KW of
// them) and, where K is short, the row blocks (16 / KW groups), and every lane streams its 16-byte chunks through a
// private FIFO of 12 slots in shared memory (cp.async): a slot is refilled as soon as it has been read, so
// 96 KB per SM are in flight all the time, no barrier is needed (a lane reads only what it copied itself) and
// two CTAs fit an SM, so the next launch on the stream can fill its FIFOs while this one drains.
// Chains of ordered launches on distinct buffers, us before -> after (static weights): 4096 x 4096, m = 1: 9.3 -> 8.2
// (8.7 -> 7.0), m = 2: 13.6 -> 9.8; 12288 x 4096: 20.6 -> 18.5 (20.6 -> 17.8); 4096 x 11008: 20.1 -> 17.0; m = 4 and 8,
// 4096 x 4096: 19.5 -> 9.6 and 9.8, 8192 x 8192: 37.5 -> 28.  What is left above the HBM time of the weights is some
// 2.5 us per launch: the predecessor's completion, the first loads' latency, the last rows' sums.
constexpr int kStreamThreads = 512;
constexpr int kStreamWarps = kStreamThreads / 32;
constexpr int kStreamLoads = 4;      // 16-byte loads of one group
constexpr int kStreamGroups = 3;     // groups in flight
constexpr int kStreamRingBytes = kStreamThreads * kStreamLoads * kStreamGroups * 16;
// order_mode 0, 1 and 2 as above; with kHoldNext the next kernel is held back until after the wait of modes 1 and 2 (used
// where these kernels stand for launches with a workspace, which are ordered whatever their flags: what was queued before
// them is complete when a flagged successor starts)

// Rows [begin, end) of this CTA.
__device__ __forceinline__ void stream_rows(int rows, int& begin, int& end) {
  begin = static_cast<int>(static_cast<int64_t>(rows) * blockIdx.x / gridDim.x);
  end = static_cast<int>(static_cast<int64_t>(rows) * (blockIdx.x + 1) / gridDim.x);
}

__device__ __forceinline__ uint4 lds_16(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

__device__ __forceinline__ void cp_async_16(uint32_t smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_dst), "l"(gsrc) : "memory");
}

// One or two right-hand sides, fp32 fused multiply-adds.  A warp takes 256-element chunks of K (16 bytes a
// lane) of four rows at a time.
template <int MRHS>
__global__ void __launch_bounds__(kStreamThreads, 2)
gemv_f16_stream_kernel(const __half* __restrict__ W, int64_t ldw, const __half* X, int64_t ldx, __half* Y,
                       int64_t ldy, int64_t ldy_inner, int rows, int K, int kw, int order_mode) {
  constexpr int kBlockRows = kStreamLoads;          // rows per block of a warp
  constexpr int kSuperRows = kStreamWarps * kBlockRows;
  extern __shared__ __align__(16) unsigned char stream_smem[];
  float* part = reinterpret_cast<float*>(stream_smem + kStreamRingBytes);   // [2][kw][MRHS][kSuperRows]
  if (order_mode != 0 && !(order_mode & kHoldNext)) griddep_launch_dependents();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rw = kStreamWarps / kw;                 // row groups
  const int kwi = warp % kw, rwi = warp / kw;
  int r_begin, r_end;
  stream_rows(rows, r_begin, r_end);
  const int blocks = (r_end - r_begin + kBlockRows - 1) / kBlockRows;
  const uint32_t slot0 = smem_u32(stream_smem) + tid * 16;

  // the group that is issued next: row block pb, elements pk ... pk + 7 of this lane
  const int k_first = kwi * 256 + lane * 8;
  const int k_step = kw * 256;
  const int k_limit = (K + 255) / 256 * 256;        // the lanes of a warp leave the chunk loop together
  int pb = rwi, pk = k_first, pslot = 0;
  if (order_mode == 0) {
    // One group per warp to the L2 ahead of the wait.  Not more: two of these CTAs fit an SM, so this one is here while the
    // predecessor streams (a decode step of one token, ordered, 4096 / 2048 wide: 243 / 107 us without, 234 / 96 with one, 250 / 97
    // with three groups, 299 / 93 with twelve).
#pragma unroll
    for (int u = 0; u < kStreamLoads; ++u)
      if (pk < K && r_begin + pb * kBlockRows + u < r_end)
        prefetch_l2(W + static_cast<int64_t>(r_begin + pb * kBlockRows + u) * ldw + pk);
    griddep_wait();
    griddep_launch_dependents();
  }
  auto issue = [&]() {
    if (pb < blocks && pk < k_limit) {
      const int row = r_begin + pb * kBlockRows;
      const __half* src = W + static_cast<int64_t>(row) * ldw + pk;
      const bool k_in = pk < K;
#pragma unroll
      for (int u = 0; u < kStreamLoads; ++u) {
        const bool in = k_in && row + u < r_end;
        cp_async_16_zfill(slot0 + (pslot * kStreamLoads + u) * kStreamThreads * 16, in ? src + u * ldw : W, in);
      }
      pk += k_step;
      if (pk >= k_limit) { pk = k_first; pb += rw; }
    }
    cp_async_commit();
    if (++pslot == kStreamGroups) pslot = 0;
  };
#pragma unroll
  for (int i = 0; i < kStreamGroups; ++i) issue();
  if (order_mode & 1) {
    griddep_wait();
    griddep_launch_dependents();
  }

  int cslot = 0, buf = 0;
  for (int sb = 0; sb < blocks; sb += kStreamWarps, buf ^= 1) {      // one superblock of up to 64 rows
    float* p = part + buf * kw * MRHS * kSuperRows;
    for (int b = sb + rwi; b < min(blocks, sb + kStreamWarps); b += rw) {
      float acc[kBlockRows][MRHS];
#pragma unroll
      for (int r = 0; r < kBlockRows; ++r)
#pragma unroll
        for (int i = 0; i < MRHS; ++i) acc[r][i] = 0.0f;
      for (int kc = kwi * 256; kc < k_limit; kc += k_step) {
        const int k = kc + lane * 8;
        uint4 xv[MRHS];
#pragma unroll
        for (int i = 0; i < MRHS; ++i)
          xv[i] = k < K ? *reinterpret_cast<const uint4*>(X + i * ldx + k) : make_uint4(0u, 0u, 0u, 0u);
        cp_async_wait<kStreamGroups - 1>();
        uint4 wv[kBlockRows];
#pragma unroll
        for (int u = 0; u < kBlockRows; ++u) wv[u] = lds_16(slot0 + (cslot * kStreamLoads + u) * kStreamThreads * 16);
        issue();
        if (++cslot == kStreamGroups) cslot = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float2 xf[MRHS];
#pragma unroll
          for (int i = 0; i < MRHS; ++i) xf[i] = __half22float2(reinterpret_cast<const __half2*>(&xv[i])[j]);
#pragma unroll
          for (int r = 0; r < kBlockRows; ++r) {
            const float2 wf = __half22float2(reinterpret_cast<const __half2*>(&wv[r])[j]);
#pragma unroll
            for (int i = 0; i < MRHS; ++i) {
              acc[r][i] = fmaf(wf.x, xf[i].x, acc[r][i]);
              acc[r][i] = fmaf(wf.y, xf[i].y, acc[r][i]);
            }
          }
        }
      }
      // four sums over 32 lanes: halve the number of values with the first two exchanges
#pragma unroll
      for (int i = 0; i < MRHS; ++i) {
        const bool hi = lane & 16, mid = lane & 8;
        float v0 = hi ? acc[2][i] : acc[0][i], v1 = hi ? acc[3][i] : acc[1][i];
        v0 += __shfl_xor_sync(0xffffffffu, hi ? acc[0][i] : acc[2][i], 16);
        v1 += __shfl_xor_sync(0xffffffffu, hi ? acc[1][i] : acc[3][i], 16);
        float v = mid ? v1 : v0;
        v += __shfl_xor_sync(0xffffffffu, mid ? v0 : v1, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        if ((lane & 7) == 0) p[(kwi * MRHS + i) * kSuperRows + (b - sb) * kBlockRows + (lane >> 3)] = v;
      }
    }
    __syncthreads();
    // the K slices of every row in slice order; the other buffer takes the next superblock's partial sums
    const int row0 = r_begin + sb * kBlockRows;
    if (tid < kSuperRows * MRHS) {
      const int i = tid / kSuperRows, r = tid - i * kSuperRows;
      if (row0 + r < r_end) {
        float s = 0.0f;
        for (int q = 0; q < kw; ++q) s += p[(q * MRHS + i) * kSuperRows + r];
        Y[i * ldy + static_cast<int64_t>(row0 + r) * ldy_inner] = __float2half_rn(s);
      }
    }
  }
  if (order_mode & 2) griddep_wait();
}

__device__ __forceinline__ void mma_f16_16x8x16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Three to 8 * NT right-hand sides: the same stream, contracted by warp-level matrix instructions (16 x 8 x 16, fp32
// accumulation).  The rate they need is small (8 multiply-adds per weight against some 23 bytes of weights per
// SM and clock); what they save is the issue slots of NT * 8 scalar multiply-adds per weight, and against a
// 128-row tcgen05 tile they save the quantisation of the rows: a CTA's rows are cut into equal blocks of at most 32,
// and absent rows cost no traffic.  The fragments need no shuffle: lane (g, t) of a fragment takes the 8
// consecutive elements at k + 8 t of row g as the K positions 2t, 2t + 1, 2t + 8, 2t + 9 of two instructions, for the
// weights and for X alike, so every product still meets its partner.  X does not fit the L1 that two resident CTAs
// leave, so its fragments come from L2 and are fetched one group ahead, which takes registers: 8 warps of up
// to 128, each with a FIFO of 24 slots (the same 96 KB where a block has 32 rows; a CTA of fewer keeps 3 KB per row in flight,
// which is why few rows over a long K go elsewhere).
constexpr int kMmaThreads = 256;
constexpr int kMmaWarps = kMmaThreads / 32;
constexpr int kMmaSlots = 24;

template <int NT>
__global__ void __launch_bounds__(kMmaThreads, 2)
gemv_f16_mma_kernel(const __half* __restrict__ W, int64_t ldw, const __half* X, int64_t ldx, __half* Y, int64_t ldy,
                    int64_t ldy_inner, int rows, int K, int m, int kw, int order_mode) {
  constexpr int kMaxRows = 32;                      // rows per block of a warp: two 16-row fragments
  constexpr int kTok = NT * 8;
  constexpr int J = 2;                              // 32-element pieces of K per group
  constexpr int kGroups = kMmaSlots / (4 * J);
  extern __shared__ __align__(16) unsigned char stream_smem[];
  float* part = reinterpret_cast<float*>(stream_smem + kMmaThreads * kMmaSlots * 16);   // [warp][kTok][16 rows]
  if (order_mode == 0) griddep_wait();
  if (!(order_mode & kHoldNext)) griddep_launch_dependents();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int rw = kMmaWarps / kw;
  const int kwi = warp % kw, rwi = warp / kw;
  int r_begin, r_end;
  stream_rows(rows, r_begin, r_end);
  const int n = r_end - r_begin;
  // equal blocks of at most 32 rows, and where K leaves several row groups at least 16 rows for each
  const int blocks = max((n + kMaxRows - 1) / kMaxRows, min(rw, (n + 15) / 16));
  const int height = blocks ? (n + blocks - 1) / blocks : 0;
  // the kw warps take groups of K in turn: together they read contiguous stretches of every row
  const int k_begin = kwi * 32 * J, k_step = kw * 32 * J;
  const uint32_t slot0 = smem_u32(stream_smem) + tid * 16;
  const uint32_t slot_last = slot0 + (kGroups - 1) * 8 * kMmaThreads * 16;

  // Rows beyond the block read its last row again and right-hand sides beyond m the last one (the same lines; nothing is
  // written for them), so that only the end of a K that is no multiple of 64 needs predicates.
  int pb = rwi, pk = k_begin;
  uint32_t pslot = slot0;
  const __half* src[4];
  auto block_rows = [&]() {
    const int row = pb * height, last = min(height, n - row) - 1;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      src[u] = W + static_cast<int64_t>(r_begin + row + max(0, min(u * 8 + g, last))) * ldw + k_begin + t * 8;
  };
  block_rows();
  auto issue = [&]() {
    if (pb < blocks && pk < K) {
      if (pk + 64 <= K) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (u * 8 < height) {
            cp_async_16(pslot + (u * 2) * kMmaThreads * 16, src[u]);
            cp_async_16(pslot + (u * 2 + 1) * kMmaThreads * 16, src[u] + 32);
          }
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const bool in = pk + j * 32 + t * 8 < K;
            cp_async_16_zfill(pslot + (u * 2 + j) * kMmaThreads * 16, in ? src[u] + j * 32 : W, in);
          }
      }
      pk += k_step;
#pragma unroll
      for (int u = 0; u < 4; ++u) src[u] += k_step;
      if (pk >= K) {
        pk = k_begin;
        pb += rw;
        if (pb < blocks) block_rows();
      }
    }
    cp_async_commit();
    pslot = pslot == slot_last ? slot0 : pslot + 8 * kMmaThreads * 16;
  };
#pragma unroll
  for (int i = 0; i < kGroups; ++i) issue();
  if (order_mode & 1) {
    griddep_wait();
    griddep_launch_dependents();
  }

  const __half* xrow[NT];                           // this lane's right-hand side of each group of eight
#pragma unroll
  for (int q = 0; q < NT; ++q) xrow[q] = X + min(q * 8 + g, m - 1) * ldx + t * 8;
  auto load_x = [&](int k, uint4 (&x)[J][NT]) {
    if (k + 64 <= K) {
#pragma unroll
      for (int j = 0; j < J; ++j)
#pragma unroll
        for (int q = 0; q < NT; ++q) x[j][q] = *reinterpret_cast<const uint4*>(xrow[q] + k + j * 32);
    } else {
#pragma unroll
      for (int j = 0; j < J; ++j)
#pragma unroll
        for (int q = 0; q < NT; ++q)
          x[j][q] = k + j * 32 + t * 8 < K ? *reinterpret_cast<const uint4*>(xrow[q] + k + j * 32)
                                           : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  uint32_t cslot = slot0;
  for (int sb = 0; sb < blocks; sb += rw) {         // one block per row group
    const int b = sb + rwi;
    float acc[2][NT][4];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int q = 0; q < NT; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[h][q][e] = 0.0f;
    if (b < blocks) {
      uint4 xn[J][NT];
      load_x(k_begin, xn);
      for (int k = k_begin; k < K; k += k_step) {
        uint4 xv[J][NT];
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
          for (int q = 0; q < NT; ++q) xv[j][q] = xn[j][q];
        load_x(k + k_step, xn);
        cp_async_wait<kGroups - 1>();
        uint4 wv[4][J];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int j = 0; j < J; ++j) wv[u][j] = lds_16(cslot + (u * J + j) * kMmaThreads * 16);
        issue();
        cslot = cslot == slot_last ? slot0 : cslot + 8 * kMmaThreads * 16;
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < NT; ++q) {
              const uint4 w0 = wv[2 * h][j], w1 = wv[2 * h + 1][j];
              mma_f16_16x8x16(acc[h][q], w0.x, w1.x, w0.y, w1.y, xv[j][q].x, xv[j][q].y);
              mma_f16_16x8x16(acc[h][q], w0.z, w1.z, w0.w, w1.w, xv[j][q].z, xv[j][q].w);
            }
      }
    }
    // 16 rows of every row group at a time: partial sums to shared memory, slices added in slice order
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h * 16 < height) {
        __syncthreads();                            // the previous sums have been read
#pragma unroll
        for (int q = 0; q < NT; ++q)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            part[(warp * kTok + q * 8 + t * 2 + (e & 1)) * 16 + g + (e >> 1) * 8] = acc[h][q][e];
        __syncthreads();
        for (int o = tid; o < rw * kTok * 16; o += kMmaThreads) {
          const int r16 = o & 15, tok = (o >> 4) % kTok, grp = (o >> 4) / kTok;
          const int r = h * 16 + r16, row = (sb + grp) * height + r;
          if (tok < m && r < height && sb + grp < blocks && row < n) {
            float s = 0.0f;
            for (int q = 0; q < kw; ++q) s += part[((grp * kw + q) * kTok + tok) * 16 + r16];
            Y[tok * ldy + static_cast<int64_t>(r_begin + row) * ldy_inner] = __float2half_rn(s);
          }
        }
      }
    }
  }
  if (order_mode & 2) griddep_wait();
}

// The same product where the stream is long (gemv_f16_deep): X does not fit the SM, so it goes through the same per-lane FIFO
// as the weights (NT of a group's 2 F + NT slots per 32 elements of K), and its trips to L2 are as deeply pipelined as the
// weights' trips to HBM.  It is read once per block, so blocks are as high as pays (16 F rows); a group is J pieces of 32
// elements, one CTA has the SM's shared memory to itself.  Ordered chains on distinct buffers, us above / here: m = 8,
// 4096 x 4096 9.9 / 9.3, 12288 x 4096 22.6 / 20.9, 8192 x 8192 28.3 / 26.0, 1024 x 8192 12.2 / 8.0, 900 x 12000 16.4 / 10.0; m = 16,
// 12288 x 4096 25.1 / 23.0, 11008 x 4096 23.9 / 21.6, 4096 x 11008 22.7 / 20.6.  On small problems its longer set-up shows:
// 1000 x 3000, m = 8, 4.9 / 5.5; 600 x 600 3.1 / 3.5.
constexpr int kMmaSlotBytes = kMmaThreads * 16;

template <int NT, int F, int J, int CTAS>
struct DeepStream {
  static constexpr int kTok = NT * 8;
  static constexpr int kSumFrags = CTAS > 1 ? 1 : F < 3 ? F : 3;      // 16-row fragments summed at a time
  static constexpr int kSumPitch = 16 * kSumFrags + 4;        // floats per right-hand side: lanes of a quad 8 banks apart
  static constexpr int kPartBytes = kMmaWarps * kTok * kSumPitch * 4;
  static constexpr int kSlots = (2 * F + NT) * J;             // 16-byte slots of a lane per 32 J elements of K
  static constexpr int kFit = ((CTAS == 1 ? 226 : 112) * 1024 - kPartBytes) / (kMmaSlotBytes * kSlots);
  static constexpr int kGroups = kFit < 8 ? kFit : 8;         // groups in flight
  static constexpr int kSmem = kGroups * kSlots * kMmaSlotBytes + kPartBytes;
  static_assert(kGroups >= 2, "a group is read while others are in flight");
};

template <int NT, int F, int J, int CTAS>
__global__ void __launch_bounds__(kMmaThreads, CTAS)
gemv_f16_deep_kernel(const __half* __restrict__ W, int64_t ldw, const __half* X, int64_t ldx, __half* Y, int64_t ldy,
                    int64_t ldy_inner, int rows, int K, int m, int kw, int order_mode) {
  using S = DeepStream<NT, F, J, CTAS>;
  constexpr int kMaxRows = 16 * F, kTok = S::kTok, kGroups = S::kGroups, kSlots = S::kSlots;
  constexpr int kXSlot = 2 * F * J;                 // X follows the weights in a group
  extern __shared__ __align__(16) unsigned char stream_smem[];
  float* part = reinterpret_cast<float*>(stream_smem + kGroups * kSlots * kMmaSlotBytes);   // [warp][kTok][kSumPitch]
  if (order_mode != 0 && !(order_mode & kHoldNext)) griddep_launch_dependents();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int rw = kMmaWarps / kw;
  const int kwi = warp % kw, rwi = warp / kw;
  int r_begin, r_end;
  stream_rows(rows, r_begin, r_end);
  const int n = r_end - r_begin;
  // equal blocks of at most 16 F rows, and where K leaves several row groups at least 16 rows for each
  const int blocks = max((n + kMaxRows - 1) / kMaxRows, min(rw, (n + 15) / 16));
  const int height = blocks ? (n + blocks - 1) / blocks : 0;
  // the kw warps take 32 J elements of K in turn: together they read contiguous stretches of every row
  const int k_begin = kwi * 32 * J, k_step = kw * 32 * J;
  const uint32_t slot0 = smem_u32(stream_smem) + tid * 16;
  const uint32_t slot_last = slot0 + (kGroups - 1) * kSlots * kMmaSlotBytes;
  auto next_group = [&](uint32_t s) { return s == slot_last ? slot0 : s + kSlots * kMmaSlotBytes; };

  // Rows beyond the block and right-hand sides beyond m are not copied: their slots hold whatever was there, which reaches
  // only rows and columns of the product that are not stored.
  int pb = rwi, pk = k_begin;
  uint32_t pslot = slot0;
  const __half* src[2 * F];
  uint32_t live = 0;                                // bit u: row u * 8 + g exists
  auto block_rows = [&]() {
    const int row = pb * height, here = min(height, n - row);
    live = 0;
#pragma unroll
    for (int u = 0; u < 2 * F; ++u) {
      if (u * 8 + g < here) live |= 1u << u;
      src[u] = W + static_cast<int64_t>(r_begin + row + u * 8 + g) * ldw + k_begin + t * 8;
    }
  };
  block_rows();
  if (order_mode == 0) {
    // What the FIFOs will hold, on its way to the L2 while the predecessor drains: a CTA gets its SM when the one before
    // leaves it, and waits for the last one (a decode step of 16 tokens, 4096 wide: 301 -> 279 us; half as much 283, twice as much 288).
#pragma unroll
    for (int i = 0; i < kGroups; ++i)
#pragma unroll
      for (int u = 0; u < 2 * F; ++u)
        if ((live >> u & 1) && pk + i * k_step + 32 * J <= K) {
#pragma unroll
          for (int j = 0; j < J; ++j) prefetch_l2(src[u] + i * k_step + j * 32);
        }
    griddep_wait();
    griddep_launch_dependents();
  }
  auto issue_w = [&]() {
    if (pb < blocks && pk < K) {
      if (pk + 32 * J <= K) {
#pragma unroll
        for (int u = 0; u < 2 * F; ++u)
          if (live >> u & 1)
#pragma unroll
            for (int j = 0; j < J; ++j) cp_async_16(pslot + (u * J + j) * kMmaSlotBytes, src[u] + j * 32);
      } else {
#pragma unroll
        for (int u = 0; u < 2 * F; ++u)
#pragma unroll
          for (int j = 0; j < J; ++j) {
            const bool in = (live >> u & 1) && pk + j * 32 + t * 8 < K;
            cp_async_16_zfill(pslot + (u * J + j) * kMmaSlotBytes, in ? src[u] + j * 32 : W, in);
          }
      }
      pk += k_step;
#pragma unroll
      for (int u = 0; u < 2 * F; ++u) src[u] += k_step;
      if (pk >= K) {
        pk = k_begin;
        pb += rw;
        if (pb < blocks) block_rows();
      }
    }
    pslot = next_group(pslot);
  };
  int xb = rwi, xk = k_begin;
  uint32_t xslot = slot0 + kXSlot * kMmaSlotBytes;
  const uint32_t xslot_last = slot_last + kXSlot * kMmaSlotBytes;
  const __half* const xrow = X + g * ldx + t * 8;   // this lane's right-hand sides: g, g + 8, ...
  auto issue_x = [&]() {
    if (xb < blocks && xk < K) {
#pragma unroll
      for (int q = 0; q < NT; ++q)
        if (q * 8 + g < m)
#pragma unroll
          for (int j = 0; j < J; ++j) {
            const bool in = xk + j * 32 + t * 8 < K;
            cp_async_16_zfill(xslot + (q * J + j) * kMmaSlotBytes, in ? xrow + q * 8 * ldx + xk + j * 32 : X, in);
          }
      xk += k_step;
      if (xk >= K) {
        xk = k_begin;
        xb += rw;
      }
    }
    xslot = xslot == xslot_last ? slot0 + kXSlot * kMmaSlotBytes : xslot + kSlots * kMmaSlotBytes;
  };
  // The first groups' weights and, after the wait of mode 1, their X are commit groups of their own; from then on a group is
  // one.  Whatever precedes X's group i is complete when at most kGroups - 1 later ones are pending, so one count serves all.
#pragma unroll
  for (int i = 0; i < kGroups; ++i) {
    issue_w();
    cp_async_commit();
  }
  if (order_mode & 1) {
    griddep_wait();
    griddep_launch_dependents();
  }
#pragma unroll
  for (int i = 0; i < kGroups; ++i) {
    issue_x();
    cp_async_commit();
  }

  uint32_t cslot = slot0;
  for (int sb = 0; sb < blocks; sb += rw) {         // one block per row group
    const int b = sb + rwi;
    float acc[F][NT][4];
#pragma unroll
    for (int h = 0; h < F; ++h)
#pragma unroll
      for (int q = 0; q < NT; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[h][q][e] = 0.0f;
    if (b < blocks) {
      for (int k = k_begin; k < K; k += k_step) {
        cp_async_wait<kGroups - 1>();
        uint4 xv[NT][J], wv[2 * F][J];
#pragma unroll
        for (int q = 0; q < NT; ++q)
#pragma unroll
          for (int j = 0; j < J; ++j) xv[q][j] = lds_16(cslot + (kXSlot + q * J + j) * kMmaSlotBytes);
#pragma unroll
        for (int u = 0; u < 2 * F; ++u)
          if ((u & ~1) * 8 < height)
#pragma unroll
            for (int j = 0; j < J; ++j) wv[u][j] = lds_16(cslot + (u * J + j) * kMmaSlotBytes);
        issue_w();
        issue_x();
        cp_async_commit();
        cslot = next_group(cslot);
#pragma unroll
        for (int h = 0; h < F; ++h)
          if (h * 16 < height)
#pragma unroll
            for (int j = 0; j < J; ++j)
#pragma unroll
              for (int q = 0; q < NT; ++q) {
                const uint4 w0 = wv[2 * h][j], w1 = wv[2 * h + 1][j];
                mma_f16_16x8x16(acc[h][q], w0.x, w1.x, w0.y, w1.y, xv[q][j].x, xv[q][j].y);
                mma_f16_16x8x16(acc[h][q], w0.z, w1.z, w0.w, w1.w, xv[q][j].z, xv[q][j].w);
              }
      }
    }
    // some fragments of every row group at a time: partial sums to shared memory, slices added in slice order
#pragma unroll
    for (int h0 = 0; h0 < F; h0 += S::kSumFrags) {
      if (h0 * 16 < height) {
        __syncthreads();                            // the previous sums have been read
#pragma unroll
        for (int h = h0; h < F && h < h0 + S::kSumFrags; ++h)
#pragma unroll
          for (int q = 0; q < NT; ++q)
#pragma unroll
            for (int e = 0; e < 4; ++e)
              part[(warp * kTok + q * 8 + t * 2 + (e & 1)) * S::kSumPitch + (h - h0) * 16 + g + (e >> 1) * 8] = acc[h][q][e];
        __syncthreads();
        constexpr int kSumRows = 16 * S::kSumFrags;
        for (int o = tid; o < rw * kTok * kSumRows; o += kMmaThreads) {
          const int rr = o % kSumRows, tok = (o / kSumRows) % kTok, grp = (o / kSumRows) / kTok;
          const int r = h0 * 16 + rr, row = (sb + grp) * height + r;
          if (tok < m && r < height && sb + grp < blocks && row < n) {
            float s = 0.0f;
            for (int q = 0; q < kw; ++q) s += part[((grp * kw + q) * kTok + tok) * S::kSumPitch + rr];
            Y[tok * ldy + static_cast<int64_t>(r_begin + row) * ldy_inner] = __float2half_rn(s);
          }
        }
      }
    }
  }
  if (order_mode & 2) griddep_wait();
}

// Sums the split-K partials in slice order (deterministic) and rounds once.
__global__ void gemv_splitk_reduce_kernel(const float* __restrict__ partial, __half* __restrict__ Y, int64_t ldy,
                                          int64_t ldy_inner, int rows, int m, int split_k) {
  griddep_wait();
  griddep_launch_dependents();
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * m) return;
  const int i = idx / rows, r = idx - i * rows;
  float s = 0.0f;
  for (int ks = 0; ks < split_k; ++ks) s += __ldcg(&partial[((int64_t)ks * m + i) * rows + r]);
  Y[(int64_t)i * ldy + (int64_t)r * ldy_inner] = __float2half_rn(s);
}

size_t gemv_f16_workspace_bytes(int rows, int m, int split_k) {
  return split_k > 1 ? (size_t)split_k * m * rows * sizeof(float) : 0;
}

int gemv_f16_default_split(int rows, int K, int sm_count) {
  // Cut K only when there are too few rows to keep enough bytes in flight: a warp holds 4 KiB of loads, and
  // the stream needs some 24 warps per SM before HBM saturates (512 rows x 500 000: split 4 reads at 2.9 TB/s,
  // split 16 at 6.5).  The partials cost a second launch and forbid overlapping with the neighbouring
  // launches, so beyond four warps per SM only very long rows are cut.
  const int groups = (rows + 1) / 2;
  int split = 1;
  while (split < 16 && K / (split * 2) >= 2048 &&
         ((int64_t)groups * split < (int64_t)sm_count * 4 ||
          ((int64_t)groups * split < (int64_t)sm_count * 24 && K / (split * 2) >= 16384)))
    split *= 2;
  return split;
}

// Set by gemv_f16_launch for the duration of one call: how the launch orders itself after the
// kernel queued before it (see order_mode in the kernel).
static thread_local int independent = 0;

template <int MRHS, int RPW, int UNROLL>
static int launch_gemv(const __half* W, int64_t ldw, const __half* X, int64_t ldx, __half* Y, int64_t ldy,
                       int64_t ldy_inner, float* partial, int rows, int K, int m, int split_k, int sm_count,
                       cudaStream_t stream, int64_t* launches) {
  const int row_groups = (rows + RPW - 1) / RPW;
  const int warps = 8;
  int blocks = (row_groups + warps - 1) / warps;
  const int max_blocks = sm_count * 8;
  if (blocks > max_blocks) blocks = max_blocks;
  int k_per_split = (K + split_k - 1) / split_k;
  k_per_split = (k_per_split + 255) / 256 * 256;
  dim3 grid(blocks, split_k);
  // split-K shares its scratch with neighbouring launches, so it always orders itself after them
  const int indep = split_k == 1 ? independent : 0;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = grid;
  lc.blockDim = dim3(warps * 32);
  lc.dynamicSmemBytes = 0;
  lc.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = attr;
  lc.numAttrs = 1;
  if (cudaLaunchKernelEx(&lc, gemv_f16_kernel<MRHS, RPW, UNROLL>, W, ldw, X, ldx, Y, ldy, ldy_inner, partial, rows, K,
                         m, split_k, k_per_split, indep) != cudaSuccess) {
    (void)cudaGetLastError();
    gemv_f16_kernel<MRHS, RPW, UNROLL><<<grid, warps * 32, 0, stream>>>(W, ldw, X, ldx, Y, ldy, ldy_inner, partial,
                                                                        rows, K, m, split_k, k_per_split, indep);
  }
  ++*launches;
  if (split_k > 1) {
    const int n = rows * m;
    if (launch_overlapped(gemv_splitk_reduce_kernel, dim3((n + 255) / 256), dim3(256), 0, stream, partial, Y, ldy, ldy_inner,
                          rows, m, split_k) != cudaSuccess)
      return HELIX_ERR_CUDA;
    ++*launches;
  }
  return cudaGetLastError() == cudaSuccess ? HELIX_OK : HELIX_ERR_CUDA;
}

// (rows per warp, 16-byte loads in flight per row and thread) variants compiled in.
template <int MRHS>
static int launch_gemv_variant(int rpw, int unroll, const __half* W, int64_t ldw, const __half* X, int64_t ldx,
                               __half* Y, int64_t ldy, int64_t ldy_inner, float* partial, int rows, int K, int m,
                               int split_k, int sm_count, cudaStream_t stream, int64_t* launches) {
#define HELIX_GEMV_CASE(R, U)                                                                                 \
  if (rpw == R && unroll == U)                                                                                \
    return launch_gemv<MRHS, R, U>(W, ldw, X, ldx, Y, ldy, ldy_inner, partial, rows, K, m, split_k, sm_count, \
                                   stream, launches);
  HELIX_GEMV_CASE(1, 2)
  HELIX_GEMV_CASE(1, 4)
  HELIX_GEMV_CASE(1, 8)
  HELIX_GEMV_CASE(1, 16)
  HELIX_GEMV_CASE(2, 2)
  HELIX_GEMV_CASE(2, 4)
  HELIX_GEMV_CASE(2, 8)
#undef HELIX_GEMV_CASE
  return HELIX_ERR_UNSUPPORTED;
}

// Warps that split K: the smallest power of two whose shares of whole `unit`s cover K.
static int stream_k_warps(int K, int unit, int warps) {
  int kw = warps;
  while (kw > 1 && (int64_t)(kw / 2) * unit >= K) kw /= 2;
  return kw;
}

template <typename... Params, typename... Args>
static int launch_stream(void (*kern)(Params...), int& attr_dev, int grid, int threads, int smem, cudaStream_t stream,
                         int64_t* launches, Args... args) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (attr_dev != dev) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return HELIX_ERR_CUDA;
    attr_dev = dev;
  }
  if (launch_overlapped(kern, dim3(grid), dim3(threads), smem, stream, args...) != cudaSuccess) return HELIX_ERR_CUDA;
  ++*launches;
  return HELIX_OK;
}

// Streams that are worth the deep kernel's set-up: some 8 MB where K is long, 20 MB otherwise (us, above / deep: 1184 x 4096, m = 8,
// 7.3 / 6.7; 700 x 8192 12.0 / 9.8; 300 x 4096 5.2 / 5.4; 3582 x 3048, m = 6, 7.3 / 7.2; 1852 x 3288, m = 4, 7.0 / 7.4; 22912 x 792, m = 3,
// 11.6 / 14.4).
static bool gemv_f16_deep(int rows, int K) { return K >= 1024 && (int64_t)rows * K > (K >= 4096 ? 4 << 20 : 10 << 20); }

int gemv_f16_stream_launch(const void* W, int64_t ldw, const void* X, int64_t ldx, void* Y, int64_t ldy,
                           int64_t ldy_inner, int rows, int K, int m, int sm_count, int order_mode,
                           cudaStream_t stream, int64_t* launches) {
  if (!W || !X || !Y || rows <= 0 || K <= 0 || m <= 0 || m > 16) return HELIX_ERR_INVALID;
  if (ldw == 0) ldw = K;
  if (ldx == 0) ldx = K;
  if (ldy == 0) ldy = rows;
  if (ldy_inner == 0) ldy_inner = 1;
  if ((K & 7) || (ldw & 7) || (ldx & 7) || (reinterpret_cast<uintptr_t>(W) & 15) ||
      (reinterpret_cast<uintptr_t>(X) & 15))
    return HELIX_ERR_ALIGN;
  const __half* w = static_cast<const __half*>(W);
  const __half* x = static_cast<const __half*>(X);
  __half* y = static_cast<__half*>(Y);
  int grid = std::min(sm_count, rows);
  // Independent launches run side by side: a small one on few CTAs, so that several fit the machine (us per launch, 148 CTAs /
  // this / the plain kernel that used to run here: 2048 x 2048, m = 1, 2.1 / 1.45 / 1.5; 1184 x 4096, m = 4, 3.8 / 1.8 / 2.3).  The order
  // of a row's sums does not depend on the grid.
  if (order_mode == 2) {
    const int64_t kb = (int64_t)rows * K * 2 >> 10;
    grid = (int)std::min<int64_t>(grid, std::max<int64_t>({1, kb / 256, std::min<int64_t>(32, kb / 128)}));
  }
  static thread_local int attr_dev[4] = {-1, -1, -1, -1};   // device the kernel's shared-memory size was last raised on
  if (m <= 2) {
    const int kw = stream_k_warps(K, 256, kStreamWarps);
    const int smem = kStreamRingBytes + 2 * kStreamWarps * m * kStreamWarps * kStreamLoads * 4;
    if (m == 1)
      return launch_stream(gemv_f16_stream_kernel<1>, attr_dev[0], grid, kStreamThreads, smem, stream, launches, w, ldw, x, ldx, y, ldy,
                           ldy_inner, rows, K, kw, order_mode);
    return launch_stream(gemv_f16_stream_kernel<2>, attr_dev[1], grid, kStreamThreads, smem, stream, launches, w, ldw, x, ldx, y, ldy,
                         ldy_inner, rows, K, kw, order_mode);
  }
  if (!gemv_f16_deep(rows, K)) {
    const int kw = stream_k_warps(K, 64, kMmaWarps);
    const int smem = kMmaThreads * kMmaSlots * 16 + kMmaWarps * (m <= 8 ? 8 : 16) * 16 * 4;
    if (m <= 8)
      return launch_stream(gemv_f16_mma_kernel<1>, attr_dev[2], grid, kMmaThreads, smem, stream, launches, w, ldw, x, ldx, y, ldy,
                           ldy_inner, rows, K, m, kw, order_mode);
    return launch_stream(gemv_f16_mma_kernel<2>, attr_dev[3], grid, kMmaThreads, smem, stream, launches, w, ldw, x, ldx, y, ldy,
                         ldy_inner, rows, K, m, kw, order_mode);
  }
  auto deep = [&](auto nt, auto f, auto j, auto ctas) {
    constexpr int NT = decltype(nt)::value, F = decltype(f)::value, J = decltype(j)::value, CTAS = decltype(ctas)::value;
    const int kw = stream_k_warps(K, 32 * J, kMmaWarps);
    static thread_local int deep_dev = -1;
    return launch_stream(gemv_f16_deep_kernel<NT, F, J, CTAS>, deep_dev, grid, kMmaThreads, DeepStream<NT, F, J, CTAS>::kSmem, stream,
                         launches, w, ldw, x, ldx, y, ldy, ldy_inner, rows, K, m, kw, order_mode);
  };
  const std::integral_constant<int, 1> one{};
  const std::integral_constant<int, 2> two{};
  const std::integral_constant<int, 4> four{};
  // J sets the order of a row's sums, so it follows from the sizes alone (us at J = 2 / 4: 1024 x 8192, m = 8, 8.7 / 8.0, 4096 x
  // 4096 9.3 / 9.3; 1200 x 16384, m = 16, 17.7 / 15.2).  F and the CTAs to an SM do not: blocks of 64 rows where they replace two of
  // 32 that would be half empty, or where X is twice as long (5120 x 5120, m = 8, F = 2 / 4: 13.9 / 12.9; 12288 x 4096, m = 16, 23.7 /
  // 23.0); independent launches share SMs (8656 x 1280, m = 3: 5.8 alone on an SM, 4.6 two to one).
  const bool share = order_mode == 2;
  const int per_cta = (rows + grid - 1) / grid;
  if (rows < 2400) {
    if (m > 8) return deep(two, two, four, one);
    return share ? deep(one, one, four, two) : deep(one, two, four, one);
  }
  if (m > 8) return share ? deep(two, two, two, two) : per_cta > 32 ? deep(two, four, two, one) : deep(two, two, two, one);
  return share ? deep(one, two, two, two) : per_cta > 32 && per_cta <= 48 ? deep(one, four, two, one) : deep(one, two, two, one);
}

// Which GEMVs without a configuration of their own the streaming kernels run (whatever their flags, which change no bits).
// `split`: what gemv_f16_default_split says, `scratch`: there is room for its partial sums.  us, ordered, kernel above /
// streaming:
static bool gemv_f16_streams(int rows, int K, int m, int split, bool scratch, int sm_count) {
  const int64_t work = (int64_t)rows * K;
  if (m <= 2) {
    // Below 2 M elements a lone launch is all latency and the plain grid is shorter (256 x 256: 1.4 / 1.9).
    if (work < 1 << 21) return false;
    // Streaming needs no partial sums in memory and cuts K among the warps of a CTA, so it also takes row counts for which
    // the kernel above would split K over CTAs (700 x 12000: 11.9 / 6.7); with K beyond 32768 and few rows the split keeps
    // more SMs equally busy.
    if (split > 1) return rows >= sm_count && K <= 32768;
    // Many short rows: every 64 of them end in a barrier and a sum over the warps.  m = 1: 4096 x 768 3.3 / 3.5, 5000 x 1536
    // 5.4 / 5.7, 8192 x 1024 4.8 / 5.6, 12000 x 3072 14.8 / 15.7; 4096 x 1280 4.7 / 4.7, 6000 x 2048 6.9 / 7.1 (with static
    // weights 5.7 / 5.5), 8192 x 4096 13.6 / 13.2; 12000 x 256 with static weights 3.1 / 2.5, otherwise 3.6 / 3.7.
    return m == 2 || rows < 4096 || K > 3072 || (rows < 8192 && K > 1536) || (rows < 5000 && K > 768) ||
           (rows >= 10000 && K < 512);
  }
  // A CTA's chain over K takes some time per 1000 elements whatever m, the split kernel's m times K / split.  Split / streaming, the
  // kernel for small streams: m = 3, 64 x 65536 15.3 / 66; m = 8, 64 x 65536 36 / 74 (split 16); from 1024 rows on the slices are more
  // warps than fit.  The deep one, 0.6 us per 1000: m = 3, 111 x 60672 15.2 / 34.4, 120 x 40280 11.8 / 24.2, 644 x 52288 88 / 31; m = 4, 186 x
  // 22344 14.0 / 19.0, 248 x 39640 23.4 / 24.8; m = 5, 142 x 42960 19.9 / 25.6, 374 x 16584 22.1 / 14.1; m = 8, 296 x 16384 20.5 / 16.0.
  if (scratch && rows < 1024) {
    if (!gemv_f16_deep(rows, K)) return split < m || (split == m && rows < 64);
    return rows >= 256 || K < (m <= 4 ? 16384 : 40000);
  }
  return !(m == 3 && K <= 256 && rows <= 512);         // 256 x 256: 1.9 / 2.2
}

// Skinny products: the streaming kernels against the stream-K tcgen05 tiles (or, without scratch, plain tiles, which lose
// everywhere).  us, tiles / streaming.  Up to eight rows streaming wins at every size where rows of W start on 32 bytes (m = 3, 1827 x 14336
// 17.2 / 12.8, 12496 x 16384 71 / 69; m = 8, 1024 x 14336 14.4 / 11.2, 8737 x 27904 83 / 81); where they do not, a copy of 64 bytes
// touches a third sector and large ones lose (16512 x 10072 62 / 69, 22016 x 11512 86 / 100, but 9216 x 872 9.7 / 7.1).
// Nine to sixteen rows bring twice the X: m = 16, 1283 x 19968 17.4 / 19.0, 1200 x 16384 16.0 / 15.2; m = 12, 2525 x 17584 23.1 / 24.9,
// 2330 x 15968 20.6 / 19.4, 4992 x 16128 34.2 / 32.3; m = 16, 5760 x 1024 9.5 / 7.6, 16384 x 6144 41.0 / 40.5, 24576 x 4096 41.0 / 42.0, 18944 x 4096
// 30.6 / 33.2, 19000 x 4096 34.2 / 31.9; m = 12, 21329 x 768 12.6 / 13.3; 2816 x 8792 (rows on 16 bytes) 16.8 / 18.1.
bool gemv_f16_stream_covers(const void* W, int64_t ldw, const void* X, int64_t ldx, int rows, int K, int m, int sm_count,
                            bool scratch) {
  if (m < 1 || m > 16 || rows < 1024 || K < 512 || (K & 7) || ((ldw ? ldw : K) & 7) || ((ldx ? ldx : K) & 7) ||
      (reinterpret_cast<uintptr_t>(W) & 15) || (reinterpret_cast<uintptr_t>(X) & 15))
    return false;
  if (m <= 2 || !scratch) return true;
  const int64_t work = (int64_t)rows * K;
  const bool on_sectors = ((ldw ? ldw : K) & 15) == 0 && (reinterpret_cast<uintptr_t>(W) & 31) == 0;
  if (!on_sectors && (work > (m > 8 ? 12 << 20 : 64 << 20) || (rows < 24 * sm_count && K > (m > 8 ? 8192 : 10240)))) return false;
  if (m <= 8) return K <= 32768;
  return rows <= 20480 && (rows <= 18000 || K >= 1024) && (rows > 4096 || K <= 16384);
}

int gemv_f16_launch(const helix_cfg_t* cfg, const void* W, int64_t ldw, const void* X, int64_t ldx, void* Y,
                    int64_t ldy, int64_t ldy_inner, int rows, int K, int m, void* ws, size_t ws_bytes,
                    int sm_count, int order_mode, cudaStream_t stream, int64_t* launches) {
  struct Scope {
    explicit Scope(int v) { independent = v; }
    ~Scope() { independent = 0; }
  } scope(order_mode);
  if (!W || !X || !Y || rows <= 0 || K <= 0 || m <= 0 || m > 8) return HELIX_ERR_INVALID;
  if (ldw == 0) ldw = K;
  if (ldx == 0) ldx = K;
  if (ldy == 0) ldy = rows;
  if (ldy_inner == 0) ldy_inner = 1;
  if ((K & 7) || (ldw & 7) || (ldx & 7) || (reinterpret_cast<uintptr_t>(W) & 15) ||
      (reinterpret_cast<uintptr_t>(X) & 15))
    return HELIX_ERR_ALIGN;
  int split_k = (cfg && cfg->tile_m != 0 && cfg->split_k > 0) ? cfg->split_k
                                                              : gemv_f16_default_split(rows, K, sm_count);
  if (split_k > 1 && (K + split_k - 1) / split_k < 256) split_k = 1;
  const size_t need = gemv_f16_workspace_bytes(rows, m, split_k);
  const bool scratch = need > 0 && ws && ws_bytes >= need;
  if (!(cfg && cfg->tile_m != 0) && gemv_f16_streams(rows, K, m, split_k, scratch, sm_count)) {
    const int order = scratch && order_mode != 0 ? order_mode | kHoldNext : order_mode;
    return gemv_f16_stream_launch(W, ldw, X, ldx, Y, ldy, ldy_inner, rows, K, m, sm_count, order, stream, launches);
  }
  if (need > 0 && (!ws || ws_bytes < need)) {
    if (cfg && cfg->tile_m != 0 && cfg->split_k > 1) return HELIX_ERR_WORKSPACE;
    split_k = 1;  // automatic choice falls back to the workspace-free variant
  }
  const __half* w = static_cast<const __half*>(W);
  const __half* x = static_cast<const __half*>(X);
  __half* y = static_cast<__half*>(Y);
  float* part = static_cast<float*>(ws);
  // tile_n = rows per warp, load_group = loads in flight per row; defaults favour deep
  // memory-level parallelism (one pass over K per warp where K allows)
  int rpw = (cfg && cfg->tile_m != 0 && cfg->tile_n > 0) ? cfg->tile_n : (m <= 2 ? 2 : 1);
  int unroll = (cfg && cfg->tile_m != 0 && cfg->load_group > 0) ? cfg->load_group : (m <= 4 ? 4 : 2);
  if (m == 1) return launch_gemv_variant<1>(rpw, unroll, w, ldw, x, ldx, y, ldy, ldy_inner, part, rows, K, m, split_k, sm_count, stream, launches);
  if (m == 2) return launch_gemv_variant<2>(rpw, unroll, w, ldw, x, ldx, y, ldy, ldy_inner, part, rows, K, m, split_k, sm_count, stream, launches);
  if (m <= 4) return launch_gemv_variant<4>(rpw, unroll, w, ldw, x, ldx, y, ldy, ldy_inner, part, rows, K, m, split_k, sm_count, stream, launches);
  return launch_gemv_variant<8>(rpw, unroll, w, ldw, x, ldx, y, ldy, ldy_inner, part, rows, K, m, split_k, sm_count, stream, launches);
}

// ---------------------------------------------------------------------------------------------
// Split-K GEMV whose partial sums live in a buffer that is part of the library image.
//
// Some users of this library may not create device memory at the moment they need a GEMV: a
// decode loop that has handed every byte of HBM to its own pool cannot call cudaMalloc (it may
// fail, and it synchronises the device).  For them the fp32 partials of the split-K variant are
// kept in the fixed array below instead of a caller-supplied workspace.  Every GPU on which the
// library is loaded carries these 4 MiB until the process exits.
//
// In host code the name `g_gemv_static_scratch` is only a handle for the symbol, not an address
// the GPU understands; the device address is looked up once per device with
// cudaGetSymbolAddress (that device being current) and that pointer is what the kernels get.
constexpr size_t kGemvStaticFloats = size_t(1) << 20;  // 4 MiB of fp32 partials
static __device__ __align__(256) float g_gemv_static_scratch[kGemvStaticFloats];

size_t gemv_f16_static_capacity_floats() { return kGemvStaticFloats; }

// The set-up (symbol lookup) happens in the first call made on each device, so that first call
// should come before any stream capture.  All calls share the one array: it still holds
// the previous call's partials when a call starts, which is harmless because the kernel writes
// every slot the reduction reads before it is read (nothing has to start at zero) -- but two
// calls that may run on the GPU at the same time (different streams) would overwrite each
// other's partials, so callers must order them.  Nothing here allocates or frees memory.
int gemv_f16_static_launch(const void* W, int64_t ldw, const void* X, int64_t ldx, void* Y, int64_t ldy,
                           int64_t ldy_inner, int rows, int K, int m, int split_k, int sm_count,
                           cudaStream_t stream, int64_t* launches) {
  if (!W || !X || !Y || rows <= 0 || K <= 0 || m <= 0 || m > 8 || split_k < 1) return HELIX_ERR_INVALID;
  if (ldw == 0) ldw = K;
  if (ldx == 0) ldx = K;
  if (ldy == 0) ldy = rows;
  if (ldy_inner == 0) ldy_inner = 1;
  if ((K & 7) || (ldw & 7) || (ldx & 7) || (reinterpret_cast<uintptr_t>(W) & 15) ||
      (reinterpret_cast<uintptr_t>(X) & 15))
    return HELIX_ERR_ALIGN;
  if (split_k > 1 && (K + split_k - 1) / split_k < 256) split_k = 1;
  // a single pass over K (split_k = 1, asked for or after the clamp above) never touches the array
  if (split_k > 1 && (size_t)split_k * (size_t)m * (size_t)rows > kGemvStaticFloats) return HELIX_ERR_CAPACITY;

  static std::mutex mu;
  static float* scratch_on_device[64] = {nullptr};
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return HELIX_ERR_NODEVICE;
  float* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!scratch_on_device[dev]) {
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_gemv_static_scratch) != cudaSuccess || !p) return HELIX_ERR_CUDA;
      scratch_on_device[dev] = static_cast<float*>(p);
    }
    scratch = scratch_on_device[dev];
  }
  const __half* w = static_cast<const __half*>(W);
  const __half* x = static_cast<const __half*>(X);
  __half* y = static_cast<__half*>(Y);
  const int rpw = m <= 2 ? 2 : 1;
  const int unroll = m <= 4 ? 4 : 2;
  if (m == 1) return launch_gemv_variant<1>(rpw, unroll, w, ldw, x, ldx, y, ldy, ldy_inner, scratch, rows, K, m, split_k, sm_count, stream, launches);
  if (m == 2) return launch_gemv_variant<2>(rpw, unroll, w, ldw, x, ldx, y, ldy, ldy_inner, scratch, rows, K, m, split_k, sm_count, stream, launches);
  if (m <= 4) return launch_gemv_variant<4>(rpw, unroll, w, ldw, x, ldx, y, ldy, ldy_inner, scratch, rows, K, m, split_k, sm_count, stream, launches);
  return launch_gemv_variant<8>(rpw, unroll, w, ldw, x, ldx, y, ldy, ldy_inner, scratch, rows, K, m, split_k, sm_count, stream, launches);
}

}  // namespace helix
