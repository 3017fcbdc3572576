// True-fp32 GEMV for 1..8 right-hand sides: Y[i, r] = sum_k W[r, k] * X[i, k], FFMA only.
//
// Counterpart of the reference's mySGemvKernel_Stage4<float> (src_template/Ampere_FP32/
// gemv_template_fp32.cu:153-218), which no reference script builds: W is streamed once with 128-bit
// loads that bypass L1, several loads in flight per thread, each lane of a warp keeps one fused
// multiply-add chain per (row, right-hand side) over the K elements it owns, and the 32 partial sums meet
// in a warp-shuffle tree.  The order of that sum is fixed (lane chains over ascending k, then the xor tree
// 16, 8, 4, 2, 1), so the result is reproducible bit for bit; with split_k > 1 the K slices are summed in
// slice order by a second kernel.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace helix {

template <int MRHS, int RPW, int UNROLL>
__global__ void __launch_bounds__(256)
gemv_f32_kernel(const float* __restrict__ W, int64_t ldw, const float* __restrict__ X, int64_t ldx,
                float* __restrict__ Y, int64_t ldy, int64_t ldy_inner, float* __restrict__ partial, int rows, int K,
                int m, int split_k, int k_per_split) {
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
    const float* wrow[RPW];
#pragma unroll
    for (int r = 0; r < RPW; ++r) wrow[r] = W + (int64_t)min(r0 + r, rows - 1) * ldw;

    // a lane owns the four consecutive elements at k0 + 4 * lane of every 128-element stretch
    for (int k0 = k_begin + lane * 4; k0 < k_end; k0 += 128 * UNROLL) {
      uint4 wv[UNROLL][RPW];
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const int k = k0 + u * 128;
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
          if (k < k_end) wv[u][r] = ldg_stream_16(wrow[r] + k);
          else wv[u][r] = make_uint4(0u, 0u, 0u, 0u);
        }
      }
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const int k = k0 + u * 128;
        if (k < k_end) {
#pragma unroll
          for (int i = 0; i < MRHS; ++i) {
            if (i < m) {
              const float4 xv = __ldg(reinterpret_cast<const float4*>(X + (int64_t)i * ldx + k));
#pragma unroll
              for (int r = 0; r < RPW; ++r) {
                acc[r][i] = fmaf(__uint_as_float(wv[u][r].x), xv.x, acc[r][i]);
                acc[r][i] = fmaf(__uint_as_float(wv[u][r].y), xv.y, acc[r][i]);
                acc[r][i] = fmaf(__uint_as_float(wv[u][r].z), xv.z, acc[r][i]);
                acc[r][i] = fmaf(__uint_as_float(wv[u][r].w), xv.w, acc[r][i]);
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
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < RPW; ++r) {
        if (r0 + r < rows) {
#pragma unroll
          for (int i = 0; i < MRHS; ++i) {
            if (i < m) {
              if (split_k == 1) Y[(int64_t)i * ldy + (int64_t)(r0 + r) * ldy_inner] = acc[r][i];
              else partial[((int64_t)ks * m + i) * rows + r0 + r] = acc[r][i];
            }
          }
        }
      }
    }
  }
}

// Streaming kernel, the library's choice where K is not cut: one persistent CTA per SM with an equal share of the rows.
// A warp owns RB rows at a time over the whole of K (the order of its sums is the one stated above), and every lane
// streams its 16-byte chunks through a private FIFO of 12 slots in shared memory (cp.async; a lane reads only
// what it copied, so there are no barriers): 96 KB per SM in flight however many registers the sums take.  The grid of
// the kernel above is 512 CTAs for 8192 rows, i.e. four on some SMs and three on others.
constexpr int kStream32Threads = 512;
constexpr int kStream32Loads = 4;
constexpr int kStream32Groups = 3;
constexpr int kStream32RingBytes = kStream32Threads * kStream32Loads * kStream32Groups * 16;

template <int MRHS, int RB>
__global__ void __launch_bounds__(kStream32Threads, MRHS <= 2 ? 2 : 1)
gemv_f32_stream_kernel(const float* __restrict__ W, int64_t ldw, const float* X, int64_t ldx, float* Y, int64_t ldy,
                       int64_t ldy_inner, int rows, int K, int m, int kw) {
  constexpr int U = kStream32Loads / RB;            // 128-element stretches of K per group
  constexpr int kWarps = kStream32Threads / 32;
  constexpr int kStep = U * 128;                    // elements of K per group
  extern __shared__ __align__(16) unsigned char stream_smem[];
  __shared__ float part[kWarps][RB * MRHS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r_begin = static_cast<int>(static_cast<int64_t>(rows) * blockIdx.x / gridDim.x);
  const int r_end = static_cast<int>(static_cast<int64_t>(rows) * (blockIdx.x + 1) / gridDim.x);
  const int blocks = (r_end - r_begin + RB - 1) / RB;
  const uint32_t slot0 = smem_u32(stream_smem) + tid * 16;

  // kw warps share a row block, taking its groups of K in turn (kw = 1: the order stated at the top of this file)
  const int rw = kWarps / kw, kwi = warp % kw, rwi = warp / kw;
  int pb = rwi, pk = kwi * kStep, pslot = 0;        // next group to issue: row block, first element
  // one group per warp to the L2 ahead of the wait, as in the fp16 kernel
#pragma unroll
  for (int r = 0; r < RB; ++r)
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (pk + u * 128 + lane * 4 < K && r_begin + pb * RB + r < r_end)
        prefetch_l2(W + static_cast<int64_t>(r_begin + pb * RB + r) * ldw + pk + u * 128 + lane * 4);
  griddep_wait();
  griddep_launch_dependents();
  auto issue = [&]() {
    if (pb < blocks && pk < K) {
      const int row = r_begin + pb * RB;
      const float* src = W + static_cast<int64_t>(row) * ldw + pk + lane * 4;
#pragma unroll
      for (int r = 0; r < RB; ++r)
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const bool in = pk + u * 128 + lane * 4 < K && row + r < r_end;
          cp_async_16_zfill(slot0 + (pslot * kStream32Loads + r * U + u) * kStream32Threads * 16,
                            in ? src + r * ldw + u * 128 : W, in);
        }
      pk += kw * kStep;
      if (pk >= K) { pk = kwi * kStep; pb += rw; }
    }
    cp_async_commit();
    if (++pslot == kStream32Groups) pslot = 0;
  };
#pragma unroll
  for (int i = 0; i < kStream32Groups; ++i) issue();

  int cslot = 0;
  for (int sb = 0; sb < blocks; sb += rw) {
    const int b = sb + rwi;
    const int r0 = r_begin + b * RB;
    float acc[RB][MRHS];
#pragma unroll
    for (int r = 0; r < RB; ++r)
#pragma unroll
      for (int i = 0; i < MRHS; ++i) acc[r][i] = 0.0f;
    for (int k0 = b < blocks ? kwi * kStep : K; k0 < K; k0 += kw * kStep) {
      // X first: all loads of a group are independent (a right-hand side that does not exist reads the last one)
      float4 xv[U][MRHS];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = min(k0 + u * 128 + lane * 4, K - 4);
#pragma unroll
        for (int i = 0; i < MRHS; ++i) xv[u][i] = *reinterpret_cast<const float4*>(X + min(i, m - 1) * ldx + k);
      }
      cp_async_wait<kStream32Groups - 1>();
      float4 wv[RB][U];
#pragma unroll
      for (int r = 0; r < RB; ++r)
#pragma unroll
        for (int u = 0; u < U; ++u)
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(wv[r][u].x), "=f"(wv[r][u].y), "=f"(wv[r][u].z), "=f"(wv[r][u].w)
                       : "r"(slot0 + (cslot * kStream32Loads + r * U + u) * kStream32Threads * 16)
                       : "memory");
      issue();
      if (++cslot == kStream32Groups) cslot = 0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (k0 + u * 128 + lane * 4 < K) {
#pragma unroll
          for (int i = 0; i < MRHS; ++i)
#pragma unroll
            for (int r = 0; r < RB; ++r) {
              acc[r][i] = fmaf(wv[r][u].x, xv[u][i].x, acc[r][i]);
              acc[r][i] = fmaf(wv[r][u].y, xv[u][i].y, acc[r][i]);
              acc[r][i] = fmaf(wv[r][u].z, xv[u][i].z, acc[r][i]);
              acc[r][i] = fmaf(wv[r][u].w, xv[u][i].w, acc[r][i]);
            }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < RB; ++r)
#pragma unroll
      for (int i = 0; i < MRHS; ++i) {
        float v = acc[r][i];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (kw > 1) {
          if (lane == 0) part[warp][r * MRHS + i] = v;
        } else if (lane == 0 && r0 + r < r_end && i < m) {
          Y[i * ldy + static_cast<int64_t>(r0 + r) * ldy_inner] = v;
        }
      }
    if (kw > 1) {                                   // the shares of K in the order of the warps
      __syncthreads();
      for (int o = tid; o < rw * RB * MRHS; o += kStream32Threads) {
        const int grp = o / (RB * MRHS), e = o - grp * (RB * MRHS), r = e / MRHS, i = e - r * MRHS;
        const int row = r_begin + (sb + grp) * RB + r;
        if (row < r_end && i < m) {
          float sum = 0.0f;
          for (int q = 0; q < kw; ++q) sum += part[grp * kw + q][e];
          Y[i * ldy + static_cast<int64_t>(row) * ldy_inner] = sum;
        }
      }
      __syncthreads();
    }
  }
}

// Sums the split-K partials in slice order (deterministic).
__global__ void gemv_f32_splitk_reduce_kernel(const float* __restrict__ partial, float* __restrict__ Y, int64_t ldy,
                                              int64_t ldy_inner, int rows, int m, int split_k) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * m) return;
  const int i = idx / rows, r = idx - i * rows;
  float s = 0.0f;
  for (int ks = 0; ks < split_k; ++ks) s += partial[((int64_t)ks * m + i) * rows + r];
  Y[(int64_t)i * ldy + (int64_t)r * ldy_inner] = s;
}

size_t gemv_f32_workspace_bytes(int rows, int m, int split_k) {
  return split_k > 1 ? (size_t)split_k * m * rows * sizeof(float) : 0;
}

int gemv_f32_default_split(int rows, int K, int sm_count) {
  const int groups = (rows + 1) / 2;
  int split = 1;
  // as the fp16 kernel: beyond four warps per SM only very long rows are cut
  while (split < 16 && K / (split * 2) >= 1024 &&
         ((int64_t)groups * split < (int64_t)sm_count * 4 ||
          ((int64_t)groups * split < (int64_t)sm_count * 24 && K / (split * 2) >= 8192)))
    split *= 2;
  return split;
}

template <int MRHS, int RPW, int UNROLL>
static int launch_gemv32(const float* W, int64_t ldw, const float* X, int64_t ldx, float* Y, int64_t ldy,
                         int64_t ldy_inner, float* partial, int rows, int K, int m, int split_k, int sm_count,
                         cudaStream_t stream, int64_t* launches) {
  const int row_groups = (rows + RPW - 1) / RPW;
  const int warps = 8;
  int blocks = std::min((row_groups + warps - 1) / warps, sm_count * 8);
  int k_per_split = (K + split_k - 1) / split_k;
  k_per_split = (k_per_split + 127) / 128 * 128;
  gemv_f32_kernel<MRHS, RPW, UNROLL><<<dim3(blocks, split_k), warps * 32, 0, stream>>>(
      W, ldw, X, ldx, Y, ldy, ldy_inner, partial, rows, K, m, split_k, k_per_split);
  ++*launches;
  if (split_k > 1) {
    const int n = rows * m;
    gemv_f32_splitk_reduce_kernel<<<(n + 255) / 256, 256, 0, stream>>>(partial, Y, ldy, ldy_inner, rows, m, split_k);
    ++*launches;
  }
  return cudaGetLastError() == cudaSuccess ? HELIX_OK : HELIX_ERR_CUDA;
}

template <int MRHS, int RB>
static int launch_stream32(const float* W, int64_t ldw, const float* X, int64_t ldx, float* Y, int64_t ldy,
                           int64_t ldy_inner, int rows, int K, int m, int kw, int sm_count, cudaStream_t stream,
                           int64_t* launches) {
  auto kern = gemv_f32_stream_kernel<MRHS, RB>;
  static thread_local int attr_dev = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (attr_dev != dev) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kStream32RingBytes) != cudaSuccess)
      return HELIX_ERR_CUDA;
    // one CTA of these per SM: what its FIFOs leave of the shared memory is L1 for X, which every row block reads again
    if (MRHS > 2 && cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 50) != cudaSuccess)
      return HELIX_ERR_CUDA;
    attr_dev = dev;
  }
  if (launch_overlapped(kern, dim3(std::min(sm_count, rows)), dim3(kStream32Threads), kStream32RingBytes, stream, W, ldw, X, ldx,
                        Y, ldy, ldy_inner, rows, K, m, kw) != cudaSuccess)
    return HELIX_ERR_CUDA;
  ++*launches;
  return HELIX_OK;
}

// Which GEMVs without a configuration of their own the streaming kernel runs.  us, the kernel above / streaming:
static bool gemv_f32_streams(int rows, int K, int m, int split, int sm_count) {
  const int per_sm = (rows + sm_count - 1) / sm_count;
  if (m > 1 && K < 512) return false;                  // 10000 x 304, m = 2: 5.3 / 6.7
  if (split > 1) {
    if (rows < sm_count || K > 32768) return false;
    // cut only because K is very long: sharing it among warps pays with few rows, or where m makes the kernel above issue bound
    // (16384 long: m = 1, 3000 rows 44.6 / 40.6, 6000 66 / 72; m = 2, 1300 26.1 / 25.1, 2048 29.1 / 33.8; m = 3, 2048 43.8 / 42.0,
    // 3000 51 / 62; m = 5, 3000 70 / 62)
    return m >= 4 || per_sm <= (m == 1 ? 32 : m == 2 ? 10 : 16);
  }
  // Short rows: a warp takes whole rows, so its few loads per row leave its FIFO empty between rows (m = 1: 3000 x 256 2.8 / 2.9,
  // 6000 x 768 5.9 / 6.3, 6000 x 1500 10.1 / 9.5; m = 2: 4096 x 768 4.9 / 5.7; m = 5: 3000 x 768 6.2 / 6.5)
  if (m == 1) return per_sm <= 16 || (K >= 512 && per_sm <= 32) || K >= 1024;
  if (per_sm <= 32) return K >= 1024 || per_sm <= 16 || m == 3 || m == 4 || m == 8;
  // Several rows per warp: two of them do not earn the second right-hand side's reads back (m = 2: 4800 x 8192 35 / 50, 8192 x 8192
  // 45 / 51) but in the middle of the range (12000 x 2048 21.4 / 19.5); blocks of four should fill the CTA's 16 warps (m = 3:
  // 4800 x 4096, 9 blocks, 23.5 / 26.8; 8192 x 4096, 14 blocks, 38.3 / 30.3; 12000 x 4096, 21 blocks, 44.1 / 45.4), unless the kernel
  // above, whose cost follows m, spends more on a full set of right-hand sides (m = 4: 6000 x 2048 17.2 / 15.8, 6000 x 512 6.0 / 6.2;
  // m = 8: 6000 x 4096 36.6 / 33.4, 4800 x 1024 10.4 / 11.2).
  if (m == 2) return per_sm > 64 && K >= 1024 && K <= 4096;
  const int blocks = (per_sm + 3) / 4, turns = (blocks + 15) / 16;
  return blocks * 5 >= turns * 64 || (m == 4 && K >= 1024) || (m >= 7 && K >= 2048);
}

int gemv_f32_launch(const helix_cfg_t* cfg, const float* W, int64_t ldw, const float* X, int64_t ldx, float* Y,
                    int64_t ldy, int64_t ldy_inner, int rows, int K, int m, void* ws, size_t ws_bytes, int sm_count,
                    cudaStream_t stream, int64_t* launches) {
  if (!W || !X || !Y || rows <= 0 || K <= 0 || m <= 0 || m > 8) return HELIX_ERR_INVALID;
  if (ldw == 0) ldw = K;
  if (ldx == 0) ldx = K;
  if (ldy == 0) ldy = rows;
  if (ldy_inner == 0) ldy_inner = 1;
  if ((K & 3) || (ldw & 3) || (ldx & 3) || (reinterpret_cast<uintptr_t>(W) & 15) ||
      (reinterpret_cast<uintptr_t>(X) & 15))
    return HELIX_ERR_ALIGN;
  const bool own = cfg && cfg->tile_m != 0;
  int split_k = (own && cfg->split_k > 0) ? cfg->split_k : gemv_f32_default_split(rows, K, sm_count);
  if (split_k > 1 && (K + split_k - 1) / split_k < 128) split_k = 1;
  const size_t need = gemv_f32_workspace_bytes(rows, m, split_k);
  if (need > 0 && (!ws || ws_bytes < need)) {
    if (own && cfg->split_k > 1) return HELIX_ERR_WORKSPACE;
    split_k = 1;
  }
  if (!own && gemv_f32_streams(rows, K, m, split_k, sm_count)) {
    // rows per warp: as many as share one read of X while the warps of an SM still have a block each; where the library
    // would have cut K (few rows), the warps of a CTA share a row block's K instead
    const int per_sm = (rows + sm_count - 1) / sm_count;
#define HELIX_STREAM32(MR, RB, KW) \
  return launch_stream32<MR, RB>(W, ldw, X, ldx, Y, ldy, ldy_inner, rows, K, m, KW, sm_count, stream, launches)
    if (split_k > 1) {
      if (m == 1) HELIX_STREAM32(1, 2, 8);
      if (m == 2) HELIX_STREAM32(2, 2, 8);
      if (m <= 4) HELIX_STREAM32(4, 4, 16);
      HELIX_STREAM32(8, 4, 16);
    }
    if (m == 1) { if (per_sm > 32) HELIX_STREAM32(1, 2, 1); HELIX_STREAM32(1, 1, 1); }
    if (m == 2) { if (per_sm > 32) HELIX_STREAM32(2, 2, 1); HELIX_STREAM32(2, 1, 1); }
    if (m <= 4) { if (per_sm > 32) HELIX_STREAM32(4, 4, 1); HELIX_STREAM32(4, 2, 1); }
    if (per_sm > 32) HELIX_STREAM32(8, 4, 1);
    HELIX_STREAM32(8, 2, 1);
#undef HELIX_STREAM32
  }
  float* part = static_cast<float*>(ws);
  // tile_n = rows per warp (1 or 2), load_group = 16-byte loads in flight per row and thread (2, 4 or 8)
  const int rpw = (own && cfg->tile_n > 0) ? cfg->tile_n : (m <= 2 ? 2 : 1);
  const int unroll = (own && cfg->load_group > 0) ? cfg->load_group : (m <= 4 ? 4 : 2);
#define HELIX_GEMV32_CASE(MR, R, U)                                                                          \
  if (rpw == R && unroll == U)                                                                               \
    return launch_gemv32<MR, R, U>(W, ldw, X, ldx, Y, ldy, ldy_inner, part, rows, K, m, split_k, sm_count, stream, \
                                   launches);
#define HELIX_GEMV32_M(MR) \
  HELIX_GEMV32_CASE(MR, 1, 2) HELIX_GEMV32_CASE(MR, 1, 4) HELIX_GEMV32_CASE(MR, 1, 8) HELIX_GEMV32_CASE(MR, 2, 2) \
  HELIX_GEMV32_CASE(MR, 2, 4)
  if (m == 1) { HELIX_GEMV32_M(1) }
  else if (m == 2) { HELIX_GEMV32_M(2) }
  else if (m <= 4) { HELIX_GEMV32_M(4) }
  else { HELIX_GEMV32_M(8) }
#undef HELIX_GEMV32_M
#undef HELIX_GEMV32_CASE
  return HELIX_ERR_UNSUPPORTED;
}

}  // namespace helix
