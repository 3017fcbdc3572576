// Shared device helpers: bounded mbarrier waits, TMA / tcgen05 PTX wrappers.
// sm_100a only.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/helix_b200.h"

namespace helix {

// A wait that has not completed after this many nanoseconds gives up: the kernel
// stores HELIX_ERR_TIMEOUT in the status word and drains instead of spinning.
constexpr unsigned long long kWaitLimitNs = 2000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long global_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Division of a non-negative 31-bit integer by a divisor fixed at launch, as a multiply and a
// shift (round-up reciprocal: mul = ceil(2^(31 + ceil(log2 d)) / d), exact for 0 <= a < 2^31).
// A hardware-emulated integer division costs a single thread some 150 cycles, and the tile
// decoders below sit on the critical path between two tiles of a persistent CTA.
struct FastDiv {
  uint32_t d, mul, shr;
};
inline FastDiv make_fastdiv(int divisor) {
  FastDiv f{static_cast<uint32_t>(divisor > 0 ? divisor : 1), 0u, 0u};
  if (f.d > 1) {
    uint32_t lg = 0;
    while ((1ull << lg) < f.d) ++lg;
    const uint32_t p = 31 + lg;
    f.mul = static_cast<uint32_t>(((1ull << p) + f.d - 1) / f.d);
    f.shr = p - 32;
  }
  return f;
}
__device__ __forceinline__ int fast_div(int a, const FastDiv& f) {
  return f.d == 1 ? a : static_cast<int>(__umulhi(static_cast<uint32_t>(a), f.mul) >> f.shr);
}
__device__ __forceinline__ void fast_divmod(int a, const FastDiv& f, int& q, int& r) {
  q = fast_div(a, f);
  r = a - q * static_cast<int>(f.d);
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// The same test, but the thread may be parked by the hardware for up to `hint_ns` while the phase is incomplete
// (it issues nothing meanwhile, unlike a polling loop).
__device__ __forceinline__ bool mbar_try_wait_parked(uint64_t* bar, uint32_t parity, uint32_t hint_ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}
// Bounded wait.  Returns false (after recording the failure) when the limit ran out or another role of
// this CTA already gave up.  While the phase is incomplete the thread is parked by the hardware (a
// try_wait with a suspend-time hint) instead of polling: a polling warp competes with the MMA-issuing
// warp for its scheduler and for the shared-memory pipe (measured 3-7 % on narrow-tile kernels).
// One rolled loop: there are dozens of waits in a kernel, and code that a launch of a few us fetches for nothing costs it time.
__device__ __forceinline__ bool mbar_wait_limit(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                int* status_dev, unsigned long long limit_ns) {
  unsigned long long t0 = 0;
#pragma unroll 1
  for (int i = 0;; ++i) {
    if (mbar_try_wait_parked(bar, parity, 20000u)) return true;
    if ((i & 7) != 7) continue;
    if (*abort_flag) return false;
    const unsigned long long now = global_timer_ns();
    if (t0 == 0) t0 = now;
    if (now - t0 > limit_ns) {
      *abort_flag = 1;
      if (status_dev) atomicExch(status_dev, (int)HELIX_ERR_TIMEOUT);
      return false;
    }
  }
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          int* status_dev) {
  return mbar_wait_limit(bar, parity, abort_flag, status_dev, kWaitLimitNs);
}

// ---------------------------------------------------------------- proxies / fences
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// ---------------------------------------------------------------- TMA (no multicast anywhere)
__device__ __forceinline__ void tma_prefetch_desc(const void* desc) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(desc)) : "memory");
}
// 3-D tiled load: coordinates (x = innermost element index, y = row, z = batch).
// x * sizeof(element) must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const void* desc, uint64_t* bar, int x, int y,
                                            int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
      "[%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(desc)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// 4-D im2col load from an NHWC tensor (map dimensions C, W, H, N): `pixels-per-column` pixels
// starting at base pixel (w, h, n) and walking the map's bounding box in W, then H, then N with
// the map's traversal strides; each pixel contributes `channels-per-pixel` channels from c, read
// at (w + off_w, h + off_h).  Pixels outside the tensor arrive as zeros and still count towards
// the transaction bytes.  c * sizeof(element) must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_im2col_4d(void* smem_dst, const void* desc, uint64_t* bar, int c, int w,
                                                   int h, int n, uint16_t off_w, uint16_t off_h) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, "
      "%6}], [%2], {%7, %8};" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(desc)), "r"(smem_u32(bar)), "r"(c), "r"(w), "r"(h), "r"(n), "h"(off_w),
      "h"(off_h)
      : "memory");
}

// ---------------------------------------------------------------- cp.async (16-byte, zero-fill)
__device__ __forceinline__ void cp_async_16_zfill(uint32_t smem_dst, const void* gsrc, bool valid) {
  const int src_bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_dst), "l"(gsrc), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Wait until at most n (0..6) of this thread's cp.async groups are still in flight.
__device__ __forceinline__ void cp_async_wait_dyn(int n) {
  switch (n) {
    case 0: cp_async_wait<0>(); break;
    case 1: cp_async_wait<1>(); break;
    case 2: cp_async_wait<2>(); break;
    case 3: cp_async_wait<3>(); break;
    case 4: cp_async_wait<4>(); break;
    case 5: cp_async_wait<5>(); break;
    default: cp_async_wait<6>(); break;
  }
}

// Arrival on `bar` that fires when all cp.async copies this thread issued before it have
// completed; does not raise the barrier's pending count, so it must be part of the init count.
__device__ __forceinline__ void cp_async_mbar_arrive_noinc(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// ---------------------------------------------------------------- tcgen05 / TMEM
template <int NCOLS>
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(NCOLS)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <int NCOLS>
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(NCOLS) : "memory");
}

// Shared-memory matrix descriptor of a K-major tile stored as rows of 128 bytes with the
// 128-byte swizzle (what a TMA box {64 halves, rows} with SWIZZLE_128B writes): groups of 8
// rows are 1024 bytes apart (stride byte offset); the leading byte offset is unused for
// swizzled K-major operands.  Bits: [0,14) address>>4, [16,30) LBO>>4, [32,46) SBO>>4,
// [46,48) version = 1, [61,64) layout = 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>(1) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

// The same for rows of 64 bytes (a box of 32 halves with SWIZZLE_64B: groups of 8 rows are 512 bytes apart, layout = 4) or of
// 32 bytes (16 halves with SWIZZLE_32B: 256 bytes, layout = 6).
template <int ROW_BYTES>
__device__ __forceinline__ uint64_t umma_desc_narrow(uint32_t smem_addr) {
  static_assert(ROW_BYTES == 64 || ROW_BYTES == 32, "swizzled rows");
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>(1) << 16;
  d |= static_cast<uint64_t>(8 * ROW_BYTES >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(ROW_BYTES == 64 ? 4 : 6) << 61;
  return d;
}

// Instruction descriptor of tcgen05.mma.kind::f16 with fp16 A/B (both K-major) and fp32 D.
// Bits: [4,6) D format (1 = f32), [7,10) A format (0 = f16), [10,13) B format, 15/16 majors
// (0 = K), [17,23) N>>3, [24,29) M>>4.
__host__ __device__ constexpr uint32_t umma_idesc_f16(int m, int n) {
  return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

__device__ __forceinline__ void umma_f16_ss(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                            bool accumulate) {
  const uint32_t acc = accumulate ? 1u : 0u;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(acc)
      : "memory");
}
// The same two instructions for a warp that walks its issue loop convergently: every lane executes the
// statement, one elected lane issues.  With all loop state warp-uniform the compiler keeps descriptors and
// addresses in uniform registers; a loop run by one lane of a diverged warp pays a register-to-uniform move per
// operand instead (measured on a 64-deep slab of four MMAs plus commit: 398 -> 284 cycles of issue time).
__device__ __forceinline__ void umma_f16_ss_elect(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                  bool accumulate) {
  const uint32_t acc = accumulate ? 1u : 0u;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void umma_commit_elect(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar))
      : "memory");
}
// mbarrier arrival once every previously issued tcgen05.mma of this thread has completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp receives row (lane base + i).
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// 16 lanes x 64 columns as fragments of 8 x 8: in r[4 i ... 4 i + 3] thread t of the warp receives columns 8 i + 2 (t % 4) and
// the next one of row t / 4 (r[4 i], r[4 i + 1]) and of row t / 4 + 8.
__device__ __forceinline__ void tmem_ld_16x256b_x8(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ---------------------------------------------------------------- TMA store (shared -> global)
// 3-D tiled store of one box; elements outside the tensor are not written.  x * sizeof(element)
// must be a multiple of 16 bytes and no coordinate may be negative.
__device__ __forceinline__ void tma_store_3d(const void* desc, const void* smem_src, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
          reinterpret_cast<uint64_t>(desc)),
      "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// until the bulk stores committed by this thread have finished READING shared memory
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// until at most one committed bulk store of this thread is still reading shared memory
__device__ __forceinline__ void tma_store_wait_read_1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }
// until they have completed altogether
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ---------------------------------------------------------------- epilogue staging
// A warp's 32 rows (lane = row) x 64 accumulator columns, rounded once to fp16, into a 128-byte-swizzled box of 32 x 128
// bytes in shared memory (the layout a TMA store with SWIZZLE_128B reads).
__device__ __forceinline__ void stage_rows_f16(uint32_t row_base, const uint32_t (&lo)[32], const uint32_t (&hi)[32],
                                               int lane) {
#pragma unroll
  for (int ch = 0; ch < 8; ++ch) {
    const uint32_t* src = ch < 4 ? &lo[ch * 8] : &hi[(ch - 4) * 8];
    __half2 h0 = __floats2half2_rn(__uint_as_float(src[0]), __uint_as_float(src[1]));
    __half2 h1 = __floats2half2_rn(__uint_as_float(src[2]), __uint_as_float(src[3]));
    __half2 h2 = __floats2half2_rn(__uint_as_float(src[4]), __uint_as_float(src[5]));
    __half2 h3 = __floats2half2_rn(__uint_as_float(src[6]), __uint_as_float(src[7]));
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_base + ((ch ^ (lane & 7)) << 4)),
                 "r"(*reinterpret_cast<uint32_t*>(&h0)), "r"(*reinterpret_cast<uint32_t*>(&h1)),
                 "r"(*reinterpret_cast<uint32_t*>(&h2)), "r"(*reinterpret_cast<uint32_t*>(&h3))
                 : "memory");
  }
}
// The transposed box: 64 accumulator columns become 64 rows of 128 bytes, `chunk` ... chunk + 3 of whose eight 16-byte
// chunks are this warp's 32 rows (lo: rows 0 ... 15, hi: 16 ... 31, as tmem_ld_16x256b_x8 delivers them).  A transposing
// stmatrix writes 8 rows x 4 chunks without a bank conflict.
__device__ __forceinline__ void stage_columns_f16(uint32_t box, const uint32_t (&lo)[32], const uint32_t (&hi)[32], int chunk,
                                                  int lane) {
  auto pack = [](uint32_t a, uint32_t b) {
    const __half2 h = __floats2half2_rn(__uint_as_float(a), __uint_as_float(b));
    return *reinterpret_cast<const uint32_t*>(&h);
  };
  const uint32_t dst = box + (lane & 7) * 128 + (((chunk + (lane >> 3)) ^ (lane & 7)) << 4);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(dst + i * 1024),
                 "r"(pack(lo[4 * i], lo[4 * i + 1])), "r"(pack(lo[4 * i + 2], lo[4 * i + 3])),
                 "r"(pack(hi[4 * i], hi[4 * i + 1])), "r"(pack(hi[4 * i + 2], hi[4 * i + 3]))
                 : "memory");
}
// Such a box to rows of C that TMA cannot store (a leading dimension or base that is no multiple of 16 bytes): row by row
// with the lanes along the columns, 4 bytes each, shifted by one element where a row starts on an odd one.  (A lane per row
// writes 2 bytes to 32 different lines per instruction: 2595 x 1685 x 200 took 50.8 us instead of 19.)  dst: row 0, column
// 0 of the block; `rows` and `cols` of it exist.
__device__ __forceinline__ void drain_box_any(uint32_t box, __half* dst, int64_t ldc, int rows, int cols) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  auto element = [&](int r, int e) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(box + r * 128 + (((e >> 3) ^ (r & 7)) << 4) + (e & 7) * 2) : "memory");
    return v;
  };
#pragma unroll 4
  for (int r = 0; r < rows; ++r) {
    __half* d = dst + r * ldc;
    const int odd = static_cast<int>(reinterpret_cast<uintptr_t>(d) >> 1) & 1;
    const int e = 2 * lane + odd;
    const uint16_t v0 = element(r, e), v1 = element(r, (e + 1) & 63);
    if (e + 1 < cols) *reinterpret_cast<uint32_t*>(d + e) = static_cast<uint32_t>(v0) | static_cast<uint32_t>(v1) << 16;
    else if (e < cols) *reinterpret_cast<uint16_t*>(d + e) = v0;
    if (odd && lane == 0) *reinterpret_cast<uint16_t*>(d) = element(r, 0);
  }
  __syncwarp();   // the box is free again
}

// ---------------------------------------------------------------- named barriers (sub-CTA groups)
// All `nthreads` threads of the group (whole warps) must call these the same number of times.
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
// Barrier that also tells every thread whether `pred` held for all of them.
__device__ __forceinline__ bool named_bar_and(int id, int nthreads, bool pred) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %3, 0;\n\t"
      "bar.red.and.pred p, %1, %2, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(id), "r"(nthreads), "r"(static_cast<uint32_t>(pred))
      : "memory");
  return r != 0;
}

// ---------------------------------------------------------------- programmatic dependent launch
// launch_dependents: the next kernel on the stream may start being scheduled (when it was launched
// with the programmatic-serialization attribute).  wait: returns once every kernel this one depends
// on has completed and its memory is visible.  Both are no-ops for a plain launch.
// A kernel of an ordered launch calls launch_dependents after its wait: its successor may be flagged not to wait itself,
// and then starts -- and reads -- with nothing behind it but this call, while the caller only vouches for THIS launch
// not writing its operands.  Whatever was queued earlier must be complete by then.  (Nothing is lost by it: until the
// predecessor is complete the successor's CTAs could only sit beside ours.)  One exception: a GEMM whose next kernel is its own stream-K
// fix-up, which is never flagged, calls it ahead of its wait (gemm_f16_tc.cu, fixup_next).  Flagged launches call it at entry, so that
// a run of them overlaps as a whole.  A step of sixteen one-token GEMVs with static weights takes 236.8 us that way and
// 244.1 when every one of them holds its successor back: the launch after the next fills its FIFOs while this one's last rows drain.
__device__ __forceinline__ void griddep_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Reads a kernel's parameters once: their lines are cold in every launch, and a role that meets them one after the other
// behind griddep_wait() pays for each (2300 cycles from the wait to the first load in the GEMM kernel).
template <typename P>
__device__ __forceinline__ void touch_params(const P& p) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(&p);
#pragma unroll
  for (unsigned i = 0; i < sizeof(P) / 4; i += 8) asm volatile("" ::"r"(w[i]));
}

// Asks the L2 for a line before griddep_wait().  Nothing is read: should the predecessor still write there, the load after the wait
// sees what it wrote (the L2 is where both meet).
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void tma_prefetch_3d(const void* desc, int x, int y, int z) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(reinterpret_cast<uint64_t>(desc)), "r"(x),
               "r"(y), "r"(z)
               : "memory");
}

// ---------------------------------------------------------------- misc loads
__device__ __forceinline__ uint4 ldg_stream_16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

}  // namespace helix
