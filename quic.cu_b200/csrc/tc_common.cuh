// Shared pieces of the tcgen05 kernels: mbarrier waits with a time limit, UMMA
// descriptors (K-major, 128-byte swizzle), TMA 2-D loads and tensor-map creation.
#pragma once
#include <cuda.h>

#include "decode_kernels.cuh"

namespace quic {

constexpr int kTileN = 128;   // rows of the weight-side tile (UMMA M)
constexpr int kBlockK = 64;   // k per swizzle atom: 64 fp16 = one 128-byte swizzle row (a GEMM stage holds two)
constexpr uint32_t kWaitLimitUs = 2000000;  // a bounded wait gives up after two seconds

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
// A probe that may sleep for 20 us: fewer of them beside the CTA's other roles (prefill of 16 x 2048 tokens 30.35 -> 30.13 ms).
__device__ __forceinline__ bool mbar_try_long(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity), "r"(20000u)
      : "memory");
  return done != 0;
}
// Time in units of 1.024 us.
__device__ __forceinline__ uint32_t clock_us() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return (uint32_t)(t >> 10);
}
// Bounded wait for the phase with the given parity; false after `limit_us`.  A probe sleeps until the phase is complete
// or some us are over; the clock is read by a wait whose first probe has failed.  (A limit in probes is none: 2^22 of them were
// 16.6 s where nothing came, and with a limit of probes of 4 us each the tests of late stages failed.)
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit_us = kWaitLimitUs) {
  bool done = mbar_try(bar, parity);
  if (!done) {
    const uint32_t t0 = clock_us();
    do done = mbar_try_long(bar, parity);
    while (!done && clock_us() - t0 < limit_us);
  }
  return done;
}
// A wait for what other roles of the CTA bring about: it also ends when one of those has given up.
__device__ __forceinline__ bool mbar_wait_unless(uint32_t bar, uint32_t parity, const volatile int* given_up, uint32_t limit_us) {
  bool done = mbar_try(bar, parity);
  if (!done) {
    const uint32_t t0 = clock_us();
    do done = mbar_try_long(bar, parity);
    while (!done && *given_up == 0 && clock_us() - t0 < limit_us);
  }
  return done;
}
__device__ __forceinline__ void pause_us(uint32_t us) {
  const uint32_t t0 = clock_us();
  while (clock_us() - t0 < us) __nanosleep(1000);
}
// The same wait for roles that are many warps wide and not on the critical path of the MMA
// issue: sleeps between probes so the probes do not crowd the issuing thread's instructions
// out of the shared-memory pipeline.
__device__ __forceinline__ bool mbar_wait_relaxed(uint32_t bar, uint32_t parity, uint32_t sleep_ns, uint32_t limit_us,
                                                  const volatile int* given_up) {
  bool done = mbar_try(bar, parity);
  if (!done) {
    const uint32_t t0 = clock_us();
    do {
      __nanosleep(sleep_ns);
      done = mbar_try(bar, parity);
    } while (!done && *given_up == 0 && clock_us() - t0 < limit_us);
  }
  return done;
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// N (2, 4 or a multiple of 8) consecutive fp32 columns of this thread's TMEM lane: all loads in
// flight, one wait
template <int N>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, float (&v)[N]) {
  static_assert(N == 2 || N == 4 || (N % 8 == 0 && N >= 8), "2, 4 or whole 8-column loads");
  uint32_t r[N];
  if constexpr (N == 2) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr));
  } else if constexpr (N == 4) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
  } else {
#pragma unroll
    for (int q = 0; q < N / 8; ++q)
      asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(r[8 * q + 0]), "=r"(r[8 * q + 1]), "=r"(r[8 * q + 2]), "=r"(r[8 * q + 3]), "=r"(r[8 * q + 4]),
                     "=r"(r[8 * q + 5]), "=r"(r[8 * q + 6]), "=r"(r[8 * q + 7])
                   : "r"(taddr + 8u * q));
  }
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = __uint_as_float(r[i]);
}

// N blocks of 16 lanes x 8 fp32 columns: a thread has columns 2 (t % 4) and + 1 of lanes t / 4 (v[.][0], v[.][1]) and t / 4 + 8
template <int N>
__device__ __forceinline__ void tmem_ld_16x8(uint32_t taddr, float (&v)[N][4]) {
  uint32_t r[4 * N];
#pragma unroll
  for (int q = 0; q < N; ++q)
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[4 * q]), "=r"(r[4 * q + 1]), "=r"(r[4 * q + 2]), "=r"(r[4 * q + 3])
                 : "r"(taddr + 8u * q));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 4 * N; ++i) v[i / 4][i % 4] = __uint_as_float(r[i]);
}
// a block here and one there, one wait
__device__ __forceinline__ void tmem_ld_16x8_two(uint32_t ta, uint32_t tb, float (&a)[4], float (&b)[4]) {
  uint32_t r[8];
#pragma unroll
  for (int q = 0; q < 2; ++q)
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[4 * q]), "=r"(r[4 * q + 1]), "=r"(r[4 * q + 2]), "=r"(r[4 * q + 3])
                 : "r"(q == 0 ? ta : tb));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    a[i] = __uint_as_float(r[i]);
    b[i] = __uint_as_float(r[4 + i]);
  }
}

// 32 consecutive fp32 columns of this thread's TMEM lane: two loads in flight, one wait
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
#pragma unroll
  for (int q = 0; q < 2; ++q)
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[16 * q + 0]), "=r"(r[16 * q + 1]), "=r"(r[16 * q + 2]), "=r"(r[16 * q + 3]), "=r"(r[16 * q + 4]),
          "=r"(r[16 * q + 5]), "=r"(r[16 * q + 6]), "=r"(r[16 * q + 7]), "=r"(r[16 * q + 8]), "=r"(r[16 * q + 9]),
          "=r"(r[16 * q + 10]), "=r"(r[16 * q + 11]), "=r"(r[16 * q + 12]), "=r"(r[16 * q + 13]),
          "=r"(r[16 * q + 14]), "=r"(r[16 * q + 15])
        : "r"(taddr + 16u * q));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// K-major, 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);  // start address
  d |= (uint64_t)1 << 16;                    // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;                    // descriptor version of this architecture
  d |= (uint64_t)2 << 61;                    // SWIZZLE_128B
  return d;
}
// kind::f16, fp16 x fp16 -> fp32, both operands K-major, M = m, N = n.
__device__ __forceinline__ uint32_t umma_idesc_f16(int m, int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ uint32_t umma_idesc_f16(int n) { return umma_idesc_f16(kTileN, n); }
// One lane of a converged warp.  An MMA issued under it, with descriptors that are advanced by adds, takes 25-50 clocks of
// the issuing warp (M = 64, N = 16 .. M = 128, N = 64); under `lane == 0`, 69.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
// Records that a wait gave up in an error word of the device or of page-locked host memory; an earlier record stays.
__device__ __forceinline__ void tc_report(int* status, int code) {
  volatile int* const word = status;
  if (*word == 0) *word = code;
}
// The way out of a CTA in which a wait gave up: nobody may have waited for its last MMAs and copies, which use its shared memory
// and its tensor memory.  All threads, after the barrier that every role has reached; `issuer`: the thread that issued
// the MMAs; `bar`: a barrier for one arrival, not in use.  The MMAs are waited for; a copy, which waits for nothing, lands within
// microseconds of its request and is given a millisecond.
__device__ __forceinline__ void drain_failed_warp(bool issuer, uint32_t bar) {  // (where one warp issues and frees)
  if (issuer) {
    umma_commit(bar);
    mbar_wait(bar, 0);
    tc_fence_after();
    pause_us(1000);
  }
  __syncwarp();
  tc_fence_before();
}
__device__ __forceinline__ void drain_failed(bool issuer, uint32_t bar) {
  drain_failed_warp(issuer, bar);
  __syncthreads();
  tc_fence_after();
}

// Byte offset of 16-byte chunk c (0..7) of row r inside a swizzled tile.
__device__ __forceinline__ uint32_t sw128_offset(int r, int c) { return r * 128 + ((c ^ (r & 7)) << 4); }

// Untiled bulk copy global -> shared (both addresses 16-byte aligned, size a multiple of 16),
// completing `bytes` of the barrier's transaction count.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// Brings a tensor map (a kernel parameter) into the descriptor cache ahead of its first copy, so
// that copy does not wait for the descriptor fetch.
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// 2-D tiled TMA load into this CTA's shared memory; completion is counted in bytes on `bar`.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

// ---- host side ----------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime's driver entry point lookup (no link-time
// dependency on the driver library).
inline EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// Tiled map of a tensor of `rank` dimensions, innermost first; elements past the end read as zero.  A thread that has
// made no runtime call yet has no current context, and this may be its first: it is then given the device's.
inline int make_tiled_map(CUtensorMap* map, CUtensorMapDataType type, int rank, const void* ptr, const cuuint64_t* dims,
                          const cuuint64_t* strides, const cuuint32_t* box, CUtensorMapSwizzle swizzle,
                          CUtensorMapL2promotion promotion) {
  EncodeTiledFn fn = encode_tiled();
  QUIC_REQUIRE(fn != nullptr, QUIC_E_CUDA, "tensor map: cuTensorMapEncodeTiled is not available");
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  auto encode = [&] {
    return fn(map, type, (cuuint32_t)rank, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
              promotion, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = encode();
  if (r != CUDA_SUCCESS) {
    int dev = 0;
    QUIC_CUDA(cudaGetDevice(&dev));
    QUIC_CUDA(cudaSetDevice(dev));
    r = encode();
  }
  QUIC_REQUIRE(r == CUDA_SUCCESS, QUIC_E_CUDA, "tensor map: cuTensorMapEncodeTiled failed");
  return QUIC_OK;
}

// 2-D row-major tensor [rows, cols] of `elem_bytes` elements, box [box_rows, box_cols].
inline int make_map(CUtensorMap* map, CUtensorMapDataType type, int elem_bytes, const void* ptr, uint64_t rows,
                    uint64_t cols, uint32_t box_rows, uint32_t box_cols, CUtensorMapSwizzle swizzle) {
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * (uint64_t)elem_bytes};
  const cuuint32_t box[2] = {box_cols, box_rows};
  return make_tiled_map(map, type, 2, ptr, dims, strides, box, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
}


}  // namespace quic
