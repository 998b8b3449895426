// Causal prefill attention on tcgen05 with TMA-staged tiles (GQA 14:2, head_dim 64): the
// throughput form of attn_prefill.cu for prompts of 128 tokens and more.
//
// Replaces the reference's prefill attention (kernels/flash_attn_prefill_pytorch.py:10 = torch
// SDPA with a causal + left-pad mask; kernels/cuda/flash_attn_prefill.cu:87, wgmma + TMA on
// Hopper).  Same mathematics as attn_prefill.cu: fp32 online softmax over the keys
// 0 .. position of each query row; the probabilities multiply V as fp16 and are summed in fp32.
//
// One CTA owns 128 query rows of one (sequence, query head) and walks the key tiles of 64
// tokens its rows may see.  Per tile:
//   S = Q K^T      tcgen05.mma, A = Q tile (128 x 64, loaded once), B = K tile (64 x 64), both
//                  K-major in the 128-byte swizzle TMA writes; S (128 x 64 fp32) in tensor memory;
//   softmax        four warps; a thread owns one query row (TMEM lane = row): two passes over its 64
//                  scores in tensor memory, the maximum and P = exp2(..) rounded to fp16, which
//                  replaces the scores as the A operand of the second product;
//   O += P V       tcgen05.mma, A in tensor memory, B = the V tile as it lies in the cache
//                  (token-major: the transposed form of the operand), O (128 x 64 fp32) in tensor memory.
// O is rescaled in tensor memory where a row of the warp has a new maximum (leaving it until the maximum
// had grown by 2^8 was 8 % faster and cost a tenth of the precision).  The exponentials bound the
// whole: 64 per row and tile at sixteen a clock and SM are 111 us at 16 x 2048.
// The stages of a tile wait for one another; what hides that is the four CTAs of an SM (128 TMEM
// columns and 49 KB each) or, for a grid that is too small for it, scores that run a tile ahead (256 columns).
// The form before it had eight warps that shared rows, transposed V and kept O in registers, two
// CTAs an SM, us (launches of a graph): 1 x 512 14.7 -> 11.7, 8 x 517 33 -> 24,
// 16 x 2048 360 -> 231 (521 TFLOP/s of causal flops; 244 after seconds of it, under the power limit).
//
// Roles: warps 0-3 softmax and epilogue, warp 4 TMA producer (two stages of K and V), warp 5 MMA issuer.
// Every wait is bounded; a wait that runs out sets word 0 of the tensor path's error words
// and the CTA leaves with its MMAs and copies complete and its tensor memory released.
#include "tc_common.cuh"

namespace quic {
namespace {

constexpr int kQRows = 128;   // query rows per CTA (UMMA M)
constexpr int kKeys = 64;     // keys per tile (UMMA N of the first product, K of the second)
constexpr int kSoftmaxWarps = 4;  // one per TMEM lane quarter
constexpr int kAttThreads = (kSoftmaxWarps + 2) * 32;
constexpr uint32_t kQBytes = kQRows * 128;   // 128 rows x 64 halves
constexpr uint32_t kTileBytes = kKeys * 128;  // 64 rows x 64 halves
constexpr uint32_t kSmemQ = 0, kSmemK = kQBytes, kSmemV = kSmemK + 2 * kTileBytes, kSmemTotal = kSmemV + 2 * kTileBytes + 1024;
constexpr float kPShift = 8.f;  // P = 2^(score - maximum + 8): probabilities down to 2^-22 stay normal in fp16

struct PrefillTcArgs {
  const int32_t* seq_start;
  const int32_t* seq_len;
  const int32_t* seq_slot;
  const int32_t* seq_off;  // or nullptr
  half* out;               // [rows][896]
  int32_t rows, s_max, n_slots;
  float scale_log2;        // softmax scale x log2(e)
  uint32_t wait_limit_us;
  int32_t skip_tile;       // test hook: this key tile never comes; below -1, all come late (-1: none)
};

__device__ __forceinline__ uint32_t pack2(float x, float y) {
  const half2 h = __floats2half2_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ void mbar_arrive_cta(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// 2^x, one MUFU instruction (x = -inf gives 0)
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// two fp32 lanes per instruction
__device__ __forceinline__ uint64_t pair2(float x, float y) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ void unpair2(uint64_t d, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(d)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// D[tmem] (+)= A[tmem] . B, A fp16 packed two to a column
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

template <bool kAhead>
__global__ void __launch_bounds__(kAttThreads, kAhead ? 2 : 4)
    attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                           const __grid_constant__ CUtensorMap tm_v, const PrefillTcArgs a, int* status) {
  // columns: S, O with P in S's place; or S of even and of odd tiles, O, P
  constexpr uint32_t kTmemCols = kAhead ? 256 : 128, kColS1 = kAhead ? 64 : 0, kColO = kAhead ? 128 : 64, kColP = kAhead ? 192 : 0;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar_q, bar_full[2], bar_empty[2], bar_s[2], bar_p, bar_drain;
  __shared__ uint32_t tmem_base_s;
  __shared__ int fail_s;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int head = blockIdx.x, seq = blockIdx.y;
  const int len = a.seq_len[seq];  // (the sequence tables are not written by the kernels before this one)
  const int r0 = ((int)gridDim.z - 1 - (int)blockIdx.z) * kQRows;  // the longest key ranges of all are launched first
  if (r0 >= len) return;
  const int start = a.seq_start[seq];
  const int off = a.seq_off != nullptr ? max(a.seq_off[seq], 0) : 0;
  const int kv_len = off + len;
  const int slot = a.seq_slot[seq];
  if (slot < 0 || slot >= a.n_slots) return;
  const int kvh = head / (kHeads / kKvHeads);
  const int kv_row0 = (slot * kKvHeads + kvh) * a.s_max;  // first row of the (slot, kv head) in the cache plane
  const int n_tiles = (min(kv_len, off + r0 + kQRows) + kKeys - 1) / kKeys;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;

  if (tid == 0) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
    mbar_init(smem_u32(&bar_q), 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
      mbar_init(smem_u32(&bar_s[s]), 1);
    }
    mbar_init(smem_u32(&bar_p), kSoftmaxWarps);
    mbar_init(smem_u32(&bar_drain), 1);
    fail_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_s = tmem_base_s, tmem_o = tmem_base_s + kColO, tmem_p = tmem_base_s + kColP;
  pdl_launch_dependents();
  pdl_wait();  // queries and cache rows come from the kernels before this one

  bool issuer = false;
  if (warp == kSoftmaxWarps) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      mbar_expect_tx(smem_u32(&bar_q), kQBytes);
      tma_load_2d(base + kSmemQ, &tm_q, 0, head * a.rows + start + r0, smem_u32(&bar_q));
      for (int i = 0; i < n_tiles; ++i) {
        const int st = i & 1;
        if (i >= 2 && !mbar_wait(smem_u32(&bar_empty[st]), ((i >> 1) - 1) & 1, a.wait_limit_us)) {
          fail_s = 2;
          break;
        }
        if (a.skip_tile < -1) pause_us(-a.skip_tile);
        const uint32_t full = smem_u32(&bar_full[st]);
        mbar_expect_tx(full, 2 * kTileBytes);
        if (i != a.skip_tile) tma_load_2d(base + kSmemK + st * kTileBytes, &tm_k, 0, kv_row0 + i * kKeys, full);
        tma_load_2d(base + kSmemV + st * kTileBytes, &tm_v, 0, kv_row0 + i * kKeys, full);
      }
    }
  } else if (warp == kSoftmaxWarps + 1) {
    // ---------------- MMA issuer ----------------
    issuer = elect_one();
    if (issuer) {
      const uint64_t q0 = umma_desc_sw128(base + kSmemQ), k0 = umma_desc_sw128(base + kSmemK), v0 = umma_desc_sw128(base + kSmemV);
      const uint32_t idesc = umma_idesc_f16(kKeys);         // M = 128, N = 64
      const uint32_t idesc_v = idesc | (1u << 16);           // B transposed: N (the head dims) contiguous
      auto scores = [&](int i) {
        const int st = i & 1;
        if (!mbar_wait(smem_u32(&bar_full[st]), (i >> 1) & 1, a.wait_limit_us)) return false;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_f16(tmem_s + kColS1 * st, q0 + 2 * k, k0 + (uint64_t)(st * (kTileBytes / 16)) + 2 * k, idesc, k > 0 ? 1u : 0u);
        umma_commit(smem_u32(&bar_s[st]));
        return true;
      };
      bool ok = mbar_wait(smem_u32(&bar_q), 0, a.wait_limit_us) && scores(0);
      for (int i = 0; ok && i < n_tiles; ++i) {
        const int st = i & 1;
        if (kAhead && i + 1 < n_tiles) ok = scores(i + 1);  // S(i - 1), the buffer's last, has been read: P(i - 1) came
        if (!ok || !mbar_wait(smem_u32(&bar_p), i & 1, a.wait_limit_us)) {  // P(i) is in tensor memory, O rescaled where need be
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 4; ++k)  // sixteen tokens a step: two groups of eight rows of the V tile, eight columns of P
          umma_f16_ts(tmem_o, tmem_p + 8u * k, v0 + (uint64_t)(st * (kTileBytes / 16)) + k * (2048 / 16), idesc_v,
                      (i > 0 || k > 0) ? 1u : 0u);
        umma_commit(smem_u32(&bar_empty[st]));
        if (!kAhead && i + 1 < n_tiles)  // P(i) shares S's columns: its product has to be complete
          ok = mbar_wait(smem_u32(&bar_empty[st]), (i >> 1) & 1, a.wait_limit_us) && scores(i + 1);
      }
      if (!ok) fail_s = 3;
    }
  } else {
    // ---------------- softmax, epilogue ----------------
    const int row = 32 * warp + lane;          // TMEM lane
    const int pos = off + r0 + row;            // position of the row in its sequence
    const uint32_t lane_addr = (uint32_t)(32 * warp) << 16;
    const int last = min(pos, kv_len - 1);     // the row's last key
    float m_ref = -INFINITY, l_run = 0.f;
    bool ok = true;
    const uint32_t limit = 4 * a.wait_limit_us;  // (the issuer waits up to three times between two tiles' scores)
    for (int i = 0; i < n_tiles; ++i) {
      const int t0 = i * kKeys;
      const uint32_t tmem_si = tmem_s + kColS1 * (i & 1) + lane_addr;
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_s[i & 1]), (i >> 1) & 1, limit));
      if (!ok) break;
      tc_fence_after();
      // a tile wholly below the diagonal of all 128 rows needs no mask (CTA-uniform)
      const bool unmasked = t0 + kKeys - 1 <= min(off + r0, kv_len - 1);
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};  // independent chains
      float s[kAhead ? 64 : 32];  // with registers to spare the scores stay for the second pass
      auto load = [&](int h) {
        float (&part)[32] = *reinterpret_cast<float(*)[32]>(&s[kAhead ? 32 * h : 0]);
        tmem_ld32(tmem_si + 32u * h, part);
        if (!unmasked) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (t0 + 32 * h + j > last) part[j] = -INFINITY;
        }
      };
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        load(h);
        const float* part = &s[kAhead ? 32 * h : 0];
#pragma unroll
        for (int j = 0; j < 32; j += 2) mx[(j >> 1) & 3] = max3(mx[(j >> 1) & 3], part[j], part[j + 1]);
      }
      if (kAhead && i > 0) {  // P(i - 1) has been multiplied: P and O may be written
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_empty[(i - 1) & 1]), ((i - 1) >> 1) & 1, limit));
        if (!ok) break;
        tc_fence_after();
      }
      const float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * a.scale_log2;  // (the scale is positive)
      if (i == 0) {
        m_ref = mt;  // finite: every row sees key 0
      } else if (__any_sync(0xffffffffu, mt > m_ref)) {
        const float m_new = fmaxf(m_ref, mt), alpha = ex2(m_ref - m_new);
        l_run *= alpha;
        m_ref = m_new;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float v[16];
          uint32_t w[16];
          tmem_ld_cols<16>(tmem_o + lane_addr + 16u * c, v);
#pragma unroll
          for (int j = 0; j < 16; ++j) w[j] = __float_as_uint(v[j] * alpha);
          tmem_st16(tmem_o + lane_addr + 16u * c, w);
        }
      }
      const uint64_t scale2 = pair2(a.scale_log2, a.scale_log2), ref2 = pair2(kPShift - m_ref, kPShift - m_ref);
      uint64_t l2[2] = {0ull, 0ull};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t w[16];
        if (!kAhead) load(h);
        const float* part = &s[kAhead ? 32 * h : 0];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float p0, p1;
          unpair2(fma2(pair2(part[2 * j], part[2 * j + 1]), scale2, ref2), p0, p1);
          p0 = ex2(p0);  // 2^-inf = 0 for masked keys
          p1 = ex2(p1);
          w[j] = pack2(p0, p1);
          const float2 pr = __half22float2(*reinterpret_cast<const half2*>(&w[j]));
          l2[j & 1] = add2(l2[j & 1], pair2(pr.x, pr.y));  // what the product will see: the weights sum to one
        }
        tmem_st16(tmem_p + lane_addr + 16u * h, w);  // (behind the scores that are still to be read)
      }
      float la, lb;
      unpair2(add2(l2[0], l2[1]), la, lb);
      l_run += la + lb;
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cta(smem_u32(&bar_p));
    }
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_empty[(n_tiles - 1) & 1]), ((n_tiles - 1) >> 1) & 1, limit));
    tc_fence_after();
    ok = __all_sync(0xffffffffu, ok && !fail_s);
    if (!ok && fail_s == 0) fail_s = 1;
    if (ok) {
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      half* op = a.out + (size_t)(start + r0 + row) * kHidden + head * kHeadDim;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float o[32];
        tmem_ld32(tmem_o + lane_addr + 32u * h, o);
        if (r0 + row < len) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint4 u;
            u.x = pack2(o[8 * c + 0] * inv, o[8 * c + 1] * inv);
            u.y = pack2(o[8 * c + 2] * inv, o[8 * c + 3] * inv);
            u.z = pack2(o[8 * c + 4] * inv, o[8 * c + 5] * inv);
            u.w = pack2(o[8 * c + 6] * inv, o[8 * c + 7] * inv);
            reinterpret_cast<uint4*>(op)[4 * h + c] = u;
          }
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (fail_s != 0) {
    if (tid == 0) tc_report(status, (fail_s << 16) | 0x2000 | ((int)blockIdx.z & 0x1fff));
    drain_failed(issuer, smem_u32(&bar_drain));
  }
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base_s), "r"(kTmemCols) : "memory");
}

}  // namespace

// Whether the tcgen05 form takes this call (otherwise attn_prefill.cu's mma.sync kernels do).
bool attn_prefill_tc_supported(int n_seq, int max_len, int rows, int s_max, int n_slots) {
  return max_len >= kQRows && (int64_t)n_slots * kKvHeads * s_max < (1ll << 31) && (int64_t)kHeads * rows < (1ll << 31);
}

int attn_prefill_tc_launch(const void* q, const void* kcache, const void* vcache, const int32_t* seq_start,
                           const int32_t* seq_len, const int32_t* seq_slot, const int32_t* seq_off, int32_t n_seq,
                           int32_t max_len, int32_t rows, int32_t s_max, int32_t n_slots, float scale, void* out,
                           cudaStream_t stream, bool pdl) {
  CUtensorMap tm_q, tm_k, tm_v;
  int rc = make_map(&tm_q, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, q, (uint64_t)kHeads * rows, kHeadDim, kQRows, kHeadDim,
                    CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != QUIC_OK) return rc;
  const uint64_t kv_rows = (uint64_t)n_slots * kKvHeads * s_max;
  rc = make_map(&tm_k, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, kcache, kv_rows, kHeadDim, kKeys, kHeadDim,
                CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != QUIC_OK) return rc;
  rc = make_map(&tm_v, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, vcache, kv_rows, kHeadDim, kKeys, kHeadDim,
                CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != QUIC_OK) return rc;
  int* status = tc_status_words();
  QUIC_REQUIRE(status != nullptr, QUIC_E_CUDA, "attn_prefill: no address for the tensor path's error words");
  PrefillTcArgs a = {};
  a.seq_start = seq_start;
  a.seq_len = seq_len;
  a.seq_slot = seq_slot;
  a.seq_off = seq_off;
  a.out = (half*)out;
  a.rows = rows;
  a.s_max = s_max;
  a.n_slots = n_slots;
  tc_test_hook(&a.wait_limit_us, &a.skip_tile);
  a.scale_log2 = (scale > 0.f ? scale : 0.125f) * 1.4426950408889634f;
  // Up to four CTAs an SM in all: too few to hide a tile's latency, so its scores run a tile ahead, in twice
  // the tensor memory (plain / ahead, us: 1 x 512 15.0 / 11.7, 1 x 2048 46.5 / 34.8, 4 x 1000 28.8 / 28.2,
  // 8 x 517 22.0 / 23.6, 16 x 2048 231 / 273).
  const dim3 grid(kHeads, n_seq, (max_len + kQRows - 1) / kQRows);
  const bool ahead = (int64_t)grid.x * grid.y * grid.z <= 4 * 148;
  auto kernel = ahead ? attn_prefill_tc_kernel<true> : attn_prefill_tc_kernel<false>;
  QUIC_CUDA(ahead ? allow_smem<attn_prefill_tc_kernel<true>>(kSmemTotal) : allow_smem<attn_prefill_tc_kernel<false>>(kSmemTotal));
  QUIC_CUDA(launch(kernel, grid, dim3(kAttThreads), kSmemTotal, stream, pdl, tm_q, tm_k, tm_v, a, status));
  return QUIC_OK;
}

}  // namespace quic
