// Dense fp16 GEMM for many rows, y[M, N] = x[M, K] . W[N, K]^T, on pairs of SMs
// (tcgen05.mma.cta_group::2), with bias or SwiGLU in the epilogue, and the unpacking of int4 weights to
// the fp16 operand it reads.
//
// A prefill of a few thousand tokens and more is bound by the tensor cores.  The W4A16 kernel
// (w4_gemm_tc.cu) unpacks its weight tile again for every 256 rows, in the loop that feeds the MMAs, and
// reads each operand tile into one SM only: 770-870 TFLOP/s.  At these sizes a layer's weights are
// cheaper to unpack once per call (15 M weights, 30 MB written) than a hundred times, and two SMs
// then share one 256 x NT tile: each holds 128 of its token rows and half of its weight rows, so
// an SM reads 32 KB per 64-wide k block of 512 tensor cycles.
//
// One persistent CTA pair per two SMs takes tiles in turn, weight tile fastest (the pairs that run
// together share token rows, the weights stay in L2).  Warp 0 loads (each CTA its own half of
// both operands, the bytes counted on the leading CTA's barrier), warp 1 of the leading CTA
// issues the MMAs, warps 2-17 read the accumulator back (four per lane quarter: with one, the
// epilogue's 16 us a tile hid 4 us of MMAs); there are two accumulators of 256
// columns, so the epilogue of a tile runs under the next tile's MMAs.  Token rows are on
// the M side: a thread of the epilogue owns a row and, with 128 gate and 128 up columns in a tile, both
// factors of its SwiGLU outputs.  Waits are bounded by the clock: one that runs out sets word 0
// of the tensor path's error words and the pair leaves with its MMAs and copies complete and its tensor memory released.
#include "tc_common.cuh"

namespace quic {
namespace {

constexpr int kPairStages = 5, kPairEpilogueWarps = 16, kPairThreads = 64 + 32 * kPairEpilogueWarps;
constexpr uint32_t kPairPitch = 80;                                        // staged row: 32 halves, padded
constexpr uint32_t kPairStaging = kPairEpilogueWarps * 32 * kPairPitch;
constexpr uint32_t kPairA = 128 * 128;                                     // 128 token rows x 64 k

template <int NT>
struct PairSmem {
  static constexpr uint32_t kB = NT / 2 * 128;  // half of the weight rows x 64 k
  static constexpr uint32_t kStage = kPairA + kB;
  static constexpr uint32_t kTotal = kPairStages * kStage + kPairStaging + 1024;
};

struct PairArgs {
  const half* bias;  // [N] or nullptr
  half* y;           // [M, N], or [M, N / 2] with SwiGLU
  float* part;       // split K: [splits][M][N] fp32 partial sums (then y and bias belong to the consumer)
  int m_total, n, k;
  int splits;
  int* status;
  PairRope rope;
  uint32_t wait_limit_us;
  int32_t skip_kblock;  // test hook: this k block (of 64) of a tile never comes; below -1, all come late (-1: none)
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void pair_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void pair_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the same shared-memory address in the pair's leading CTA
__device__ __forceinline__ uint32_t in_leader(uint32_t addr) {
  uint32_t ra;
  asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(ra) : "r"(addr));
  return ra;
}
// Tiled load into this CTA's shared memory whose bytes count on a barrier of the pair, given by its cluster address.
__device__ __forceinline__ void pair_load(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void pair_umma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Sixteen finished qkv outputs of a token, columns col .. col + 15 (eight stored pairs: dims d and d + 32 side by
// side), rotated by its position (queries and keys) and written to their heads: sixteen bytes of either half.
// Same arithmetic as qkv_rope_rows_kernel, whose 150 MB at 32768 tokens (50 us a layer) this saves.
__device__ __forceinline__ void rope_store(const PairRope& r, const float (&v)[16], int col, int tok, int pos, int slot, int rows) {
  const int head = col >> 6, d0 = (col & 63) >> 1;
  __align__(16) half lo[8], hi[8];
  if (head < kHeads + kKvHeads) {
    const int pp = pos < r.max_pos ? (pos < 0 ? 0 : pos) : r.max_pos - 1;
    const uint4 c4 = *reinterpret_cast<const uint4*>(r.cos_t + (size_t)pp * 32 + d0);
    const uint4 s4 = *reinterpret_cast<const uint4*>(r.sin_t + (size_t)pp * 32 + d0);
    const half* ch = reinterpret_cast<const half*>(&c4);
    const half* sh = reinterpret_cast<const half*>(&s4);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float x = __half2float(__float2half_rn(v[2 * i])), y = __half2float(__float2half_rn(v[2 * i + 1]));
      const float c = __half2float(ch[i]), sn = __half2float(sh[i]);
      lo[i] = __float2half_rn(x * c - y * sn);
      hi[i] = __float2half_rn(x * sn + y * c);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      lo[i] = __float2half_rn(v[2 * i]);
      hi[i] = __float2half_rn(v[2 * i + 1]);
    }
  }
  half* dst;
  if (head < kHeads) {
    dst = r.q + ((size_t)head * rows + tok) * kHeadDim;
  } else {
    if (pos >= r.s_max || pos < 0 || slot < 0 || slot >= r.n_slots) return;  // nothing is appended for such a row
    half* plane = head < kHeads + kKvHeads ? r.kcache : r.vcache;
    dst = plane + (((size_t)slot * kKvHeads + ((head - kHeads) & 1)) * r.s_max + pos) * kHeadDim;
  }
  *reinterpret_cast<uint4*>(dst + d0) = *reinterpret_cast<const uint4*>(lo);
  *reinterpret_cast<uint4*>(dst + 32 + d0) = *reinterpret_cast<const uint4*>(hi);
}
// arrives on the barrier of both CTAs once the MMAs issued so far are complete
__device__ __forceinline__ void pair_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"((uint16_t)3)
      : "memory");
}
// a word at the same shared-memory address of the pair's second CTA
__device__ __forceinline__ void tell_peer(uint32_t addr, int value) {
  asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %0, 1;\n\tst.shared::cluster.u32 [ra], %1;\n\t}" ::"r"(addr), "r"(value)
               : "memory");
}
__device__ __forceinline__ void arrive_leader(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(in_leader(bar)) : "memory");
}

template <int NT, bool kSwiglu, bool kRope>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w, const PairArgs a) {
  using L = PairSmem<NT>;
  constexpr int kOut = kSwiglu ? NT / 2 : NT;  // output columns of a tile
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[kPairStages], bar_empty[kPairStages], bar_acc[2], bar_free[2], bar_drain;
  __shared__ uint32_t tmem_base_s;
  __shared__ int fail_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_rank();
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int ntiles = a.n / NT, flat = ntiles * ((a.m_total + 255) / 256), tiles = flat * a.splits, kblocks = a.k / kBlockK;
  const int first = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  pair_arrive();
  if (tid == 0) {
    tma_prefetch_desc(&tm_x);
    tma_prefetch_desc(&tm_w);
    for (int s = 0; s < kPairStages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&bar_acc[s]), 1);
      mbar_init(smem_u32(&bar_free[s]), 2 * kPairEpilogueWarps);
    }
    mbar_init(smem_u32(&bar_drain), 1);
    fail_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  // An allocation of the pair is made by both CTAs, and each takes part in the other's.  So both are known to run before either
  // allocates, and neither leaves before both have given back: the next CTA on its SM, of another kernel and stream, may
  // allocate by itself at once.  (Without, a pair beside decode steps on another stream stood still for good: the first CTA's
  // allocation had returned, the second's never did.)
  pair_wait();
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base_s)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  pair_sync();
  tc_fence_after();
  const uint32_t tmem_d = tmem_base_s;
  pdl_launch_dependents();
  pdl_wait();

  bool issuer = false;
  if (warp == 0) {
    if (lane == 0) {
      int stage = 0, pass = 0;
      bool ok = true;
      for (int t = first; ok && t < tiles; t += pairs) {
        const int split = t / flat, f = t % flat, nt = f % ntiles, m0 = (f / ntiles) * 256 + (int)rank * 128;
        const int kb1 = kblocks * (split + 1) / a.splits;
        const int w0 = kSwiglu ? (int)rank * (a.n / 2) + nt * (NT / 2) : nt * NT + (int)rank * (NT / 2);
        for (int kb = kblocks * split / a.splits; kb < kb1; ++kb) {
          if (pass > 0 && !mbar_wait(smem_u32(&bar_empty[stage]), (pass - 1) & 1, a.wait_limit_us)) {
            fail_s = 2;
            ok = false;
            break;
          }
          if (a.skip_kblock < -1) pause_us(-a.skip_kblock);
          const uint32_t a_s = base + stage * L::kStage, full = smem_u32(&bar_full[stage]), lead = in_leader(full);
          if (rank == 0) mbar_expect_tx(full, 2 * L::kStage);
          if (kb != a.skip_kblock) pair_load(a_s, &tm_x, kb * kBlockK, m0, lead);
          pair_load(a_s + kPairA, &tm_w, kb * kBlockK, w0, lead);
          if (++stage == kPairStages) {
            stage = 0;
            ++pass;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && (issuer = elect_one())) {
      const uint64_t a0 = umma_desc_sw128(base), b0 = umma_desc_sw128(base + kPairA);
      // fp16 x fp16 -> fp32, both operands K-major, M = 256 over the pair, N = NT
      constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
      int stage = 0, pass = 0, j = 0;
      bool ok = true;
      for (int t = first; ok && t < tiles; t += pairs, ++j) {
        const int buf = j & 1;
        if (j >= 2 && !mbar_wait(smem_u32(&bar_free[buf]), ((j >> 1) - 1) & 1, a.wait_limit_us)) {
          fail_s = 4;
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem_d + 256u * buf;
        const int split = t / flat, nkb = kblocks * (split + 1) / a.splits - kblocks * split / a.splits;
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(smem_u32(&bar_full[stage]), pass & 1, a.wait_limit_us)) {
            fail_s = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t at = (uint64_t)(stage * (L::kStage / 16));
#pragma unroll
          for (int k = 0; k < kBlockK / 16; ++k) pair_umma(d, a0 + at + 2 * k, b0 + at + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          pair_commit(smem_u32(&bar_empty[stage]));
          if (++stage == kPairStages) {
            stage = 0;
            ++pass;
          }
        }
        if (ok) pair_commit(smem_u32(&bar_acc[buf]));
      }
      if (fail_s != 0) tell_peer(smem_u32(&fail_s), fail_s);  // (its epilogue waits for these MMAs too)
    }
  } else {
    const int quarter = warp & 3, group = (warp - 2) >> 2;  // TMEM lanes that this warp may read, 32-column share
    unsigned char* out_s = smem_raw + (base - smem_u32(smem_raw)) + kPairStages * L::kStage + (warp - 2) * 32 * kPairPitch;
    int j = 0;
    const int ld_y = kSwiglu ? a.n / 2 : a.n;
    for (int t = first; t < tiles; t += pairs, ++j) {
      const int buf = j & 1;
      const int split = t / flat, f = t % flat;
      const int row0 = (f / ntiles) * 256 + (int)rank * 128 + quarter * 32, col0 = (f % ntiles) * kOut;
      // RoPE form: the lane's token (rows past the end: none)
      const int tok = row0 + lane;
      const bool live = kRope && tok < a.m_total;
      const int pos = live ? a.rope.positions[tok] : 0, slot = live ? a.rope.slots[tok] : -1;
      // (the issuer has a wait for every k block)
      const uint32_t limit = a.wait_limit_us * (uint32_t)min(kblocks + 2, 1024);
      if (!__all_sync(0xffffffffu, mbar_wait_unless(smem_u32(&bar_acc[buf]), (j >> 1) & 1, &fail_s, limit))) {
        fail_s = 3;
        break;
      }
      tc_fence_after();
      const uint32_t taddr = tmem_d + 256u * buf + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
      for (int c = 32 * group; c < kOut; c += 128) {
        uint32_t o[16];
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          float v[16];
          tmem_ld_cols<16>(taddr + c + 16 * hh, v);
          if (!kSwiglu && a.part != nullptr) {
            if (row0 + lane < a.m_total) {
              float4* dst = reinterpret_cast<float4*>(a.part + ((size_t)split * a.m_total + row0 + lane) * a.n + col0 + c + 16 * hh);
#pragma unroll
              for (int i = 0; i < 4; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            }
            continue;
          }
          if (kSwiglu) {
            float u[16];
            tmem_ld_cols<16>(taddr + NT / 2 + c + 16 * hh, u);
#pragma unroll
            for (int i = 0; i < 16; ++i)  // the linear's outputs are fp16 tensors: round both factors
              v[i] = silu_mul(__half2float(__float2half_rn(v[i])), __half2float(__float2half_rn(u[i])));
          } else if (a.bias != nullptr) {
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              const float2 b = __half22float2(*reinterpret_cast<const half2*>(a.bias + col0 + c + 16 * hh + i));
              v[i] = __half2float(__float2half_rn(v[i])) + b.x;
              v[i + 1] = __half2float(__float2half_rn(v[i + 1])) + b.y;
            }
          }
          if constexpr (kRope) {
            if (live) rope_store(a.rope, v, col0 + c + 16 * hh, tok, pos, slot, a.m_total);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
              o[8 * hh + i] = *reinterpret_cast<const uint32_t*>(&h);
            }
          }
        }
        if (c + 128 >= kOut) {  // read out: the accumulator may be overwritten
          tc_fence_before();
          __syncwarp();
          if (lane == 0) arrive_leader(smem_u32(&bar_free[buf]));
        }
        if constexpr (!kRope) {
          if (!kSwiglu && a.part != nullptr) continue;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<uint4*>(out_s + lane * kPairPitch + 16 * i) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 4; ++i) {  // eight rows of 64 contiguous bytes per store
            const int r = 8 * i + (lane >> 2), piece = lane & 3;
            if (row0 + r < a.m_total)
              *reinterpret_cast<uint4*>(a.y + (size_t)(row0 + r) * ld_y + col0 + c + 8 * piece) =
                  *reinterpret_cast<const uint4*>(out_s + r * kPairPitch + 16 * piece);
          }
          __syncwarp();
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  if (__syncthreads_or(fail_s)) {  // (the leader may set it at any time) the last MMAs and copies, as in drain_failed(); MMAs in flight that rank 0 has not waited for make it fail
    if (tid == 0) tc_report(a.status, (fail_s << 16) | 0x2000 | (int)(blockIdx.x & 0x1fff));
    if (issuer) {
      pair_commit(smem_u32(&bar_drain));
      mbar_wait(smem_u32(&bar_drain), 0);
      tc_fence_after();
    }
    if (tid == 0) pause_us(1000);
    __syncwarp();
    tc_fence_before();
    __syncthreads();
  }
  pair_sync();  // nobody leaves while the pair's copies, arrivals or MMAs use its shared memory
  if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_d) : "memory");
  __syncwarp();
  pair_sync();
}

template <int NT, bool kSwiglu, bool kRope = false>
int run_pair(const half* x, const half* w, const PairArgs& a, cudaStream_t st) {
  CUtensorMap tm_x, tm_w;
  int rc = make_map(&tm_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x, (uint64_t)a.m_total, (uint64_t)a.k, 128, kBlockK,
                    CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != QUIC_OK) return rc;
  rc = make_map(&tm_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, w, (uint64_t)a.n, (uint64_t)a.k, NT / 2, kBlockK,
                CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != QUIC_OK) return rc;
  auto kernel = gemm_pair_kernel<NT, kSwiglu, kRope>;
  QUIC_CUDA((allow_smem<gemm_pair_kernel<NT, kSwiglu, kRope>>(PairSmem<NT>::kTotal)));
  const int64_t tiles = (int64_t)(a.n / NT) * ((a.m_total + 255) / 256) * a.splits;
  const int pairs = tiles < 74 ? (int)tiles : 74;
  QUIC_CUDA(launch(kernel, dim3(2 * pairs), dim3(kPairThreads), (size_t)PairSmem<NT>::kTotal, st, true, tm_x, tm_w, a));
  return QUIC_OK;
}

// The weight tile's width: the widest that divides N (with SwiGLU, 128 gate and 128 up columns).
int pair_nt(int n, bool swiglu) {
  if (swiglu) return n % 256 == 0 ? 256 : 0;
  return n % 256 == 0 ? 256 : n % 224 == 0 ? 224 : n % 192 == 0 ? 192 : 0;
}

// W fp16 [N][K] from packed [K/8][N] int32 words, for up to four weights in one launch: a thread takes
// 64 k of one row (reads coalesced over rows), a warp's rows leave through shared memory, 128
// contiguous bytes each.
struct UnpackJob {
  quic_w4_t w;
  half* out;
  int first_block;  // blocks of 256 rows x 64 k, rows fastest
};
struct UnpackArgs {
  UnpackJob job[4];
};
__global__ void __launch_bounds__(256) w4_unpack_kernel(const __grid_constant__ UnpackArgs a) {
  __shared__ __align__(16) unsigned char stage_s[8][32 * 144];  // a warp's 32 rows of 128 bytes, padded
  pdl_launch_dependents();
  int i = 0;
  while (i < 3 && (int)blockIdx.x >= a.job[i + 1].first_block) ++i;
  const UnpackJob& J = a.job[i];
  const int blk = (int)blockIdx.x - J.first_block, nb = (J.w.n + 255) / 256;
  const int n = (blk % nb) * 256 + (int)threadIdx.x, k0 = (blk / nb) * 64;
  const bool live = n < J.w.n;
  uint32_t word[8];
  half2 s2, zp;
  if (live) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(J.w.qw) + (size_t)(k0 / 8) * J.w.n + n;
#pragma unroll
    for (int j = 0; j < 8; ++j) word[j] = __ldg(q + (size_t)j * J.w.n);
    const int g = k0 / kGroup;
    s2 = __half2half2(reinterpret_cast<const half*>(J.w.sc)[(size_t)g * J.w.n + n]);
    const uint8_t z = reinterpret_cast<const uint8_t*>(J.w.zp)[(size_t)g * (J.w.n >> 1) + (n >> 1)];
    zp = zp_to_half2((z >> (4 * (n & 1))) & 15);
  }
  unsigned char* mine = stage_s[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  if (live) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      half2 d[4];
      dequant8(word[j], zp, s2, d);  // d[p] = (k = p, k = p + 4)
      const uint32_t u0 = *reinterpret_cast<uint32_t*>(&d[0]), u1 = *reinterpret_cast<uint32_t*>(&d[1]);
      const uint32_t u2 = *reinterpret_cast<uint32_t*>(&d[2]), u3 = *reinterpret_cast<uint32_t*>(&d[3]);
      *reinterpret_cast<uint4*>(mine + lane * 144 + 16 * j) =
          make_uint4(__byte_perm(u0, u1, 0x5410), __byte_perm(u2, u3, 0x5410), __byte_perm(u0, u1, 0x7632),
                     __byte_perm(u2, u3, 0x7632));
    }
  }
  __syncwarp();
  pdl_wait();  // the fp16 copies may still be read by the previous layer's linears
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int r = 4 * j + (lane >> 3), row = n - lane + r;
    if (row < J.w.n)
      *reinterpret_cast<uint4*>(J.out + (size_t)row * J.w.k + k0 + 8 * (lane & 7)) =
          *reinterpret_cast<const uint4*>(mine + r * 144 + 16 * (lane & 7));
  }
}

}  // namespace

bool gemm_pair_supported(int m, int n, int k, bool swiglu) {
  return m >= 1 && m <= (1 << 24) && k >= kBlockK && k % kBlockK == 0 && pair_nt(n, swiglu) != 0;
}

// K splits: while the tiles leave most pairs idle, at least eight k blocks each (down at 1024 rows is 16
// tiles of 76 k blocks: 28 us in one piece).
int gemm_pair_splits(int m, int n, int k) {
  const int64_t tiles = (int64_t)(n / pair_nt(n, false)) * ((m + 255) / 256);
  int s = tiles >= 74 ? 1 : (int)(74 / tiles);
  if (s > k / kBlockK / 8) s = k / kBlockK / 8;
  return s < 1 ? 1 : s > 16 ? 16 : s;
}

// About how long a packed linear takes here, in us: the fp16 copy of the weight, full waves of tiles over 74 pairs, the
// output's stores, and the sum of K splits (constants from the four layer shapes at 400..8192 rows, mean error 7 %).
double gemm_pair_us(int m, int n, int k) {
  const int nt = pair_nt(n, false), splits = gemm_pair_splits(m, n, k);
  const int64_t tiles = (int64_t)(n / nt) * ((m + 255) / 256) * splits;
  const double out_mb = 2e-6 * m * n, wave = 0.3 + 1.4e-3 * nt * (k / kBlockK) / splits;
  return 6.0 + 0.4e-6 * n * k + (double)((tiles + 73) / 74) * wave + 0.1 * out_mb + (splits > 1 ? 2.5 + 0.8 * splits * out_mb : 0.0);
}

// `part` (gemm_pair_splits x m x n fp32, may be null): where that is more than one split their partial sums
// stay there for a consumer, y is not written and *splits says how many.
int gemm_pair(const half* x, const half* w, const half* bias, half* y, int m, int n, int k, bool swiglu, cudaStream_t st,
              float* part, int* splits) {
  QUIC_REQUIRE(gemm_pair_supported(m, n, k, swiglu), QUIC_E_SHAPE, "gemm_pair: unsupported shape");
  QUIC_REQUIRE(((uintptr_t)x | (uintptr_t)w | (uintptr_t)y | (uintptr_t)part) % 16 == 0 && (uintptr_t)bias % 4 == 0, QUIC_E_ARG,
               "gemm_pair: tensors must be 16-byte aligned, the bias 4-byte");
  PairArgs a = {bias, y, nullptr, m, n, k, 1, tc_status_words()};
  tc_test_hook(&a.wait_limit_us, &a.skip_kblock);
  if (splits != nullptr) *splits = 0;
  if (part != nullptr && gemm_pair_splits(m, n, k) > 1) {
    a.part = part;
    a.splits = *splits = gemm_pair_splits(m, n, k);
  }
  QUIC_REQUIRE(a.status != nullptr, QUIC_E_CUDA, "gemm_pair: no address for the tensor path's error words");
  if (swiglu) return run_pair<256, true>(x, w, a, st);
  switch (pair_nt(n, false)) {
    case 256: return run_pair<256, false>(x, w, a, st);
    case 224: return run_pair<224, false>(x, w, a, st);
    default: return run_pair<192, false>(x, w, a, st);
  }
}

// The fused qkv linear with RoPE and the KV append in its epilogue: y never exists.
int gemm_pair_qkv(const half* x, const half* w, const half* bias, int m, const PairRope& rope, cudaStream_t st) {
  static_assert(kQkvN % 192 == 0 && 192 % kHeadDim == 0, "whole heads in a tile");
  QUIC_REQUIRE(((uintptr_t)x | (uintptr_t)w) % 16 == 0 && (uintptr_t)bias % 4 == 0, QUIC_E_ARG,
               "gemm_pair: tensors must be 16-byte aligned, the bias 4-byte");
  PairArgs a = {bias, nullptr, nullptr, m, kQkvN, kHidden, 1, tc_status_words(), rope};
  tc_test_hook(&a.wait_limit_us, &a.skip_kblock);
  QUIC_REQUIRE(a.status != nullptr, QUIC_E_CUDA, "gemm_pair: no address for the tensor path's error words");
  return run_pair<192, false, true>(x, w, a, st);
}

// Packed weights -> fp16 [N][K] copies in `out[i]`, up to four in one launch; dense ones are passed over.
int w4_unpack(const quic_w4_t* const* w, half* const* out, int count, cudaStream_t st) {
  UnpackArgs a = {};
  int blocks = 0;
  for (int i = 0; i < 4; ++i) {
    a.job[i].first_block = blocks;
    if (i >= count || w[i]->w16 != nullptr) continue;
    a.job[i].w = *w[i];
    a.job[i].out = out[i];
    blocks += ((w[i]->n + 255) / 256) * (w[i]->k / 64);
  }
  QUIC_CUDA(launch(w4_unpack_kernel, dim3(blocks), dim3(256), 0, st, true, a));
  return QUIC_OK;
}

}  // namespace quic
