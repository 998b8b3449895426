// Stand-alone GQA decode attention over long caches: every (row, KV head) is cut into `splits` equal
// ranges of its OWN tokens, one CTA each; six warps take the 64-token tiles of the range in turn, each
// with a shared-memory stage of its own that it refills by TMA as soon as the tile is in registers.
//
// Memory latency and too few bytes in flight bounded its predecessors: the split kernel with direct loads
// (attn_decode_mma_kernel) kept HBM at a third of its rate and spent sixteen mma rows on seven heads, and
// one CTA per (row, KV head) (attn_decode_stream_kernel) leaves SMs idle unless rows x 2 happens to be
// near a multiple of 148.  Here two CTAs share an SM (2 x 96 KB of copies in flight), the products keep
// the tokens or the head dims on the M side of the mma (seven of eight columns used), and the splits of
// a (row, KV head) are one thread-block cluster that merges over distributed shared memory: no scratch,
// no counters.  Measured, rows x tokens, us before -> after (before: the faster of those two):
//   1 x 1024 7.3 -> 4.8, 1 x 8192 15.8 -> 7.0, 4 x 4096 11.8 -> 6.2, 16 x 1024 11.2 -> 5.1,
//   16 x 8192 28.6 -> 14.2, 33 x 8000 49 -> 23, 64 x 8192 50 -> 40, 256 x 7800 170 -> 129.
//
// Same mathematics as fad_decode_kernel + fad_combine_kernel of the reference
// (kernels/cuda/flash_attn_decode.cu:12,104): fp32 softmax over the tokens [start_b, end_b) of
// each row, rows without tokens give zeros (:118-121).
#include "attn_flow_tile.cuh"
#include "decode_kernels.cuh"

namespace quic {
namespace {

constexpr int kGroupHeads = kHeads / kKvHeads;  // 7
constexpr int kFlowWarps = 6;
constexpr uint32_t kFlowTile = kWarpChunk * kHeadDim * 2;  // 8 KB: 64 tokens x 128 bytes
constexpr uint32_t kFlowStage = 2 * kFlowTile;             // K tile, V tile
constexpr int kFlowSmem = kFlowWarps * kFlowStage + 1024;

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// a float of CTA `rank` of the cluster, at this CTA's shared-memory address
__device__ __forceinline__ float ld_peer(uint32_t addr, int rank) {
  float v;
  asm volatile(
      "{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %1, %2;\n\tld.shared::cluster.f32 %0, [ra];\n\t}"
      : "=f"(v)
      : "r"(addr), "r"(rank)
      : "memory");
  return v;
}
// 4-D tiled load: (head dim, token, KV head, row)
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c1, int c2, int c3, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

__global__ void __launch_bounds__(kFlowWarps * 32, 2)
    attn_decode_flow_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                            const AttnArgs a, int* status) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[kFlowWarps];
  __shared__ float m_s[kFlowWarps][8], l_s[kFlowWarps][8];
  __shared__ __align__(16) float o_s[kFlowWarps][kGroupHeads][kHeadDim];
  __shared__ float part_s[kGroupHeads * 66];  // this split's sums, {max, sum} behind each head's
  __shared__ int fail_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t k_s = base + warp * kFlowStage, v_s = k_s + kFlowTile, bar = smem_u32(&bar_full[warp]);
  if (tid == 0) {
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
    for (int i = 0; i < kFlowWarps; ++i) mbar_init(smem_u32(&bar_full[i]), 1);
    fail_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  pdl_launch_dependents();
  pdl_wait();  // the set-up runs under the kernel in front
  int t_begin = a.start != nullptr ? a.start[b] : 0, t_end = a.end != nullptr ? a.end[b] : a.s_cap, plane = b;
  if (a.pos != nullptr) {  // a decode step: the row's slot, up to the token that it has just appended
    plane = a.rows[b];
    t_end = __ldcg(a.pos + plane) + 1;
  }
  if (t_end > a.s_cap) t_end = a.s_cap;
  if (t_begin < 0) t_begin = 0;
  // this split's tiles: an equal share of the tiles that hold the row's tokens
  const int tile0 = t_begin / kWarpChunk;
  const int tiles = t_end > t_begin ? (t_end + kWarpChunk - 1) / kWarpChunk - tile0 : 0;
  const int i0 = (int)((int64_t)tiles * split / a.splits), i1 = (int)((int64_t)tiles * (split + 1) / a.splits);

  auto request = [&](int i) {
    if (lane == 0) {
      mbar_expect_tx(bar, kFlowStage);
      tma_load_4d(k_s, &tm_k, (tile0 + i) * kWarpChunk, kvh, plane, bar);
      tma_load_4d(v_s, &tm_v, (tile0 + i) * kWarpChunk, kvh, plane, bar);
    }
  };
  if (i0 + warp < i1) request(i0 + warp);
  uint32_t qb[4][2];  // Q^T fragments: column g = head (column 7 is zero)
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(
        a.q + ((size_t)b * kHeads + kvh * kGroupHeads + (g < kGroupHeads ? g : 0)) * kHeadDim + 16 * ks + 2 * t);
    qb[ks][0] = g < kGroupHeads ? q[0] : 0u;
    qb[ks][1] = g < kGroupHeads ? q[4] : 0u;
  }
  FlowState st;
  uint32_t parity = 0;
  for (int i = i0 + warp; i < i1; i += kFlowWarps) {
    if (!__all_sync(0xffffffffu, mbar_wait(bar, parity))) {
      if (lane == 0) fail_s = 1;
      mbar_wait(bar, parity);  // (no exit under a copy in flight)
      break;
    }
    parity ^= 1u;
    uint32_t V[4][4][4];
    float sc[4][4];
    flow_scores(k_s, v_s, qb, lane, V, sc);
    // the stage is in registers: refill it (the reads come before the copy, another proxy)
    fence_proxy_async();
    __syncwarp();
    if (i + kFlowWarps < i1) request(i + kFlowWarps);
    flow_attend(st, V, sc, (tile0 + i) * kWarpChunk, t_begin, t_end, a.scale, lane);
  }
  // ---- the warps meet in shared memory ----
  flow_store(st, m_s[warp], l_s[warp], o_s[warp], lane);
  __syncthreads();
  if (fail_s != 0 && tid == 0)  // a bounded wait gave up: say so (the row's output is then invalid)
    tc_report(status, (7 << 16) | 0x4000 | ((int)blockIdx.z & 0x3fff));
  for (int idx = tid; idx < kGroupHeads * kHeadDim; idx += kFlowWarps * 32) {
    const int h = idx >> 6, d = idx & 63;
    float mx = -INFINITY, num = 0.f, den = 0.f;
#pragma unroll
    for (int w = 0; w < kFlowWarps; ++w) mx = fmaxf(mx, m_s[w][h]);
    if (mx != -INFINITY) {
#pragma unroll
      for (int w = 0; w < kFlowWarps; ++w) {
        const float e = __expf(m_s[w][h] - mx);
        den = fmaf(e, l_s[w][h], den);
        num = fmaf(e, o_s[w][h][d], num);
      }
    }
    const int qh = kvh * kGroupHeads + h;
    if (a.splits == 1) {
      a.out[((size_t)b * kHeads + qh) * kHeadDim + d] = __float2half_rn(den > 0.f ? num / den : 0.f);
    } else {
      part_s[h * 66 + d] = num;
      if (d == 0) {
        part_s[h * 66 + 64] = mx;
        part_s[h * 66 + 65] = den;
      }
    }
  }
  if (a.splits > 1) {
    cluster_sync();  // every split's sums are in its CTA's shared memory
    const int per = (kGroupHeads * kHeadDim + a.splits - 1) / a.splits;  // outputs that this CTA merges
    for (int idx = split * per + tid; idx < min((split + 1) * per, kGroupHeads * kHeadDim); idx += kFlowWarps * 32) {
      const int h = idx >> 6, d = idx & 63;
      const uint32_t at = smem_u32(part_s + h * 66);
      float mr8[8], lr8[8], or8[8], mx = -INFINITY, num = 0.f, den = 0.f;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const bool on = r < a.splits;
        mr8[r] = on ? ld_peer(at + 64 * 4, r) : -INFINITY;
        lr8[r] = on ? ld_peer(at + 65 * 4, r) : 0.f;
        or8[r] = on ? ld_peer(at + d * 4, r) : 0.f;
        mx = fmaxf(mx, mr8[r]);
      }
      if (mx != -INFINITY) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float e = __expf(mr8[r] - mx);
          den = fmaf(e, lr8[r], den);
          num = fmaf(e, or8[r], num);
        }
      }
      a.out[((size_t)b * kHeads + kvh * kGroupHeads + h) * kHeadDim + d] = __float2half_rn(den > 0.f ? num / den : 0.f);
    }
    cluster_sync();  // nobody leaves while its shared memory is read
  }
}

// (head dim, token, KV head, row) over planes with any strides; tokens past the end read as zero
int make_kv_map(CUtensorMap* map, const void* p, int64_t stride_b, int64_t stride_h, int b, int s) {
  const cuuint64_t dims[4] = {(cuuint64_t)kHeadDim, (cuuint64_t)s, (cuuint64_t)kKvHeads, (cuuint64_t)b};
  const cuuint64_t strides[3] = {kHeadDim * 2, (cuuint64_t)stride_h * 2, (cuuint64_t)stride_b * 2};
  const cuuint32_t box[4] = {kHeadDim, kWarpChunk, 1, 1};
  return make_tiled_map(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, p, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
}

}  // namespace

// Splits of a (row, KV head).  While the CTAs have an SM each, latency counts: about four 64-token tiles
// for a CTA's six warps (1 x 1500 in one piece 7.0 us, in five 4.6).  Beyond that two CTAs share an SM and
// a split has to be worth its merge, 1.3 us: ten tiles and up (37 x 1290 in one piece 9.1 us, in four
// 12.2).  Two splits never beat one by more than they vary, and eight CTAs are a portable cluster
// (sixteen, merged through global memory, gained 3 % at 1 x 32768 and lost everywhere else).
int attn_flow_splits(int b, int s_max) {
  const int tiles = (s_max + kWarpChunk - 1) / kWarpChunk, ctas = kKvHeads * b;
  int own = 148 / ctas, shared = 2 * 148 / ctas;
  if (own > tiles / 4) own = tiles / 4;
  if (shared > tiles / 10) shared = tiles / 10;
  const int s = own > shared ? own : shared;
  return s < 3 ? 1 : s > 8 ? 8 : s;
}

int launch_attn_flow(const AttnArgs& a, int batch, int* status, cudaStream_t stream, int n_slots) {
  QUIC_REQUIRE(status != nullptr, QUIC_E_ARG, "attn_decode: no status word");
  CUtensorMap tm_k, tm_v;
  const int planes = n_slots > 0 ? n_slots : batch;
  int rc = make_kv_map(&tm_k, a.k, a.stride_b, a.stride_h, planes, a.s_cap);
  if (rc != QUIC_OK) return rc;
  rc = make_kv_map(&tm_v, a.v, a.stride_b, a.stride_h, planes, a.s_cap);
  if (rc != QUIC_OK) return rc;
  QUIC_CUDA(allow_smem<attn_decode_flow_kernel>(kFlowSmem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.splits, kKvHeads, batch);
  cfg.blockDim = dim3(kFlowWarps * 32);
  cfg.dynamicSmemBytes = kFlowSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)a.splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  // Only where two CTAs share an SM anyway: the CTAs of the next call find room beside those of this one, and where each
  // was to have an SM to itself some then share one (16 x 8192 16.4 -> 14.9 us a call, 9 x 8252 11.2 -> 11.8).  What it hides is
  // the set-up, and only behind a kernel that triggers early, one of this library's: those times are of calls in a row.
  cfg.numAttrs = pdl_enabled() && (n_slots > 0 || kKvHeads * batch * a.splits > 148) ? 2 : 1;
  QUIC_CUDA(cudaLaunchKernelEx(&cfg, attn_decode_flow_kernel, tm_k, tm_v, a, status));
  return QUIC_OK;
}

}  // namespace quic
