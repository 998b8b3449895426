// The four linears of a layer for a few rows (a decode batch, a short prompt), each in ONE launch
// with everything that stands around it: RMSNorm on the way in; bias, RoPE and KV append, residual
// add or SwiGLU on the way out.  Five launches a layer with the attention, where GEMMs with norms
// and split-K sums between them are seven or eight.
//
// Replaces, for up to 128 rows, rmsnorm.cu:39-86, marlin.cu:1527 (gemm.cu:36 for un-quantised
// weights), rope.cu:44-61, swiglu.cu:31-33 and the residual adds of src/model.py:211-224, with
// their rounding points.
//
// What bounds a layer of these sizes is not its work (64 rows: 0.4 us of weights, 0.8 us of MMAs) but the chain: 1.2-2 us
// from the last store of a kernel to the return of the next one's dependency wait, a round trip through L2 for its
// input, and shared memory (128 bytes a clock; the MMAs of a 128-wide stage read 36 KB).  So:
//
//   * The token rows are the M side of tcgen05.mma (64 or 128), the CTA's weight rows its N side.  A CTA owns all of K (an
//     eighth for `down`), so its weights are few and stay in shared memory: they are unpacked (or fetched by TMA,
//     un-quantised) BEFORE the dependency wait, under the kernels in front; a launch brings the next one's weights into
//     L2.  After the wait only rows move.
//   * 18 CTAs for qkv, 14 for o_proj, 134 for gate|up, 112 for down: neighbours in the chain find SMs of their own (an
//     attention of 64 rows has 128 CTAs), but for gate|up and down, and start early.  With 148, 98 and 56 CTAs of gate|up
//     and o_proj a fifth of gate|up started after its wait had returned and took 3 us longer.
//   * Norms: the kernel that writes the residual stream leaves sums of squares (one per row and CTA); the one that reads it
//     adds them up and multiplies the rows on their way to the MMAs.
//   * No split-K planes in global memory.  The eight CTAs of a cluster of `down` hand their sums to the one that finishes
//     the row, a bulk copy through distributed shared memory for each (remote stores of 16 bytes took twice as long), and
//     it adds them in the order of K.
//
// us per step, this / the GEMM step with norms and split-K sums between (7 or 8 launches a layer): 64 rows of 200..1500 tokens
// 834..850 / 911, 17 of 100..300 648..662 / 721, 48 of 64..200 696..710 / 768, 100 of 100..300 955 / 1080; un-quantised 17 rows
// 610..616 / 930, 40 of 300..1500 761..766 / 1123, 100 935 / 1355.
//
// Every mbarrier wait is bounded.  A role whose wait gives up says so to the CTA's others (fail_s) and goes on to the end; the CTA
// records a code, takes part in the cluster's barriers, waits for its own copies and MMAs in flight, frees its tensor memory and
// returns.  A wait for the accumulation may last as long as all of the MMA issuer's, and a CTA of a cluster sends its sums,
// whatever they are, and waits for those of the others twice as long, so that no copy is on its way to or from it when it leaves.
#include "tc_common.cuh"

namespace quic {
namespace {

constexpr int kOutRow = kHeadDim + 8;  // halves of a row of a head on its way out (another bank for every row)
enum RowsMode { kModeQkv, kModeOut, kModeSwiglu, kModeDown };

constexpr int kTileCols = 64;   // weight rows of a CTA of qkv (a head), o_proj and down
constexpr int kDownCluster = 8;  // CTAs that share the K of `down`
constexpr int kGateDense = 40;  // gate (and up) columns of a CTA, un-quantised: whole 1024-byte swizzle groups
constexpr int kGateCtas = 134;  // packed: 18 or 19 pairs of columns a CTA
constexpr int kGatePairs = kInter / 2 / kGateCtas, kGateMore = kInter / 2 % kGateCtas;
static_assert(kRowsSsq == kHidden / kTileCols, "sums of squares of a row");
constexpr int kConsumers = 512, kWarpsC = kConsumers / 32, kThreads = kConsumers + 64;  // + TMA warp, MMA warp
constexpr int kStageK = 2 * kBlockK;  // a stage of rows: two swizzle atoms, one quantisation group
constexpr uint32_t kSmemBudget = 223 * 1024;  // (of 227 KB, beside the barriers)

template <int MODE, int M, bool DENSE>
struct Cfg {
  static constexpr bool split = MODE == kModeDown;
  static constexpr bool norm = MODE == kModeQkv || MODE == kModeSwiglu;
  static constexpr int k = MODE == kModeDown ? kInter : kHidden, groups = k / kGroup;  // 38, 7
  static constexpr int cluster = split ? kDownCluster : 1;
  static constexpr int n_stages = (groups + cluster - 1) / cluster;  // of K in a CTA, at most
  // weight rows on the N side (multiples of 8 at M = 64, of 16 at M = 128; what is past a CTA's columns is never read back)
  static constexpr int n = MODE == kModeSwiglu ? 80 : kTileCols;
  static constexpr uint32_t cols = n <= 64 ? 64 : 128;  // of tensor memory
  static constexpr uint32_t w_atom = n * 128u, x_atom = M * 128u, w_stage = 2 * w_atom, x_stage = 2 * x_atom;
  static constexpr uint32_t ln_bytes = norm ? k * 2u + M * 8u : 0u;  // norm weights, the rows' factors
  static constexpr int own = M / cluster;                          // rows that a CTA of a cluster finishes
  static constexpr uint32_t red_bytes = split ? M * kTileCols * 4u : 0u;  // their parts
  // As many stages of rows as fit.  (Every role takes every stage, in order: a parity can only be that of the use it waits for.)
  static constexpr int fit = (int)((kSmemBudget - 1024u - n_stages * w_stage - ln_bytes - red_bytes) / x_stage);
  static constexpr int slots = fit >= n_stages ? n_stages : fit;
  static constexpr uint32_t off_ring = n_stages * w_stage, off_ln = off_ring + slots * x_stage, off_red = off_ln + ln_bytes;
  static constexpr size_t smem = off_red + red_bytes + 1024;
  static_assert(slots >= 2 && smem <= kSmemBudget && slots * x_stage >= red_bytes, "shared memory of a CTA");
  static constexpr int rounds = (2 * n_stages * (MODE == kModeSwiglu ? 4 * (kGatePairs + 1) : n) + kConsumers - 1) / kConsumers;
};

__device__ __forceinline__ void mbar_arrive_one(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// shared memory of this CTA -> that of a peer, counted in bytes on the peer's barrier
__device__ __forceinline__ void bulk_to_peer(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void prefetch_l2_bulk(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cons_bar() { asm volatile("bar.sync 1, %0;" ::"n"(kConsumers) : "memory"); }
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t mul_h2(uint32_t a, half2 b) {
  const half2 h = __hmul2(u32_as_half2(a), b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float round_h(float v) { return __half2float(__float2half_rn(v)); }

// columns that a CTA of packed gate|up weights owns
__device__ __forceinline__ int gate_first(int cta) { return 2 * (cta * kGatePairs + min(cta, kGateMore)); }
__device__ __forceinline__ int gate_count(int cta) { return 2 * (kGatePairs + (cta < kGateMore ? 1 : 0)); }

template <int MODE, int M, bool DENSE>
__global__ void __launch_bounds__(kThreads, 1)
    rows_linear_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w, const RowsArgs a) {
  using C = Cfg<MODE, M, DENSE>;
  constexpr int kS = C::slots, kOwn = C::own, kR = C::rounds;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[3 * kS + kR + 3];
  uint64_t* const bar_x = bars;               // a stage of rows landed
  uint64_t* const bar_ready = bar_x + kS;     // ... and is normalised
  uint64_t* const bar_empty = bar_ready + kS;  // ... and its MMAs are complete
  uint64_t* const bar_w = bar_empty + kS;     // a round of the CTA's weights is in shared memory (un-quantised: all of them)
  uint64_t &bar_done = bar_w[kR], &bar_red = bar_w[kR + 1], &bar_drain = bar_w[kR + 2];
  static_assert(3 * kS + kR + 3 <= 32, "a lane sets up a barrier");
  constexpr uint32_t kIssuerWaits = C::n_stages + kR;
  __shared__ uint32_t tmem_s;
  __shared__ int fail_s;
  __shared__ float ssq_s[4][M];
  __shared__ int slot_s[M], pos_s[M];  // qkv: of the rows

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* gen = smem_raw + (base - smem_u32(smem_raw));
  const int m0 = blockIdx.z * M;
  // this CTA's share of K (stages of 128) and of the weight rows; in a cluster, blockIdx.x is the rank
  const int rank = C::split ? (int)blockIdx.x : 0;
  const int stage0 = rank * C::groups / C::cluster, n_st = (rank + 1) * C::groups / C::cluster - stage0;
  const int cta_n = C::split ? blockIdx.y : blockIdx.x;
  const int n0 = MODE != kModeSwiglu ? cta_n * kTileCols : DENSE ? cta_n * kGateDense : gate_first(cta_n);
  // SwiGLU: gate columns of the CTA, and the weight row its up columns start at
  const int gcols = DENSE ? min(kGateDense, kInter - n0) : gate_count(cta_n);
  const int up0 = DENSE ? kGateDense : gcols;
  // Every CTA reads all the rows: each starts at another stage, or all would ask for the same lines of L2 at the same time.
  const int turn = C::split ? 0 : cta_n % n_st;
  auto atom_of = [&](int id) {  // id / ncols
    constexpr int few = (1 << 20) / (4 * kGatePairs) + 1, more = (1 << 20) / (4 * kGatePairs + 4) + 1;  // (exact below 4096)
    return MODE != kModeSwiglu ? id / kTileCols : (id * (gcols > 2 * kGatePairs ? more : few)) >> 20;
  };
  auto k_stage = [&](int it) {  // the it-th stage that this CTA multiplies
    const int at = it + turn;
    return stage0 + (at >= n_st ? at - n_st : at);
  };
  const int ncols = MODE == kModeSwiglu && !DENSE ? 2 * gcols : kTileCols, items = 2 * n_st * ncols;  // a packed item: eight words of a column, an atom

  // Packed weights are on their way before anything else: a CTA that finds its SM late has little time for them.
  uint32_t q[kR][8], zp[kR];
  half sc[kR];
  if (!DENSE && warp < kWarpsC) {
    const int N = a.w.n;
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const int id = tid + r * kConsumers;
      if (id < items) {
        const int it = atom_of(id), c = id - it * ncols, g = k_stage(it >> 1);
        const int col = MODE == kModeSwiglu && c >= gcols ? kInter + n0 + c - gcols : n0 + c;
        const uint32_t* src = reinterpret_cast<const uint32_t*>(a.w.qw) + (size_t)(g * 16 + (it & 1) * 8) * N + col;
#pragma unroll
        for (int j = 0; j < 8; ++j) q[r][j] = ldg_nc_u32(src + (size_t)j * N);
        sc[r] = __ldg(reinterpret_cast<const half*>(a.w.sc) + (size_t)g * N + col);
        zp[r] = __ldg(a.w.zp + (size_t)g * (N >> 1) + (col >> 1)) >> (4 * (col & 1));
      }
    }
  }

  if (warp == kWarpsC) {
    if (lane < 3 * kS + kR + 3)
      mbar_init(smem_u32(&bars[lane]), lane >= kS && lane < 2 * kS ? kWarpsC : lane >= 3 * kS && lane < 3 * kS + kR && !DENSE ? kWarpsC : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
      fail_s = 0;
      if (C::split) mbar_expect_tx(smem_u32(&bar_red), C::red_bytes);
      if (!C::norm) tma_prefetch_desc(&tm_x);
      if (DENSE) tma_prefetch_desc(&tm_w);
    }
  }
  if (warp == kWarpsC + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "r"(C::cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_d = tmem_s;
  if (C::split) cluster_arrive();  // (a peer's shared memory is written only once the peer runs)
  pdl_launch_dependents();

  // The accumulator comes back in blocks of 16 rows and 8 columns, a thread with two columns of rows g and g + 8.  At M = 64
  // rows 16 q .. 16 q + 15 are lanes 32 q .. 32 q + 15 of tensor memory, at M = 128 a warp has two blocks of rows.
  constexpr int kHalves = M / 64;
  const int quarter = warp & 3, cgroup = (warp >> 2) & 3, g = lane >> 2, c2 = 2 * (lane & 3);
  const uint32_t lane_addr = tmem_d + ((uint32_t)(quarter * 32) << 16);
  auto row_of = [&](int h, int i) { return quarter * (16 * kHalves) + 16 * h + 8 * i + g; };  // (of the tile)
  auto here = [&](int h, int i) { return warp < kWarpsC && m0 + row_of(h, i) < a.rows; };
  // `down`: a thread finishes four columns of a row that the CTA owns
  const int frow = tid >> 4, fcol = (tid & 15) * 4, fm = m0 + rank * kOwn + frow;
  const bool finishes = C::split && tid < kOwn * 16 && fm < a.rows;
  // what the epilogue adds: residual, or cosines and sines; of a thread's (block of rows, row, block of columns)
  constexpr bool kAdds = MODE == kModeQkv || MODE == kModeOut;
  uint32_t ea[kAdds ? kHalves : 1][2][2] = {}, eb[kAdds ? kHalves : 1][2][2] = {}, bias2[2] = {};
  uint2 fres = {};
  // norm: weights; per row the power of two in 1 / rms (both halves of a word) and what is left of it
  uint4* const ln_s = reinterpret_cast<uint4*>(gen + C::off_ln);
  uint32_t* const pow_s = reinterpret_cast<uint32_t*>(ln_s + C::k / 8);
  float* const rest_s = reinterpret_cast<float*>(pow_s + M);

  bool issuer = false;
  if (warp == kWarpsC) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      if (DENSE) {
        const uint32_t full = smem_u32(&bar_w[0]);
        constexpr int boxes = MODE == kModeSwiglu ? 2 : 1, box_bytes = (MODE == kModeSwiglu ? kGateDense : C::n) * 128;
        mbar_expect_tx(full, (uint32_t)(2 * n_st * boxes * box_bytes));
        for (int it = 0; it < 2 * n_st; ++it)
          for (int i = 0; i < boxes; ++i)  // (rows past the end of the matrix read as zero)
            tma_load_2d(base + it * C::w_atom + i * box_bytes, &tm_w, k_stage(it >> 1) * kStageK + (it & 1) * kBlockK, n0 + i * kInter, full);
      }
      pdl_wait();
      int issued = 0;
      for (int s = 0, pass = 0; !C::norm && issued < n_st; ++issued) {
        if (pass > 0 && !mbar_wait(smem_u32(&bar_empty[s]), (pass - 1) & 1, a.wait_limit_us)) {
          fail_s = 2;
          break;
        }
        const uint32_t full = smem_u32(&bar_x[s]);
        if (a.skip_stage < -1) pause_us(-a.skip_stage);
        mbar_expect_tx(full, C::x_stage);
        if (issued != a.skip_stage) tma_load_3d(base + C::off_ring + s * C::x_stage, &tm_x, 0, m0, 2 * k_stage(issued), full);
        if (++s == kS) s = 0, ++pass;
      }
      // weights that the next launch will find in L2
      const int ctas = gridDim.x * gridDim.y * gridDim.z, cta = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
#pragma unroll
      for (int i = 0; i < (DENSE ? 1 : 3); ++i) {
        const int64_t part = (a.next_bytes[i] / ctas + 127) / 128 * 128, left = a.next_bytes[i] - part * cta;
        if (left > 0) prefetch_l2_bulk(static_cast<const char*>(a.next_w[i]) + part * cta, (uint32_t)(left < part ? left : part) & ~15u);
      }
      // no copy may be on its way into this CTA's shared memory when it ends, whatever became of the other roles
      for (int i = issued > kS ? issued - kS : 0; i < issued; ++i)
        if (!mbar_wait(smem_u32(&bar_x[i % kS]), (i / kS) & 1, a.wait_limit_us)) fail_s = 2;
      if (DENSE && !mbar_wait(smem_u32(&bar_w[0]), 0, a.wait_limit_us)) fail_s = 1;
    }
  } else if (warp == kWarpsC + 1) {
    // ---------------- MMA issuer ----------------
    issuer = elect_one();
    if (issuer) {
      const uint32_t idesc = umma_idesc_f16(M, C::n);
      const uint64_t x0 = umma_desc_sw128(base + C::off_ring), w0 = umma_desc_sw128(base);
      bool ok = true;
      for (int it = 0, s = 0, pass = 0, r = 0; it < n_st; ++it) {
        const int need = DENSE ? 1 : (2 * (it + 1) * ncols + kConsumers - 1) / kConsumers;  // rounds of weights up to this stage
        for (; r < need && ok; ++r) ok = mbar_wait(smem_u32(&bar_w[r]), 0, a.wait_limit_us);
        if (it == 0) pdl_wait();  // the rows cannot be here earlier, and the limit is not for the kernel in front
        ok = ok && mbar_wait(smem_u32(C::norm ? &bar_ready[s] : &bar_x[s]), pass & 1, a.wait_limit_us);
        if (!ok) break;
        if (it == 0) tc_fence_after();
        const uint64_t x = x0 + (uint64_t)(s * (C::x_stage / 16)), w = w0 + (uint64_t)(it * (C::w_stage / 16));
#pragma unroll
        for (int k = 0; k < kStageK / 16; ++k)
          umma_f16(tmem_d, x + (k / 4) * (C::x_atom / 16) + 2 * (k % 4), w + (k / 4) * (C::w_atom / 16) + 2 * (k % 4), idesc,
                   (it > 0 || k > 0) ? 1u : 0u);
        if (it + kS < n_st) umma_commit(smem_u32(&bar_empty[s]));
        if (it == n_st - 1) umma_commit(smem_u32(&bar_done));
        if (++s == kS) s = 0, ++pass;
      }
      if (!ok) fail_s = 3;
    }
  } else {
    // ---------------- weights: a thread turns eight packed words of a column into one 128-byte row of an atom ----------------
    if (C::norm && tid < C::k / 8) ln_s[tid] = __ldg(reinterpret_cast<const uint4*>(a.ln) + tid);
    if (MODE == kModeQkv) {
      const half* bias = reinterpret_cast<const half*>(a.w.bias) + n0 + cgroup * 16 + c2;
      bias2[0] = __ldg(reinterpret_cast<const uint32_t*>(bias));
      bias2[1] = __ldg(reinterpret_cast<const uint32_t*>(bias + 8));
    }
    if (!DENSE) {
#pragma unroll
      for (int r = 0; r < kR; ++r) {
        const int id = tid + r * kConsumers;
        if (id < items) {
          const int it = atom_of(id), c = id - it * ncols;
          const half2 s2 = __half2half2(sc[r]), z2 = zp_to_half2((int)(zp[r] & 15));
          unsigned char* dst = gen + it * C::w_atom;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            half2 d[4];
            dequant8(q[r][j], z2, s2, d);  // d[p] = (k = p, k = p + 4)
            const uint32_t u0 = *reinterpret_cast<uint32_t*>(&d[0]), u1 = *reinterpret_cast<uint32_t*>(&d[1]);
            const uint32_t u2 = *reinterpret_cast<uint32_t*>(&d[2]), u3 = *reinterpret_cast<uint32_t*>(&d[3]);
            uint4 o;
            o.x = __byte_perm(u0, u1, 0x5410);
            o.y = __byte_perm(u2, u3, 0x5410);
            o.z = __byte_perm(u0, u1, 0x7632);
            o.w = __byte_perm(u2, u3, 0x7632);
            *reinterpret_cast<uint4*>(dst + sw128_offset(c, j)) = o;
          }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive_one(smem_u32(&bar_w[r]));
      }
    }
    pdl_wait();
    // what the epilogue adds is requested before the accumulation is waited for
    if constexpr (MODE == kModeOut) {
#pragma unroll
      for (int h = 0; h < kHalves; ++h)
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (here(h, i)) {
            const half* res = a.res + (size_t)(m0 + row_of(h, i)) * kHidden + n0 + cgroup * 16 + c2;
            ea[h][i][0] = *reinterpret_cast<const uint32_t*>(res);
            ea[h][i][1] = *reinterpret_cast<const uint32_t*>(res + 8);
          }
    }
    if (finishes) fres = *reinterpret_cast<const uint2*>(a.res + (size_t)fm * kHidden + n0 + fcol);
    if (MODE == kModeQkv && tid < M) {
      int slot = m0 + tid < a.rows ? a.slots[m0 + tid] : -1;
      if (slot >= a.n_slots) slot = -1;  // a row with a slot outside the cache appends nothing
      slot_s[tid] = slot;
      pos_s[tid] = m0 + tid >= a.rows ? 0 : a.row_pos != nullptr ? a.row_pos[m0 + tid] : slot >= 0 ? __ldcg(a.pos + slot) : 0;
    }
    // Norm: a thread has one of a stage's sixteen 16-byte pieces of every 32nd row.  The rows come through registers; rows past the
    // end are left out (what their accumulators hold is never read).  By TMA and in place a stage took as long at 64
    // rows (650 clocks: shared memory gives 128 bytes a clock, and the MMAs alone read 36 KB), 0.3 us more in all at 24.
    constexpr int kRow = kConsumers / 16, kRows = M / kRow, kAhead = C::norm ? 2 : 1;  // stages in flight
    const int piece = tid & 15, r0 = tid >> 4;
    uint4 x[kAhead][kRows];
    auto load_rows = [&](int it) {
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        const int r = m0 + r0 + i * kRow;
        if (r < a.rows) x[it % kAhead][i] = __ldcg(reinterpret_cast<const uint4*>(a.x + (size_t)r * C::k + k_stage(it) * kStageK) + piece);
      }
    };
    if constexpr (C::norm) {
      // ---------------- the rows' factors: eight lanes a row, every sum requested at once ----------------
      constexpr int kPer = M * 8 / kConsumers, kParts = (kRowsSsq + 7) / 8;
      float v[kPer][kParts];
#pragma unroll
      for (int i = 0; i < kPer; ++i)
#pragma unroll
        for (int j = 0; j < kParts; ++j) {
          const int r = m0 + (tid >> 3) + i * (kConsumers / 8), at = (tid & 7) + 8 * j;
          v[i][j] = r < a.rows && at < a.n_ssq ? __ldcg(a.ssq_in + (size_t)r * kRowsSsq + at) : 0.f;
        }
#pragma unroll
      for (int it = 0; it < kAhead; ++it) load_rows(it);
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        float sum = v[i][0];
#pragma unroll
        for (int j = 1; j < kParts; ++j) sum += v[i][j];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if ((tid & 7) == 0) {
          const int r = (tid >> 3) + i * (kConsumers / 8);
          // (at most 2^15, what fp16 holds: eps below 2^-32 lets rows of zeros and of its smallest values go beyond)
          const float rs = rsqrtf(sum * (1.0f / kHidden) + a.eps), pw = fminf(__uint_as_float(__float_as_uint(rs) & 0x7f800000u), 32768.f);
          const half2 h = __float2half2_rn(pw);
          pow_s[r] = *reinterpret_cast<const uint32_t*>(&h);
          rest_s[r] = rs / pw;
        }
      }
      cons_bar();
    }
    if constexpr (MODE == kModeQkv) {  // pairs: a block of columns has four, one a thread
#pragma unroll
      for (int h = 0; h < kHalves; ++h)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int pos = pos_s[row_of(h, i)], pp = pos < a.max_pos ? (pos < 0 ? 0 : pos) : a.max_pos - 1;
          const size_t at = (size_t)pp * 32 + cgroup * 8 + (lane & 3);
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            ea[h][i][b] = __half_as_ushort(__ldg(a.cos_t + at + 4 * b));
            eb[h][i][b] = __half_as_ushort(__ldg(a.sin_t + at + 4 * b));
          }
        }
    }
    if constexpr (C::norm) {
      // ---------------- the rows' norm ----------------
      // fp16(x * 2^e * w), and the rest of 1 / rms, 1 <= r < 2, is a factor of the row's sums in the epilogue.  2^e * x is
      // exact, so there is one rounding, as fp16(x / rms * w) has, for two multiplies of pairs.  (What lies below 2^-14 of
      // the row's root mean square is rounded to fp16's subnormals first: up to 2^-25 (|w| + 1) r off, against the
      // 2^-12 |w| of a value as large as the mean.)
      half2 pw[kRows];
#pragma unroll
      for (int i = 0; i < kRows; ++i) pw[i] = u32_as_half2(pow_s[r0 + i * kRow]);
#pragma unroll
      for (int it = 0; it < C::n_stages; ++it) {
        const int s = it % kS;
        const uint4 w = ln_s[k_stage(it) * 16 + piece];
        if (it >= kS && !mbar_wait(smem_u32(&bar_empty[s]), (it / kS - 1) & 1, a.wait_limit_us)) {
          fail_s = 1;
          break;
        }
        unsigned char* const at = gen + C::off_ring + s * C::x_stage + (piece >> 3) * C::x_atom;
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
          if (m0 + r0 + i * kRow >= a.rows) continue;
          uint4 v = x[it % kAhead][i];
          v.x = mul_h2(mul_h2(v.x, pw[i]), u32_as_half2(w.x));
          v.y = mul_h2(mul_h2(v.y, pw[i]), u32_as_half2(w.y));
          v.z = mul_h2(mul_h2(v.z, pw[i]), u32_as_half2(w.z));
          v.w = mul_h2(mul_h2(v.w, pw[i]), u32_as_half2(w.w));
          *reinterpret_cast<uint4*>(at + sw128_offset(r0 + i * kRow, piece & 7)) = v;
        }
        if (it + kAhead < C::n_stages) load_rows(it + kAhead);
        fence_proxy_async();
        __syncwarp();
        if (a.skip_stage < -1) pause_us(-a.skip_stage);
        if (lane == 0 && it != a.skip_stage) mbar_arrive_one(smem_u32(&bar_ready[s]));
      }
    }
  }
  __syncwarp();

  bool ok = true;
  if (warp < kWarpsC) {
    ok = mbar_wait_unless(smem_u32(&bar_done), 0, &fail_s, a.wait_limit_us * (kIssuerWaits + 1));
    ok = __all_sync(0xffffffffu, ok);  // tcgen05.ld below is warp-collective
    tc_fence_after();
    if (!ok) fail_s = 3;
  }
  if constexpr (MODE == kModeQkv) {
    if (warp < kWarpsC && ok) {
      // a CTA has a head, whose stored columns (2 j, 2 j + 1) are dims (j, j + 32)
      const int head = cta_n;
      const bool turned = head < kHeads + kKvHeads;  // q and k
#pragma unroll
      for (int h = 0; h < kHalves; ++h) {
        float v[2][4];
        tmem_ld_16x8<2>(lane_addr + ((uint32_t)(16 * h) << 16) + (uint32_t)(cgroup * 16), v);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          half* dst = reinterpret_cast<half*>(gen + C::off_ring) + row_of(h, i) * kOutRow + cgroup * 8 + (lane & 3);
          const float rest = rest_s[row_of(h, i)];
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const float2 bb = __half22float2(u32_as_half2(bias2[b]));
            const float x = round_h(round_h(v[b][2 * i] * rest) + bb.x), y = round_h(round_h(v[b][2 * i + 1] * rest) + bb.y);
            const float cs = __half2float(__ushort_as_half((unsigned short)ea[h][i][b])), sn = __half2float(__ushort_as_half((unsigned short)eb[h][i][b]));
            dst[4 * b] = __float2half_rn(turned ? x * cs - y * sn : x);
            dst[4 * b + 32] = __float2half_rn(turned ? x * sn + y * cs : y);
          }
        }
      }
    }
    if (warp < kWarpsC) {  // (the ring is free: the head's rows leave from there in 16-byte pieces)
      const int head = cta_n;
      cons_bar();
      for (int r = tid >> 3; r < M && m0 + r < a.rows && ok; r += kConsumers / 8) {
        const int pos = pos_s[r], slot = slot_s[r];
        half* dst = nullptr;
        if (head < kHeads) {
          dst = a.y + (a.head_major ? (size_t)head * a.rows + m0 + r : (size_t)(m0 + r) * kHeads + head) * kHeadDim;
        } else if (slot >= 0 && pos >= 0 && pos < a.s_max) {
          half* plane = head < kHeads + kKvHeads ? a.kcache : a.vcache;
          dst = plane + (((size_t)slot * kKvHeads + (head - kHeads) % kKvHeads) * a.s_max + pos) * kHeadDim;
        }
        if (dst != nullptr)
          reinterpret_cast<uint4*>(dst)[tid & 7] = reinterpret_cast<const uint4*>(gen + C::off_ring + r * kOutRow * 2)[tid & 7];
      }
    }
  } else if constexpr (MODE == kModeOut) {
    if (warp < kWarpsC) {
#pragma unroll
      for (int h = 0; h < kHalves; ++h) {
        float v[2][4] = {};
        if (ok) tmem_ld_16x8<2>(lane_addr + ((uint32_t)(16 * h) << 16) + (uint32_t)(cgroup * 16), v);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float ssq = 0.f;
          if (here(h, i) && ok) {
            half* dst = a.y + (size_t)(m0 + row_of(h, i)) * kHidden + n0 + cgroup * 16 + c2;
#pragma unroll
            for (int b = 0; b < 2; ++b) {
              const float2 r2 = __half22float2(u32_as_half2(ea[h][i][b]));
              const uint32_t o = pack2(round_h(v[b][2 * i]) + r2.x, round_h(v[b][2 * i + 1]) + r2.y);
              *reinterpret_cast<uint32_t*>(dst + 8 * b) = o;
              const float2 f = __half22float2(u32_as_half2(o));
              ssq = fmaf(f.x, f.x, ssq);
              ssq = fmaf(f.y, f.y, ssq);
            }
          }
          ssq += __shfl_xor_sync(0xffffffffu, ssq, 1);
          ssq += __shfl_xor_sync(0xffffffffu, ssq, 2);
          if ((lane & 3) == 0) ssq_s[cgroup][row_of(h, i)] = ssq;
        }
      }
      cons_bar();
      if (tid < M && m0 + tid < a.rows)
        a.ssq_out[(size_t)(m0 + tid) * kRowsSsq + cta_n] = (ssq_s[0][tid] + ssq_s[1][tid]) + (ssq_s[2][tid] + ssq_s[3][tid]);
    }
  } else if constexpr (MODE == kModeSwiglu) {
    if (warp < kWarpsC && ok) {
      // a warp takes eight gate columns and the same up columns at a time
#pragma unroll 1
      for (int c = cgroup * 8; c < gcols; c += 32) {
#pragma unroll
        for (int h = 0; h < kHalves; ++h) {
          float gt[4], up[4];
          tmem_ld_16x8_two(lane_addr + ((uint32_t)(16 * h) << 16) + (uint32_t)c, lane_addr + ((uint32_t)(16 * h) << 16) + (uint32_t)(up0 + c), gt, up);
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (here(h, i) && c + c2 < gcols) {
              const float rest = rest_s[row_of(h, i)];
              *reinterpret_cast<uint32_t*>(a.y + (size_t)(m0 + row_of(h, i)) * kInter + n0 + c + c2) =
                  pack2(silu_mul(round_h(gt[2 * i] * rest), round_h(up[2 * i] * rest)),
                        silu_mul(round_h(gt[2 * i + 1] * rest), round_h(up[2 * i + 1] * rest)));
            }
        }
      }
    }
  } else {
    // Every row's parts go to the CTA of the cluster that finishes the row: into the (by now free) ring, then one copy for each peer.
    // A row's sixteen 16-byte pieces are turned by the row, so that the lanes of a store fall into different banks.
    if (warp < kWarpsC) {
#pragma unroll
      for (int h = 0; h < kHalves; ++h) {
        float v[2][4];
        if (ok) tmem_ld_16x8<2>(lane_addr + ((uint32_t)(16 * h) << 16) + (uint32_t)(cgroup * 16), v);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int r = row_of(h, i);
#pragma unroll
          for (int b = 0; b < 2; ++b)
            if (ok)
              *reinterpret_cast<float2*>(gen + C::off_ring + r * (kTileCols * 4) + (((cgroup * 4 + b * 2 + (c2 >> 2)) ^ (r & 7)) << 4) + (c2 & 2) * 4) =
                  make_float2(v[b][2 * i], v[b][2 * i + 1]);
        }
      }
      fence_proxy_async();
      cons_bar();
    }
    cluster_wait();  // every peer runs
    constexpr uint32_t kPart = kOwn * kTileCols * 4u;
    if (tid < C::cluster)
      bulk_to_peer(peer_addr(base + C::off_red + rank * kPart, tid), base + C::off_ring + tid * kPart, kPart,
                   peer_addr(smem_u32(&bar_red), tid));
    if (warp < kWarpsC) {
      if (!mbar_wait(smem_u32(&bar_red), 0, a.wait_limit_us * 2 * (kIssuerWaits + 1))) {
        ok = false;
        fail_s = 4;
      }
    }
    __syncwarp();
    cluster_arrive();  // this CTA has all its parts; when all have, nobody reads a ring any more
    float ssq = 0.f;
    if (finishes && ok) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4* red = reinterpret_cast<const float4*>(gen + C::off_red) + frow * (kTileCols / 4) + ((tid & 15) ^ ((rank * kOwn + frow) & 7));
#pragma unroll
      for (int s = 0; s < C::cluster; ++s) {  // in the order of K
        const float4 f = red[s * kOwn * (kTileCols / 4)];
        acc.x += f.x;
        acc.y += f.y;
        acc.z += f.z;
        acc.w += f.w;
      }
      const float2 ra = __half22float2(u32_as_half2(fres.x)), rb = __half22float2(u32_as_half2(fres.y));
      const uint2 o = make_uint2(pack2(round_h(acc.x) + ra.x, round_h(acc.y) + ra.y), pack2(round_h(acc.z) + rb.x, round_h(acc.w) + rb.y));
      *reinterpret_cast<uint2*>(a.y + (size_t)fm * kHidden + n0 + fcol) = o;
      const float2 fa = __half22float2(u32_as_half2(o.x)), fb = __half22float2(u32_as_half2(o.y));
      ssq = fmaf(fa.x, fa.x, fa.y * fa.y) + fmaf(fb.x, fb.x, fb.y * fb.y);
    }
    if (warp < kOwn * 16 / 32) {
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, o);
      if (finishes && ok && (tid & 15) == 0) a.ssq_out[(size_t)fm * kRowsSsq + cta_n] = ssq;
    }
    __syncwarp();
    cluster_wait();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kWarpsC + 1) {  // (the issuer's warp: the CTA's memory stays until it has left, whenever the others do)
    if (fail_s != 0) {
      if (lane == 0) tc_report(a.status, (fail_s << 16) | 0x2000 | (int)(blockIdx.x & 0x1fff));
      drain_failed_warp(issuer, smem_u32(&bar_drain));
    }
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(C::cols) : "memory");
  }
}

// x[b] = embed[token of row b] and the row's sum of squares.
__global__ void __launch_bounds__(224) embed_ssq_kernel(const half* __restrict__ embed, const int32_t* __restrict__ slots,
                                                        const int32_t* __restrict__ tok, int vocab, half* __restrict__ x,
                                                        float* __restrict__ ssq) {
  __shared__ float red[7];
  const int b = blockIdx.x, t = threadIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  int id = slots != nullptr ? tok[slots[b]] : tok[b];
  id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
  const uint2 v = reinterpret_cast<const uint2*>(embed + (size_t)id * kHidden)[t];
  reinterpret_cast<uint2*>(x + (size_t)b * kHidden)[t] = v;
  const float2 f = __half22float2(u32_as_half2(v.x)), g = __half22float2(u32_as_half2(v.y));
  const float s = warp_sum(f.x * f.x + f.y * f.y + g.x * g.x + g.y * g.y);
  if ((t & 31) == 0) red[t >> 5] = s;
  __syncthreads();
  if (t == 0) {
    float sum = 0.f;
    for (int i = 0; i < 7; ++i) sum += red[i];
    ssq[(size_t)b * kRowsSsq] = sum;
  }
}

template <int MODE, int M, bool DENSE>
int launch_rows(const half* x, const RowsArgs& a, cudaStream_t st, bool pdl) {
  using C = Cfg<MODE, M, DENSE>;
  CUtensorMap tm_x = {}, tm_w;
  // the rows as [K / 64][rows][64], so that one copy brings the two swizzle atoms of a stage
  const cuuint64_t dims[3] = {kBlockK, (cuuint64_t)a.rows, C::k / kBlockK}, strides[2] = {C::k * 2, kBlockK * 2};
  const cuuint32_t box[3] = {kBlockK, M, 2};
  int rc = QUIC_OK;
  if (!C::norm)
    rc = make_tiled_map(&tm_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, x, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
  if (rc != QUIC_OK) return rc;
  tm_w = tm_x;
  if (DENSE) {
    rc = make_map(&tm_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.w.w16, (uint64_t)a.w.n, C::k, MODE == kModeSwiglu ? kGateDense : C::n, kBlockK,
                  CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != QUIC_OK) return rc;
  }
  QUIC_CUDA((allow_smem<rows_linear_kernel<MODE, M, DENSE>>(C::smem)));
  const int mtiles = (a.rows + M - 1) / M;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = C::split ? dim3(C::cluster, kHidden / kTileCols, mtiles)
                : MODE == kModeSwiglu ? dim3(DENSE ? (kInter + kGateDense - 1) / kGateDense : kGateCtas, 1, mtiles)
                                      : dim3((MODE == kModeQkv ? kQkvN : kHidden) / kTileCols, 1, mtiles);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = C::smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (pdl && pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (C::split) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = C::cluster;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  QUIC_CUDA(cudaLaunchKernelEx(&cfg, rows_linear_kernel<MODE, M, DENSE>, tm_x, tm_w, a));
  return QUIC_OK;
}

template <int MODE>
int run_rows(const half* x, RowsArgs a, cudaStream_t st, bool pdl) {
  QUIC_REQUIRE(a.rows >= 1 && a.rows <= 65535 * 128, QUIC_E_SHAPE, "rows_linear: bad row count");
  a.x = x;
  a.status = tc_status_words();
  QUIC_REQUIRE(a.status != nullptr, QUIC_E_CUDA, "rows_linear: no error word");
  tc_test_hook(&a.wait_limit_us, &a.skip_stage);
  const bool dense = a.w.w16 != nullptr;
  if (a.rows <= 64) return dense ? launch_rows<MODE, 64, true>(x, a, st, pdl) : launch_rows<MODE, 64, false>(x, a, st, pdl);
  return dense ? launch_rows<MODE, 128, true>(x, a, st, pdl) : launch_rows<MODE, 128, false>(x, a, st, pdl);
}

}  // namespace

void rows_next(RowsArgs* a, const quic_w4_t* w) {
  const void* const at[3] = {w == nullptr ? nullptr : w->w16 != nullptr ? (const void*)w->w16 : (const void*)w->qw,
                             w != nullptr ? (const void*)w->sc : nullptr, w != nullptr ? (const void*)w->zp : nullptr};
  const int64_t words = w != nullptr ? (int64_t)w->n * w->k : 0;
  const bool dense = w != nullptr && w->w16 != nullptr;
  const int64_t bytes[3] = {dense ? words * 2 : words / 2, dense ? 0 : words / kGroup * 2, dense ? 0 : words / kGroup / 2};
  for (int i = 0; i < 3; ++i) {
    a->next_w[i] = at[i];
    a->next_bytes[i] = bytes[i];
  }
}
int rows_qkv(const half* x, const RowsArgs& a, cudaStream_t st) { return run_rows<kModeQkv>(x, a, st, true); }
int rows_out(const half* x, const RowsArgs& a, cudaStream_t st) { return run_rows<kModeOut>(x, a, st, true); }
int rows_swiglu(const half* x, const RowsArgs& a, cudaStream_t st) { return run_rows<kModeSwiglu>(x, a, st, true); }
int rows_down(const half* x, const RowsArgs& a, cudaStream_t st) { return run_rows<kModeDown>(x, a, st, true); }

cudaError_t launch_embed_ssq(const half* embed, const int32_t* slots, const int32_t* tok, int vocab, half* x, float* ssq, int rows,
                             cudaStream_t st, bool pdl) {
  return launch(embed_ssq_kernel, dim3(rows), dim3(224), 0, st, pdl, embed, slots, tok, vocab, x, ssq);
}

}  // namespace quic
