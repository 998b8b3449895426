// The whole decode token loop as ONE persistent kernel: 148 resident CTAs walk the 24 layers
// and the lm_head of every token of a burst and hand each layer phase's result to the next
// through tagged 16-byte words in L2, while the weights stream from HBM into a shared-memory
// ring that does not wait for that dependency chain.
//
// Replaces, for up to kMaxRows batch rows, Engine.step + QUICForCausalLM.forward with
// seq_len == 1 of the reference (src/engine.py:78-107, src/model.py:211-224, 272-303) with the
// rounding points of the kernel chain (decode_layers.cu): dequant kernels/cuda/marlin.cu:2290-2313,
// RMSNorm rmsnorm.cu:39-86, RoPE rope.cu:44-61, attention flash_attn_decode.cu:82-130, SwiGLU
// swiglu.cu:31-33, argmax sampler.cu:38-40; and for un-quantised weights gemm.cu:36.
//
// What bounds a step is not bandwidth (466 MB = 71 us at one row) but five dependent all-to-all
// exchanges per layer.  A dependent kernel launch costs 0.7 us on this part even when the
// kernel is empty and its input then takes a round trip to L2; here data and "ready" signal travel
// in one word, and what does not depend on the exchange (weights fetched, unpacked and laid out as
// mma fragments in registers, cached keys and values as fragments) is in place before the word
// arrives.  Measured per layer at one row: ~1 us from a publication to the last reader's arithmetic,
// five times, and 0.3 to 1.8 us of arithmetic and reductions per phase (the attention of one KV head
// on one SM is the longest).  Per step, persistent / kernel chain: 345 / 353 us at one row of 520
// tokens (350 / 333 at 500, where the chain needs no merge: it serves one packed row up to 512), 373 / 462 at
// two, 408 / 653 at five of 700, 445 / 667 at eight of 1000, 500 / 704 at 16 of 300; fp16 weights 348 / 494 at
// one row, 416 / 899 at eight.
//
// Roles (a CTA can have several; `na` = attention CTAs, the last ones of the grid):
//   residual   CTAs 0..55    16 output columns of o_proj AND of down; the residual stream of those
//                            columns stays in the CTA from token to token
//   qkv        CTAs 56..     one to three 16-column tiles (8 rotation pairs) of the fused QKV linear
//   gate|up    all but `na`  tiles of 8 gate + the same 8 up columns, SwiGLU in the CTA
//   attention  `na` CTAs     (row, KV head, split of the context): the cache tiles of the next layer
//                            arrive in shared memory while the other CTAs run theirs
//   lm_head    all           16-row tiles of the table, candidates exchanged, every CTA finds the argmax
// A linear's tile is 16 weight rows on the M side of mma.sync.m16n8k16 with the batch rows on N, so
// one to eight rows cost nearly the same; K is split over the 14 compute warps of the CTA, whose
// partial sums meet in shared memory.  A warp polls the words of its own slice of K straight into its
// B fragments: no staging, one barrier (the partial sums) between an input and an output, two
// where a norm needs the whole row.  tcgen05 would need its operands in shared memory first.
//
// Weight stream ("W4S" / its fp16 form): chunks of one 16-byte piece per compute thread, in the
// order the CTA's phases consume them.  Packed: a piece = the lane's A fragments of four k steps
// (one 32-bit word each), the scales and zero points of the chunk in front of them.  fp16: a piece =
// the A fragment of one k step.  A chunk belongs to a tile, not to a CTA, so any assignment of
// tiles to CTAs reads the same stream.
//
// Words: eight fp16 values (or four fp32) in one 128-bit store; the all-zero word means "not there yet".
// Each exchange buffer exists three times (layer number mod 3): a word is emptied one layer before
// it is written again, by its writer, when everybody who read its last contents has been heard from
// (transitively), and every launch leaves all of them empty.  A lm_head candidate carries the number of
// its token's last layer instead; those words are emptied when a launch starts.
//
// Waits: every poll and every mbarrier wait is bounded; on a timeout the CTA records a code in
// the status word, the others see it within a few hundred probes, all wait for their own copies in
// flight and return.  The kernel is launched cooperatively (all CTAs resident), and launches of
// one process on different streams are ordered one after another.
#include <mutex>

#include "attn_warp.cuh"
#include "decode_kernels.cuh"
#include "tc_common.cuh"

namespace quic {
namespace {

using u64 = unsigned long long;

constexpr int kCtas = 148;
constexpr int kWarps = 14;                    // compute warps; K = 896 is 56 k steps, four per warp
constexpr int kComp = kWarps * 32;            // 448 compute threads
constexpr int kThreads = kComp + 32;          // + the producer warp
constexpr int kMaxRows = 16;
constexpr int kMaxLayers = 64;
constexpr int kMaxAttnCtas = 60;
constexpr int kGroupHeads = kHeads / kKvHeads;

constexpr int kResCtas = 56, kResCols = 16;   // 56 x 16 = 896
constexpr int kQkvTiles = kQkvN / 16;         // 72
constexpr int kGuTiles = kInter / 8;          // 608
constexpr int kDownPieces = 6;                // k steps 56 p + 4 warp + j; the last piece fills 6 warps only
constexpr int kDownLastWarps = (kInter / 16 - 5 * 56) / 4;  // 6
static_assert(kResCtas * kResCols == kHidden && kDownLastWarps == 6, "tiling");

constexpr int kPieceBytes = kComp * 16;       // 7168
constexpr int kScaleBytes = kWarps * 64;      // per warp: 8 x {s_g, s_g+8, 1024 + zp_g, 64 + zp_g+8}, fp16
template <bool F16> struct Wt {
  static constexpr int chunk = F16 ? kPieceBytes : kPieceBytes + kScaleBytes;  // 7168 / 8064
  static constexpr int per_piece = F16 ? 4 : 1;                                // chunks of four k steps per warp
  static constexpr int last_down = F16 ? kDownLastWarps * 512 : kScaleBytes + kDownLastWarps * 512;
  static constexpr int off_o = kQkvTiles * per_piece;
  static constexpr int off_gu = off_o + kResCtas * per_piece;
  static constexpr int off_down = off_gu + kGuTiles * per_piece;
  static constexpr int per_layer = off_down + kResCtas * kDownPieces * per_piece;
};
static_assert(Wt<false>::chunk % 128 == 0 && Wt<true>::chunk % 128 == 0 && Wt<false>::last_down % 16 == 0, "bulk copies");

constexpr int kXWords = kHidden / 8;          // 112 words of eight halves in a row of the residual stream
constexpr int kQkvWords = kQkvN / 8;          // 144: two per tile
constexpr int kActWords = kGuTiles;           // 608: one per gate|up tile
constexpr int kPartWords = kHeads * 17;       // of a (row, split): per head 16 words of four sums and one of {max, sum}
constexpr int kMaxParts = 30;                 // rows x splits

// phase ids of a wait (status word, tags)
constexpr int kPhX = 0, kPhQkv = 1, kPhAtt = 2, kPhXb = 3, kPhAct = 4, kPhCand = 6;
constexpr uint32_t kPollLimit = 1u << 20;
// Layers are numbered through the life of an exchange area (header word 0).  A launch starts below kNumbers and
// counts at most 4096 x 64 on from there, so that within a launch no number overflows (0xFFFFFFFF and 0 would be the
// same copy) and none is zero, the tag of an area that has just been cleared.
constexpr uint32_t kNumbers = 3u << 28;
static_assert(kNumbers % 3u == 0u && (uint64_t)kNumbers + 4096u * kMaxLayers + 2u < (uint64_t(1) << 32), "numbers of a launch");

// Exchange buffers, each three times: the copy of layer number n is n % 3.
struct SyncLayout {
  int64_t x, xb, att, qkv, act, part, cand, total;  // byte offsets
};
constexpr int kXBuf = 16 * kMaxRows * kXWords, kQkvBuf = 16 * kMaxRows * kQkvWords, kActBuf = 16 * kMaxRows * kActWords;
constexpr int kPartBuf = 16 * kMaxParts * kPartWords;
__host__ __device__ constexpr SyncLayout sync_layout() {
  SyncLayout s{};
  int64_t off = 256;
  s.x = off;    off += 3 * kXBuf;
  s.xb = off;   off += 3 * kXBuf;
  s.att = off;  off += 3 * kXBuf;
  s.qkv = off;  off += 3 * kQkvBuf;
  s.act = off;  off += 3 * kActBuf;
  s.part = off; off += 3 * kPartBuf;
  s.cand = off; off += (int64_t)16 * kMaxRows * kCtas;
  s.total = (off + 255) / 256 * 256;
  return s;
}

struct PersistArgs {
  const unsigned char* chunks;  // [n_layers][Wt::per_layer][Wt::chunk]
  const half* ln;               // [n_layers][2][896] norm weights, then the final norm
  const half* bias;             // [n_layers][72][16] QKV bias in tile order
  const half* embed;
  const half* cos_t;
  const half* sin_t;
  int32_t n_layers, vocab, max_pos;
  float eps;
  half* kv;
  int32_t n_slots, s_max;
  int32_t* tok;
  int32_t* pos;
  const int32_t* rows;
  int32_t batch;
  int32_t* out_tokens;
  int32_t ring;
  int32_t* step_counter;
  half* logits;
  unsigned char* sync;  // header + exchange buffers
  int32_t steps;
  int32_t splits;  // attention splits per (row, KV head)
  int32_t chunk_tokens;  // tokens per split, a multiple of 64
  int32_t na;      // attention CTAs = 2 * batch * splits
  int32_t tq, nq;  // QKV tiles per QKV CTA, QKV CTAs
  // host-driven form: tokens to feed (by value), and mapped host memory for the results
  int32_t feed[kMaxRows];
  int32_t* feed_dst;  // where a copy would have put them: entries of `tok`
  int32_t n_feed;
  const int32_t* out_src;
  int32_t* host_out;
  int32_t n_out;
  int32_t* host_status;
  int32_t ng;      // gate|up CTAs = 148 - na
};

// ---- tagged words -----------------------------------------------------------------------
struct Word {
  u64 lo, hi;
};
__device__ __forceinline__ Word ld_word(const void* p) {
  Word w;
  asm volatile(
      "{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
      : "=l"(w.lo), "=l"(w.hi)
      : "l"(p)
      : "memory");
  return w;
}
__device__ __forceinline__ void st_word(void* p, Word w) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p), "l"(w.lo),
      "l"(w.hi)
      : "memory");
}
__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ Word word32(uint32_t a, uint32_t b, uint32_t c, uint32_t tag) {
  Word w;
  w.lo = ((u64)b << 32) | a;
  w.hi = ((u64)tag << 32) | c;
  return w;
}
// Eight halves as a word: stored with the last four bytes inverted, so that the all-zero word, which
// means "not there yet", would be a pair of 0xFFFF halves; no arithmetic result is one (the NaN
// that arithmetic makes is 0x7FFF).
__device__ __forceinline__ Word data_word(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  Word w;
  w.lo = ((u64)b << 32) | a;
  w.hi = ((u64)(~d) << 32) | c;
  return w;
}
__device__ __forceinline__ uint4 word_data(const Word& w) {
  return make_uint4((uint32_t)w.lo, (uint32_t)(w.lo >> 32), (uint32_t)w.hi, ~(uint32_t)(w.hi >> 32));
}

// What a wait needs to know.
struct Ctx {
  uint32_t* status;     // global status word
  uint32_t poll_limit;  // probes before a poll gives up
};

// Polls up to U words (addresses from `addr(u)`) whose bits are set in `pending` until each is there
// (TAG: until it carries `tag`); all loads of a round are in flight together.  On a timeout (code
// recorded in the status word) or when another CTA has reported one, sets `bad` and returns; the
// caller folds `bad` into its next CTA barrier.  `patience` multiplies the limit: waits further down
// the chain give up later, so the wait nearest to a missing word is the one that names it.  `loaded`: a
// first probe of every word is in `val` already.
// (Two probes in flight half a round trip apart, a pause between probes, one lane probing for its warp
// first: all slower, 437, 340 and 344 us per token against 322 when they were tried.)
template <int U, bool TAG, typename AddrFn>
__device__ __forceinline__ void poll_words(const Ctx& c, AddrFn addr, uint32_t pending, uint32_t tag, Word (&val)[U],
                                           int code, uint32_t patience, bool& bad, bool loaded = false) {
  uint32_t tries = 0;
  while (pending != 0u) {
    if (!loaded) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (pending & (1u << u)) val[u] = ld_word(addr(u));
    }
    loaded = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t last = (uint32_t)(val[u].hi >> 32);
      if ((pending & (1u << u)) && (TAG ? last == tag : last != 0u)) pending &= ~(1u << u);
    }
    if (pending != 0u && ((++tries) & 255u) == 0u) {
      const bool expired = tries / patience >= c.poll_limit;
      if (expired) atomicCAS(reinterpret_cast<unsigned*>(c.status), 0u, 0x100u | (uint32_t)(code & 0xFF));
      if (expired || ld_relaxed_u32(c.status) != 0u) {
        bad = true;
        return;
      }
    }
  }
}

// ---- barriers of the compute warps: bar.sync takes whole warps, so a warp whose lanes left a poll one
// by one comes together first ----
__device__ __forceinline__ void cbar() {
  __syncwarp();
  asm volatile("bar.sync 1, %0;" ::"n"(kComp) : "memory");
}
__device__ __forceinline__ bool cbar_or(bool p) {
  uint32_t r;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)p), "n"(kComp)
      : "memory");
  return r != 0u;
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// bulk copy of data that is read once per token: it should not push the small tensors out of L2
__device__ __forceinline__ u64 evict_first_policy() {
  u64 p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void bulk_load_stream(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar, u64 policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ u64 global_ns() {
  u64 t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) { return mbar_try(bar, parity); }
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}

// ---- shared memory ---------------------------------------------------------------------------
constexpr int kXStride = kHidden + 8;    // halves; 113 x 16 bytes: ldmatrix rows fall into different banks
constexpr int kSsqStride = 20;           // floats per row: 14 warps' sums
constexpr int kLmRow = kHidden * 2 + 16;  // bytes of a table row in a lm_head stage (same reason)
constexpr int kLmStage = 16 * kLmRow;
constexpr int kKvHalf = 2 * 32 * kHeadDim * 2;  // 8 KB: 32 tokens of K and of V
constexpr int kSmemMax = 232448;

extern __shared__ __align__(128) unsigned char smem_base[];

constexpr int cmax(int a, int b) { return a > b ? a : b; }
constexpr int cmin(int a, int b) { return a < b ? a : b; }
template <int MR, bool F16>
struct SL {
  static constexpr int nt_max = MR > 8 ? 6 : 7;  // gate|up tiles of a CTA
  static constexpr int u_bytes = kWarps * nt_max * MR * 64;  // partial sums of qkv, o_proj, gate|up
  static constexpr int red2_bytes = kWarps * MR * 64;  // partial sums of down
  static constexpr int xs_bytes = (MR * kXStride * 2 + 127) / 128 * 128;
  static constexpr int rope_bytes = (3 * MR * 64 + 127) / 128 * 128;
  static constexpr int fixed = u_bytes + red2_bytes + xs_bytes + kWarps * 64 /* stage */ +
                               (kGroupHeads * 66 * 4 + 16 + 9 * kHeadDim * 2 + 127) / 128 * 128 /* attention rows */ +
                               kWarps * MR * 8 /* candidates */ + rope_bytes + kMaxRows * kSsqStride * 4 + 256 /* state */ + kWarps * 64 /* residual */ + 512 /* arguments */ + 1024;
  static constexpr int n_ring = cmin((kSmemMax - fixed) / Wt<F16>::chunk, 30);
  static constexpr int ring = 0;
  static constexpr int u = n_ring * Wt<F16>::chunk;
  static constexpr int red2 = u + u_bytes;
  static constexpr int xs = red2 + red2_bytes;
  static constexpr int stage = xs + xs_bytes;
  static constexpr int att_f = (stage + kWarps * 64 + 127) / 128 * 128;                    // [7][66] floats, then the q, k, v rows
  static constexpr int att_h = att_f + (kGroupHeads * 66 * 4 + 15) / 16 * 16;
  static constexpr int cand = (att_h + 9 * kHeadDim * 2 + 127) / 128 * 128;
  static constexpr int rope = (cand + kWarps * MR * 8 + 127) / 128 * 128;
  static constexpr int ssq = rope + rope_bytes;
  static constexpr int state = ssq + kMaxRows * kSsqStride * 4;  // pos[16], slot[16], tok[16], abort, lm parities
  static constexpr int resid = state + 256;  // this CTA's elements of the residual stream
  static constexpr int args = resid + kWarps * 64;
  static constexpr int bars = args + 512;  // full[n_ring], empty[n_ring], lm_full[n_lm], lm_done
  static constexpr int kv_halves = cmin(red2 / kKvHalf, 2 * kWarps);  // half tiles that stay in shared memory
  static constexpr int n_lm = cmin(red2 / kLmStage, 7);
  static constexpr int total = bars + (2 * n_ring + n_lm + 1) * 8;
  static_assert(total <= kSmemMax && u % 128 == 0 && att_h % 16 == 0 && bars % 8 == 0 && xs % 16 == 0, "layout");
  // (a phase waits for three pieces before it gives the first slot back)
  static_assert(n_ring >= cmax(8, 3 * Wt<F16>::per_piece) && n_lm >= 3 && kv_halves > kWarps, "layout");
};
#define SMEM_HALF(...) (reinterpret_cast<half*>(smem_base + (__VA_ARGS__)))
#define SMEM_F32(...) (reinterpret_cast<float*>(smem_base + (__VA_ARGS__)))
#define SMEM_I32(...) (reinterpret_cast<int*>(smem_base + (__VA_ARGS__)))

// Position of (batch row m, tile row r) in a block of partial sums: the exclusive-or spreads the
// four rows a fragment's lanes write over the banks, and keeps the sixteen r of a row in one line.
__device__ __forceinline__ int red_index(int m, int r) { return (m * 16 + r) ^ (((m >> 1) & 3) << 3); }

// Bounded mbarrier wait (two seconds) that also ends when the CTA has given up.
template <int MR, bool F16>
__device__ __forceinline__ bool ring_wait(uint32_t bar, uint32_t parity) {
  const volatile int* abort_flag = SMEM_I32(SL<MR, F16>::state) + 48;
  u64 t0 = 0;
  for (uint32_t i = 1;; ++i) {
    if (mbar_test(bar, parity)) return true;
    if ((i & 63u) == 0u) {
      const u64 t = global_ns();
      if (i == 64u) t0 = t;
      if (*abort_flag != 0 || t - t0 > 2000000000ull) return false;
    }
  }
}

// gate|up tiles of a CTA
__device__ __forceinline__ int gu_count(const PersistArgs& a, int c) {
  const int base = kGuTiles / a.ng, rem = kGuTiles - base * a.ng;
  return base + (c >= a.ng - rem ? 1 : 0);
}
__device__ __forceinline__ int gu_first(const PersistArgs& a, int c) {
  const int base = kGuTiles / a.ng, rem = kGuTiles - base * a.ng;
  return c * base + (c > a.ng - rem ? c - (a.ng - rem) : 0);
}

// Where a compute warp stands in the ring.
struct RingPos {
  uint32_t slot, par;
};
template <int MR, bool F16>
__device__ __forceinline__ void ring_next(RingPos& p) {
  if (++p.slot == (uint32_t)SL<MR, F16>::n_ring) {
    p.slot = 0;
    p.par ^= 1u;
  }
}

// The lane's A fragments of four k steps of a tile.  Unpacking eight nibbles (a row pair's k) is a shift,
// four and-or, four subtractions and four products: with the fp16 exponent of 1024 above the low
// nibble, or that of 64 above the next one, the half is 1024 + q or 64 + q; 1024 + zp or 64 + zp comes
// off exactly, and the product with the scale is rounded once, as in dequant8 (common.cuh).
template <bool F16>
struct Piece {
  uint32_t a[4][4];
};
// The next n pieces of the warp: all waits, then all loads, then with `release` the slots go back.
// `use_last` false: the warp has no share of the last piece.
template <int MR, bool F16, int N>
__device__ __forceinline__ void load_pieces(Piece<F16> (&P)[N], int n, RingPos& p, bool release, bool use_last,
                                            int warp, int lane, bool& bad) {
  using L = SL<MR, F16>;
  constexpr int per = Wt<F16>::per_piece;
  const uint32_t base = smem_u32(smem_base), bars = base + L::bars;
  const RingPos first = p;
  RingPos q = first;
#pragma unroll
  for (int i = 0; i < N * per; ++i) {
    if (i < n * per) {
      if (!ring_wait<MR, F16>(bars + 8 * q.slot, q.par)) bad = true;
      ring_next<MR, F16>(q);
    }
  }
  p = q;
  q = first;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    if (i < n) {
      const bool use = use_last || i < n - 1;
#pragma unroll
      for (int j = 0; j < per; ++j) {
        const uint32_t ch = base + L::ring + q.slot * Wt<F16>::chunk;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        uint2 sc = make_uint2(0u, 0u);
        if (use) {
          v = lds128(ch + (F16 ? 0 : kScaleBytes) + warp * 512 + lane * 16);
          if (!F16) sc = lds64(ch + warp * 64 + (lane >> 2) * 8);
        }
        if (F16) {
          P[i].a[j][0] = v.x;
          P[i].a[j][1] = v.y;
          P[i].a[j][2] = v.z;
          P[i].a[j][3] = v.w;
        } else {
          const half2 s0 = __low2half2(u32_as_half2(sc.x)), s1 = __high2half2(u32_as_half2(sc.x));
          const half2 z0 = __low2half2(u32_as_half2(sc.y)), z1 = __high2half2(u32_as_half2(sc.y));
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t w8 = w[k] >> 8;
            const half2 h[4] = {__hmul2(__hsub2(u32_as_half2((w[k] & 0x000f000fu) | 0x64006400u), z0), s0),
                                __hmul2(__hsub2(u32_as_half2((w[k] & 0x00f000f0u) | 0x54005400u), z1), s1),
                                __hmul2(__hsub2(u32_as_half2((w8 & 0x000f000fu) | 0x64006400u), z0), s0),
                                __hmul2(__hsub2(u32_as_half2((w8 & 0x00f000f0u) | 0x54005400u), z1), s1)};
#pragma unroll
            for (int e = 0; e < 4; ++e) P[i].a[k][e] = *reinterpret_cast<const uint32_t*>(&h[e]);
          }
        }
        ring_next<MR, F16>(q);
      }
    }
  }
  if (release) {
    // the reads come before the copy that refills the slot (another proxy; without the fence fp16
    // fragments, which nothing consumes here, were now and then the next chunk's)
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) {
      q = first;
#pragma unroll
      for (int i = 0; i < N * per; ++i) {
        if (i < n * per) {
          mbar_arrive(bars + 8 * (L::n_ring + q.slot));
          ring_next<MR, F16>(q);
        }
      }
    }
  }
}

// The lane's B fragments of a 64-wide slice of K (eight words from `first` of every row), straight from
// the exchange buffer: lane (g, t) polls words first + 2t and + 2t + 1 of rows g (and g + 8).  The k order inside
// a slice is chosen for this: a lane's sixteen k are contiguous, and the weight fragments are packed in
// the same order.  Lanes of rows beyond `nrows` hold zeros.
template <int NB>
__device__ __forceinline__ void poll_frags(const Ctx& c, const unsigned char* buf, int row_words, int first, int nrows,
                                           int lane, uint32_t (&b)[NB][8], int code, uint32_t patience, bool& bad) {
  const int g = lane >> 2, t = lane & 3;
  uint32_t pending = 0;
#pragma unroll
  for (int nb = 0; nb < NB; ++nb)
    if (g + 8 * nb < nrows) pending |= 3u << (2 * nb);
  Word v[2 * NB] = {};
  poll_words<2 * NB, false>(
      c, [&](int u) { return buf + ((size_t)(g + 8 * (u >> 1)) * row_words + first + 2 * t + (u & 1)) * 16; }, pending, 0u,
      v, code, patience, bad);
  __syncwarp();  // (lanes leave a poll one by one; the mma that follow need the whole warp)
#pragma unroll
  for (int u = 0; u < 2 * NB; ++u) {
    const uint4 d = word_data(v[u]);
    const bool on = g + 8 * (u >> 1) < nrows;
    b[u >> 1][4 * (u & 1) + 0] = on ? d.x : 0u;
    b[u >> 1][4 * (u & 1) + 1] = on ? d.y : 0u;
    b[u >> 1][4 * (u & 1) + 2] = on ? d.z : 0u;
    b[u >> 1][4 * (u & 1) + 3] = on ? d.w : 0u;
  }
}
// The attention output of slice `warp` (a head) as fragments, merged from the splits' partial results.
// With few rows the lanes of unused rows take splits of their own: lane g = row * P + q reads
// splits q, q + P, ..; the P partial merges then meet by shuffles.
__device__ __forceinline__ void poll_merged(const Ctx& c, const unsigned char* buf, int splits, int head, int nrows,
                                            int lane, uint32_t (&b)[8], int code, uint32_t patience, bool& bad) {
  const int g = lane >> 2, t = lane & 3;
  const int log_p = nrows == 1 ? 3 : (nrows == 2 ? 2 : (nrows <= 4 ? 1 : 0));
  const int P = 1 << log_p, row = g >> log_p, q = g & (P - 1);
  float m = -INFINITY, l = 0.f, acc[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) acc[i] = 0.f;
  for (int s0 = 0; s0 < splits; s0 += P) {
    const int s = s0 + q;
    const unsigned char* p = buf + ((size_t)(row * splits + s) * kPartWords + head * 17) * 16;
    const bool on = row < nrows && s < splits;
    Word v[5] = {};
    {  // one small word first: probing all of them for as long as the attention takes slows it down
      Word w[1] = {};
      poll_words<1, false>(
          c, [&](int) { return p + 16 * 16; }, on && t == 0 ? 1u : 0u, 0u, w, code, patience, bad);
      __syncwarp();
    }
    poll_words<5, false>(
        c, [&](int u) { return p + (u < 4 ? 4 * t + u : 16) * 16; }, on ? 31u : 0u, 0u, v, code, patience, bad);
    __syncwarp();
    if (on) {
      const float ms = __uint_as_float((uint32_t)v[4].lo), ls = __uint_as_float((uint32_t)(v[4].lo >> 32));
      const float mn = fmaxf(m, ms), ref = mn == -INFINITY ? 0.f : mn;
      const float e0 = __expf(m - ref), e1 = __expf(ms - ref);
      m = mn;
      l = l * e0 + ls * e1;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint4 d = word_data(v[u]);
        const uint32_t x[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[4 * u + e] = acc[4 * u + e] * e0 + __uint_as_float(x[e]) * e1;
      }
    }
  }
  for (int k = 0; k < log_p; ++k) {
    const int x = 4 << k;
    const float mo = __shfl_xor_sync(0xffffffffu, m, x), lo = __shfl_xor_sync(0xffffffffu, l, x);
    const float mn = fmaxf(m, mo), ref = mn == -INFINITY ? 0.f : mn;
    const float e0 = __expf(m - ref), e1 = __expf(mo - ref);
    m = mn;
    l = l * e0 + lo * e1;
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = acc[i] * e0 + __shfl_xor_sync(0xffffffffu, acc[i], x) * e1;
  }
  const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    b[i] = pack_half2(acc[2 * i] * inv, acc[2 * i + 1] * inv);
    if (log_p > 0) b[i] = __shfl_sync(0xffffffffu, b[i], (((g << log_p) & 7) << 2) | t);  // row g's result to lane g
  }
}
// RMSNorm in place of the fragments of whole rows (the CTA's 14 warps hold a slice each): the slices'
// sums of squares meet in shared memory, one barrier.  `lw`: the norm weights of the lane's k.
template <int MR, bool F16>
__device__ __forceinline__ bool norm_frags(uint32_t (&b)[(MR + 7) / 8][8], const uint4 (&lw)[2], int nrows, float eps,
                                           int warp, int lane, bool bad) {
  using L = SL<MR, F16>;
  constexpr int NB = (MR + 7) / 8;
  const int g = lane >> 2, t = lane & 3;
  float* ssq = SMEM_F32(L::ssq);
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    float s[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 x = __half22float2(u32_as_half2(b[nb][i]));
      s[0] = fmaf(x.x, x.x, s[0]);
      s[1] = fmaf(x.y, x.y, s[1]);
    }
    float q = s[0] + s[1];
    q += __shfl_xor_sync(0xffffffffu, q, 1);
    q += __shfl_xor_sync(0xffffffffu, q, 2);
    if (t == 0 && g + 8 * nb < nrows) ssq[(g + 8 * nb) * kSsqStride + warp] = q;
  }
  if (cbar_or(bad)) return false;
  const uint32_t w[8] = {lw[0].x, lw[0].y, lw[0].z, lw[0].w, lw[1].x, lw[1].y, lw[1].z, lw[1].w};
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    const int row = g + 8 * nb < nrows ? g + 8 * nb : 0;
    const float4* p = reinterpret_cast<const float4*>(ssq + row * kSsqStride);
    const float4 p0 = p[0], p1 = p[1], p2 = p[2];
    const float2 p3 = *reinterpret_cast<const float2*>(p + 3);
    const float sum = ((p0.x + p0.y) + (p0.z + p0.w)) + ((p1.x + p1.y) + (p1.z + p1.w)) +
                      ((p2.x + p2.y) + (p2.z + p2.w)) + (p3.x + p3.y);
    const float r = rsqrtf(sum * (1.0f / kHidden) + eps);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 x = __half22float2(u32_as_half2(b[nb][i])), l = __half22float2(u32_as_half2(w[i]));
      b[nb][i] = pack_half2(x.x * r * l.x, x.y * r * l.y);
    }
  }
  return true;
}
// The norm weights (or an embedding row's values) of the lane's k in slice `warp` of a row of 896.
__device__ __forceinline__ void load_slice(uint4 (&v)[2], const half* row, int warp, int lane) {
  const half* p = row + 64 * warp + 16 * (lane & 3);
  v[0] = ldg_nc_u128(p);
  v[1] = ldg_nc_u128(p + 8);
}

// d += tile piece x activations; N pieces with the k steps outermost, so that
// consecutive mma belong to different accumulators.
template <bool F16, int N>
__device__ __forceinline__ void pieces_mma(float (&d)[N][4], const Piece<F16>* P, const uint32_t (&b)[8]) {
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int i = 0; i < N; ++i)
      mma16816(d[i], P[i].a[j][0], P[i].a[j][1], P[i].a[j][2], P[i].a[j][3], b[2 * j], b[2 * j + 1]);
}
// One accumulator block (tile rows x 8 batch rows from row0) to the warp's partial sums.
template <int MR>
__device__ __forceinline__ void store_partial(float* red, const float (&d)[4], int row0, int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int m = row0 + 2 * t + e;
    if (m < MR) {
      red[red_index(m, g)] = d[e];
      red[red_index(m, g + 8)] = d[2 + e];
    }
  }
}
template <int MR>
__device__ __forceinline__ float sum_partials(const float* red, int warp_stride, int m, int r) {
  float v[kWarps];
#pragma unroll
  for (int w = 0; w < kWarps; ++w) v[w] = red[w * warp_stride + red_index(m, r)];
  float s = 0.f;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) s += v[w];
  return s;
}

// Final norm into the activation block of the lm_head: thread t polls word t % 112 of rows t / 112 + 4 i.
template <int MR, bool F16>
__device__ __forceinline__ bool norm_rows(const Ctx& c, const unsigned char* buf, const half* ln, int nrows, float eps,
                                          int tid, int code, uint32_t patience) {
  using L = SL<MR, F16>;
  constexpr int R = (MR + 3) / 4;
  const int r0 = tid / kXWords, w = tid - r0 * kXWords;
  float* ssq = SMEM_F32(L::ssq);
  bool bad = false;
  const uint4 lw = ldg_nc_u128(ln + 8 * w);
  uint32_t pending = 0;
#pragma unroll
  for (int i = 0; i < R; ++i)
    if (r0 + 4 * i < nrows) pending |= 1u << i;
  Word v[R] = {};
  poll_words<R, false>(
      c, [&](int i) { return buf + ((size_t)(r0 + 4 * i) * kXWords + w) * 16; }, pending, 0u, v, code, patience, bad);
  __syncwarp();
  auto floats = [](const uint4& d, float (&f)[8]) {
    const uint32_t u[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 x = __half22float2(u32_as_half2(u[e]));
      f[2 * e] = x.x;
      f[2 * e + 1] = x.y;
    }
  };
#pragma unroll
  for (int i = 0; i < R; ++i) {  // (a row is seven half warps)
    float f[8], s = 0.f;
    floats(word_data(v[i]), f);
#pragma unroll
    for (int e = 0; e < 8; ++e) s = fmaf(f[e], f[e], s);
#pragma unroll
    for (int x = 1; x < 16; x <<= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
    if ((tid & 15) == 0 && r0 + 4 * i < nrows) ssq[(r0 + 4 * i) * kSsqStride + (w >> 4)] = s;
  }
  if (cbar_or(bad)) return false;
  float l[8];
  floats(lw, l);
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = r0 + 4 * i;
    if (r < nrows) {
      float sum = 0.f, f[8];
#pragma unroll
      for (int k = 0; k < 7; ++k) sum += ssq[r * kSsqStride + k];
      const float rs = rsqrtf(sum * (1.0f / kHidden) + eps);
      floats(word_data(v[i]), f);
      uint4 o;
      o.x = pack_half2(f[0] * rs * l[0], f[1] * rs * l[1]);
      o.y = pack_half2(f[2] * rs * l[2], f[3] * rs * l[3]);
      o.z = pack_half2(f[4] * rs * l[4], f[5] * rs * l[5]);
      o.w = pack_half2(f[6] * rs * l[6], f[7] * rs * l[7]);
      *reinterpret_cast<uint4*>(SMEM_HALF(L::xs) + r * kXStride + 8 * w) = o;
    }
  }
  cbar();
  return true;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The attention works in 32-token half tiles, so that all 14 warps have one from 417 tokens on: half
// tile i of the CTA's range belongs to warp i % 14.  In shared memory a half tile is 32 rows of K and 32
// of V, 128-byte swizzle.
constexpr int kHalf = 32;
constexpr int kHalfBytes = 2 * kHalf * kHeadDim * 2;  // 8 KB
// Requests a half tile; rows from `end` on are zero.
__device__ __forceinline__ void kv_half_request(uint32_t dst, const half* kbase, const half* vbase, int t0, int end,
                                                int lane) {
#pragma unroll 4
  for (int i = 0; i < 8; ++i) {
    const int idx = lane + 32 * i, r = idx >> 3, c = idx & 7;
    const bool ok = t0 + r < end;
    const size_t off = ok ? (size_t)(t0 + r) * kHeadDim + 8 * c : 0;
    cp_async16(dst + sw128_offset(r, c), kbase + off, ok);
    cp_async16(dst + kHalfBytes / 2 + sw128_offset(r, c), vbase + off, ok);
  }
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
  uint32_t d;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}
__device__ __forceinline__ void ldsm4_trans(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}
// Both products with the tokens or the head dims on the M side of the mma and the heads on N: scores^T =
// K Q^T (A = K rows by ldmatrix), out^T = V^T P^T (A = V by transposing ldmatrix).  Seven heads fill
// seven of eight columns, where on the M side they would fill seven of sixteen rows: half the mma.
// The fragments of a warp's first half tile are in registers before q arrives.
struct KvFrags {
  uint32_t k[2][4][4];  // [16 tokens][16 dims]
  uint32_t v[4][2][4];  // [16 dims][16 tokens]
};
__device__ __forceinline__ void load_half(KvFrags& f, uint32_t tile_s, int lane) {
  const int mi = lane >> 3, mr = lane & 7;
#pragma unroll
  for (int ks = 0; ks < 4; ++ks)
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
      ldsm4(f.k[mt][ks], tile_s + sw128_offset(16 * mt + 8 * (mi & 1) + mr, 2 * ks + (mi >> 1)));
#pragma unroll
  for (int ks = 0; ks < 2; ++ks)
#pragma unroll
    for (int dt = 0; dt < 4; ++dt)
      ldsm4_trans(f.v[dt][ks], tile_s + kHalfBytes / 2 + sw128_offset(16 * ks + 8 * (mi >> 1) + mr, 2 * dt + (mi & 1)));
}
// Running softmax over the warp's half tiles: a lane's two heads are columns 2t, 2t + 1 throughout; l
// stays a per-lane partial sum (tokens g, g + 8, ..) until the end.  A score fragment becomes a P^T
// fragment by an 8 x 8 register transpose.
__device__ __forceinline__ void attend_half(const KvFrags& f, const uint32_t (&qb)[4][2], int t0, int end, float scale,
                                            int lane, float (&m)[2], float (&l)[2], float (&o)[4][4]) {
  const int g = lane >> 2;
  float sc[2][4] = {};
#pragma unroll
  for (int ks = 0; ks < 4; ++ks)
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
      mma16816(sc[mt], f.k[mt][ks][0], f.k[mt][ks][1], f.k[mt][ks][2], f.k[mt][ks][3], qb[ks][0], qb[ks][1]);
  float mx[2] = {m[0], m[1]};
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float s = t0 + 16 * mt + g + 8 * (e >> 1) < end ? sc[mt][e] * scale : -INFINITY;
      sc[mt][e] = s;
      mx[e & 1] = fmaxf(mx[e & 1], s);
    }
#pragma unroll
  for (int x = 4; x < 32; x <<= 1) {
    mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], x));
    mx[1] = fmaxf(mx[1], __shfl_xor_sync(0xffffffffu, mx[1], x));
  }
  float keep[2], ref[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    ref[e] = mx[e] == -INFINITY ? 0.f : mx[e];
    keep[e] = __expf(m[e] - ref[e]);  // (0 before the first token)
    m[e] = mx[e];
    l[e] *= keep[e];
  }
  uint32_t pb[2][2];
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const half2 ph = __floats2half2_rn(__expf(sc[mt][2 * hh] - ref[0]), __expf(sc[mt][2 * hh + 1] - ref[1]));
      l[0] += __low2float(ph);
      l[1] += __high2float(ph);
      pb[mt][hh] = movmatrix_trans(*reinterpret_cast<const uint32_t*>(&ph));
    }
#pragma unroll
  for (int dt = 0; dt < 4; ++dt)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[dt][e] *= keep[e & 1];
#pragma unroll
  for (int ks = 0; ks < 2; ++ks)
#pragma unroll
    for (int dt = 0; dt < 4; ++dt)
      mma16816(o[dt], f.v[dt][ks][0], f.v[dt][ks][1], f.v[dt][ks][2], f.v[dt][ks][3], pb[ks][0], pb[ks][1]);
}

// ---- phases -----------------------------------------------------------------------------------
// A phase alone fits the 128 registers a thread can have; what lives across phases (arguments, loop
// state, the attention role) therefore stays in shared memory, and thread and CTA indexes pass through
// an opaque move in every phase, so that nothing is kept in registers through the layer loop.
struct AttnRole {
  int row, kvh, split;
  int slot, pos;     // pos: the token of this step
  int t_lo, t_end;   // cached tokens of this split, the step's own included
};
struct SmArgs {
  PersistArgs a;
  AttnRole role;
  uint32_t poll_limit;
  int32_t withhold_layer;  // test hook: the o_proj result of this layer is not published
  uint32_t no0;            // layer number before the launch's first
  int32_t step0;
  int32_t q0, qn;          // QKV tiles of this CTA
  uint32_t row_magic;      // ceil(65536 / batch): u / batch = u * row_magic >> 16 for the small u of a phase
};
static_assert(sizeof(SmArgs) <= 512, "argument region");
struct Th {
  int tid, warp, lane;  // of the compute threads
  int cta, nrows;       // nrows = batch rows of the launch
  Ctx c;
};
template <int MR, bool F16>
__device__ __forceinline__ const SmArgs& sm_args() {
  return *reinterpret_cast<const SmArgs*>(smem_base + SL<MR, F16>::args);
}
template <int MR>
__device__ __forceinline__ Th make_th(const SmArgs& sa) {
  Th th;
  int tid = threadIdx.x, cta = blockIdx.x;
  asm volatile("" : "+r"(tid), "+r"(cta));
  th.tid = tid;
  th.warp = tid >> 5;
  th.lane = tid & 31;
  th.cta = cta;
  th.nrows = MR == 1 ? 1 : sa.a.batch;
  th.c.status = reinterpret_cast<uint32_t*>(sa.a.sync) + 1;
  th.c.poll_limit = sa.poll_limit;
  return th;
}
// Ring position and "still alive" in one returned word.
constexpr uint32_t kAlive = 0x10000u;
__device__ __forceinline__ RingPos unpack_pos(uint32_t v) { return {v & 0xFFu, (v >> 8) & 1u}; }
__device__ __forceinline__ uint32_t pack_pos(const RingPos& p) { return p.slot | (p.par << 8) | kAlive; }

// Words of layer number `no` that this CTA will publish are emptied one layer ahead, while the CTA
// waits for something else: whoever read their last contents (layer no - 3) has been heard from, and the
// fence puts the stores into L2 long before anybody polls them again.
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void empty_word(unsigned char* p) { st_word(p, Word{0ull, 0ull}); }
__device__ __forceinline__ unsigned char* copy_of(const PersistArgs& a, int64_t off, int64_t bytes, uint32_t no) {
  return a.sync + off + (int64_t)(no % 3u) * bytes;
}
__device__ __forceinline__ void empty_residual(const PersistArgs& a, const Th& th, uint32_t no) {
  constexpr SyncLayout sl = sync_layout();
  if (th.tid < 2 * th.nrows) {
    const size_t at = ((size_t)(th.tid >> 1) * kXWords + 2 * th.cta + (th.tid & 1)) * 16;
    empty_word(copy_of(a, sl.x, kXBuf, no) + at);
    empty_word(copy_of(a, sl.xb, kXBuf, no) + at);
  }
}
__device__ __forceinline__ void empty_qkv(const PersistArgs& a, const Th& th, int q0, int nt, uint32_t no) {
  constexpr SyncLayout sl = sync_layout();
  const int m = th.tid / (2 * nt), w = th.tid - m * 2 * nt;
  if (m < th.nrows) empty_word(copy_of(a, sl.qkv, kQkvBuf, no) + ((size_t)m * kQkvWords + 2 * q0 + w) * 16);
}
__device__ __forceinline__ void empty_act(const PersistArgs& a, const Th& th, int g0, int nt, uint32_t no) {
  constexpr SyncLayout sl = sync_layout();
  const int m = th.tid / nt, w = th.tid - m * nt;
  if (m < th.nrows) empty_word(copy_of(a, sl.act, kActBuf, no) + ((size_t)m * kActWords + g0 + w) * 16);
}
__device__ __forceinline__ void empty_att(const PersistArgs& a, const Th& th, int row, int kvh, int split, uint32_t no) {
  constexpr SyncLayout sl = sync_layout();
  if (a.splits > 1) {
    if (th.tid < kPartWords / 2)
      empty_word(copy_of(a, sl.part, kPartBuf, no) +
                 ((size_t)(row * a.splits + split) * kPartWords + kPartWords / 2 * kvh + th.tid) * 16);
  } else if (th.tid < kXWords / 2) empty_word(copy_of(a, sl.att, kXBuf, no) + ((size_t)row * kXWords + 56 * kvh + th.tid) * 16);
}

// QKV tiles [q0, q0 + nt) of this CTA: norm (residual stream of the layer) -> GEMV -> bias -> RoPE ->
// words for the attention CTAs.
template <int MR, bool F16>
__device__ __forceinline__ uint32_t phase_qkv(uint32_t pos, int layer, uint32_t layer_no) {
  using L = SL<MR, F16>;
  constexpr int NB = (MR + 7) / 8;
  const SmArgs& sa = sm_args<MR, F16>();
  const PersistArgs& a = sa.a;
  const Th th = make_th<MR>(sa);
  RingPos rp = unpack_pos(pos);
  const int q0 = sa.q0, nt = sa.qn;
  const int warp = th.warp, lane = th.lane;
  constexpr SyncLayout sl = sync_layout();
  bool bad = false;
  Piece<F16> A[3] = {};
  load_pieces<MR, F16>(A, nt, rp, true, true, warp, lane, bad);
  empty_qkv(a, th, q0, nt, layer_no + 1);
  uint4 lw[2];
  load_slice(lw, a.ln + (size_t)2 * layer * kHidden, warp, lane);
  // what the warp will finish: units (tile, row), two at a time; the first pair's bias ahead of the wait
  const int r16 = lane & 15, units = nt * th.nrows;
  auto bias_of = [&](int u) {
    const int i = u < units ? (int)(((uint32_t)u * sa.row_magic) >> 16) : 0;
    return a.bias[((size_t)layer * kQkvTiles + q0 + i) * 16 + r16];
  };
  half bias = bias_of(2 * warp + (lane >> 4));
  fence_gpu();
  uint32_t b[NB][8];
  if (layer == 0) {  // the tokens' embedding rows
    const int* s_tok = SMEM_I32(L::state) + 32;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const int row = (lane >> 2) + 8 * nb;
      uint4 e[2] = {};
      if (row < th.nrows) load_slice(e, a.embed + (size_t)s_tok[row] * kHidden, warp, lane);
      b[nb][0] = e[0].x; b[nb][1] = e[0].y; b[nb][2] = e[0].z; b[nb][3] = e[0].w;
      b[nb][4] = e[1].x; b[nb][5] = e[1].y; b[nb][6] = e[1].z; b[nb][7] = e[1].w;
    }
  } else {
    poll_frags<NB>(th.c, copy_of(a, sl.x, kXBuf, layer_no - 1), kXWords, 8 * warp, th.nrows, lane, b,
                   layer * 8 + kPhX, 4u, bad);
  }
  if (!norm_frags<MR, F16>(b, lw, th.nrows, a.eps, warp, lane, bad)) return 0u;
  float* red = SMEM_F32(L::u);
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      if (i < nt) {
        float d[1][4] = {};
        pieces_mma<F16>(d, A + i, b[nb]);
        store_partial<MR>(red + (warp * 3 + i) * MR * 16, d[0], 8 * nb, lane);
      }
    }
  }
  cbar();
  half* st = SMEM_HALF(L::stage) + warp * 32;
  const float2* rope = reinterpret_cast<const float2*>(smem_base + L::rope);
  unsigned char* words = copy_of(a, sl.qkv, kQkvBuf, layer_no);
  for (int u0 = 2 * warp; u0 < units; u0 += 2 * kWarps) {
    const int u = u0 + (lane >> 4);
    const bool on = u < units;
    const int i = on ? (int)(((uint32_t)u * sa.row_magic) >> 16) : 0, m = on ? u - i * th.nrows : 0;
    const int tile = q0 + i;
    float x = sum_partials<MR>(red + i * MR * 16, 3 * MR * 16, m, r16);
    x = __half2float(__float2half_rn(x + __half2float(bias)));
    const float other = __shfl_xor_sync(0xffffffffu, x, 8);
    float out = x;
    if (tile < 4 * (kHeads + kKvHeads)) {  // q and k rotate, v does not
      const float2 cs = rope[(i * MR + m) * 8 + (r16 & 7)];
      out = r16 < 8 ? x * cs.x - other * cs.y : other * cs.y + x * cs.x;
    }
    if (u0 + 2 * kWarps < units) bias = bias_of(u + 2 * kWarps);
    st[lane] = __float2half_rn(out);
    __syncwarp();
    if (on && r16 < 2) {
      const uint4 d = *reinterpret_cast<const uint4*>(st + (lane & 16) + 8 * r16);
      st_word(words + ((size_t)m * kQkvWords + 2 * tile + r16) * 16, data_word(d.x, d.y, d.z, d.w));
    }
    __syncwarp();
  }
  return pack_pos(rp);
}

// Residual columns of this CTA: the pair of rows (two half warps) a warp finishes after o_proj or
// down; the thread's element of the residual stream stays in its place in shared memory.
template <int MR, bool F16>
__device__ __forceinline__ void finish_residual(const Th& th, const float* red, unsigned char* words, bool withhold) {
  using L = SL<MR, F16>;
  const int warp = th.warp, lane = th.lane, r = lane & 15, m = 2 * warp + (lane >> 4);
  if (2 * warp >= th.nrows) return;
  const int mm = m < th.nrows ? m : th.nrows - 1;
  const float s = sum_partials<MR>(red, MR * 16, mm, r);
  half* st = SMEM_HALF(L::resid) + warp * 32;
  st[lane] = __float2half_rn(__half2float(st[lane]) + __half2float(__float2half_rn(s)));
  __syncwarp();
  if (m < th.nrows && r < 2 && !withhold) {
    const uint4 d = *reinterpret_cast<const uint4*>(st + (lane & 16) + 8 * r);
    st_word(words + ((size_t)m * kXWords + 2 * th.cta + r) * 16, data_word(d.x, d.y, d.z, d.w));
  }
  __syncwarp();
}

// o_proj (residual CTAs) and gate|up.  The weights of both are in registers before the attention
// output arrives: what lies between two exchanges is only the arithmetic.
template <int MR, bool F16>
__device__ __forceinline__ uint32_t phase_mid(uint32_t pos, int layer, uint32_t layer_no) {
  using L = SL<MR, F16>;
  // three tiles are held in registers ahead of the wait, the CTA's other tiles follow from the ring
  constexpr int NB = (MR + 7) / 8, NT = L::nt_max, kPre = 3;  // (every CTA has at least four tiles)
  const SmArgs& sa = sm_args<MR, F16>();
  const PersistArgs& a = sa.a;
  const Th th = make_th<MR>(sa);
  RingPos rp = unpack_pos(pos);
  const int warp = th.warp, lane = th.lane;
  constexpr SyncLayout sl = sync_layout();
  const int nt = gu_count(a, th.cta), g0 = gu_first(a, th.cta);
  const bool res = th.cta < kResCtas;
  bool bad = false;
  float* red = SMEM_F32(L::u);
  Piece<F16> O[1] = {};
  Piece<F16> A[kPre] = {};
  if (res) load_pieces<MR, F16>(O, 1, rp, true, true, warp, lane, bad);
  load_pieces<MR, F16>(A, kPre, rp, true, true, warp, lane, bad);
  empty_act(a, th, g0, nt, layer_no + 1);
  if (res) empty_residual(a, th, layer_no + 1);
  fence_gpu();
  uint32_t b[NB][8];
  if (res) {
    if (MR <= 8 && a.splits > 1)
      poll_merged(th.c, copy_of(a, sl.part, kPartBuf, layer_no), a.splits, warp, th.nrows, lane, b[0], layer * 8 + kPhAtt,
                  2u, bad);
    else
      poll_frags<NB>(th.c, copy_of(a, sl.att, kXBuf, layer_no), kXWords, 8 * warp, th.nrows, lane, b,
                     layer * 8 + kPhAtt, 2u, bad);
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      float d[1][4] = {};
      pieces_mma<F16>(d, O, b[nb]);
      store_partial<MR>(red + warp * MR * 16, d[0], 8 * nb, lane);
    }
    if (cbar_or(bad)) return 0u;
    finish_residual<MR, F16>(th, red, copy_of(a, sl.xb, kXBuf, layer_no), th.cta == 0 && layer == sa.withhold_layer);
  }
  uint4 lw[2];
  load_slice(lw, a.ln + (size_t)(2 * layer + 1) * kHidden, warp, lane);
  poll_frags<NB>(th.c, copy_of(a, sl.xb, kXBuf, layer_no), kXWords, 8 * warp, th.nrows, lane, b, layer * 8 + kPhXb, 1u,
                 bad);
  if (!norm_frags<MR, F16>(b, lw, th.nrows, a.eps, warp, lane, bad)) return 0u;
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    float d[kPre][4] = {};
    pieces_mma<F16>(d, A, b[nb]);
#pragma unroll
    for (int i = 0; i < kPre; ++i) {
      store_partial<MR>(red + (warp * NT + i) * MR * 16, d[i], 8 * nb, lane);
    }
  }
#pragma unroll 1
  for (int i = kPre; i < nt; ++i) {
    Piece<F16> T[1] = {};
    load_pieces<MR, F16>(T, 1, rp, true, true, warp, lane, bad);
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      float d[1][4] = {};
      pieces_mma<F16>(d, T, b[nb]);
      store_partial<MR>(red + (warp * NT + i) * MR * 16, d[0], 8 * nb, lane);
    }
  }
  if (cbar_or(bad)) return 0u;
  // gate rows 0..7 and up rows 8..15 of a tile meet in neighbouring half-groups of lanes; the eight
  // activations of a (tile, row) are one word
  unsigned char* words = copy_of(a, sl.act, kActBuf, layer_no);
  const int units = nt * th.nrows, r16 = lane & 15;
  for (int u0 = 2 * warp; u0 < units; u0 += 2 * kWarps) {
    const int u = u0 + (lane >> 4) < units ? u0 + (lane >> 4) : units - 1;
    const int i = (int)(((uint32_t)u * sa.row_magic) >> 16), m = u - i * th.nrows;
    const float x = __half2float(__float2half_rn(sum_partials<MR>(red + i * MR * 16, NT * MR * 16, m, r16)));
    const float up = __shfl_xor_sync(0xffffffffu, x, 8);
    const uint32_t y = __half_as_ushort(__float2half_rn(silu_mul(x, up)));
    const uint32_t pair = y | (__shfl_down_sync(0xffffffffu, y, 1) << 16);
    const uint32_t p1 = __shfl_down_sync(0xffffffffu, pair, 2), p2 = __shfl_down_sync(0xffffffffu, pair, 4),
                   p3 = __shfl_down_sync(0xffffffffu, pair, 6);
    if (r16 == 0 && u0 + (lane >> 4) < units)
      st_word(words + ((size_t)m * kActWords + g0 + i) * 16, data_word(pair, p1, p2, p3));
  }
  return pack_pos(rp);
}

// down: 16 columns over all 4864 activations.
template <int MR, bool F16>
__device__ __forceinline__ uint32_t phase_down(uint32_t pos, int layer, uint32_t layer_no) {
  using L = SL<MR, F16>;
  constexpr int NB = (MR + 7) / 8, kPre = 2;
  const SmArgs& sa = sm_args<MR, F16>();
  const PersistArgs& a = sa.a;
  const Th th = make_th<MR>(sa);
  RingPos rp = unpack_pos(pos);
  const int warp = th.warp, lane = th.lane, g = lane >> 2, t = lane & 3;
  constexpr SyncLayout sl = sync_layout();
  bool bad = false;
  const bool last_mine = warp < kDownLastWarps;
  Piece<F16> A[kPre] = {};
  load_pieces<MR, F16>(A, kPre, rp, true, true, warp, lane, bad);
  float* red = SMEM_F32(L::red2);
  const unsigned char* buf = copy_of(a, sl.act, kActBuf, layer_no);
  // the lane's words of piece p (slices of 64 k, 896 apart), as in poll_frags
  auto addr = [&](int nb, int p, int u) {
    return buf + ((size_t)(g + 8 * nb) * kActWords + kXWords * p + 8 * warp + 2 * t + u) * 16;
  };
  auto use = [&](float (&sum)[4], const Piece<F16>& P, const Word& w0, const Word& w1) {
    const uint4 d0 = word_data(w0), d1 = word_data(w1);
    const uint32_t b[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
    float d[1][4] = {};
    pieces_mma<F16>(d, &P, b);
#pragma unroll
    for (int e = 0; e < 4; ++e) sum[e] += d[0][e];
  };
  float sum[NB][4] = {};
  if constexpr (NB == 1) {  // all words of the lane in flight together
    uint32_t pending = 0;
    if (g < th.nrows) pending = last_mine ? 0xFFFu : 0x3FFu;
    Word v[2 * kDownPieces] = {};
    poll_words<2 * kDownPieces, false>(
        th.c, [&](int u) { return addr(0, u >> 1, u & 1); }, pending, 0u, v, layer * 8 + kPhAct, 2u, bad);
    __syncwarp();
#pragma unroll
    for (int p = 0; p < kDownPieces; ++p) {
      const bool mine = p < kDownPieces - 1 || last_mine;
      Piece<F16> T[1] = {};
      if (p >= kPre) load_pieces<MR, F16>(T, 1, rp, true, mine, warp, lane, bad);
      if (mine) use(sum[0], p < kPre ? A[p < kPre ? p : 0] : T[0], v[2 * p], v[2 * p + 1]);
    }
  } else {  // two row blocks: piece by piece, the next piece's words requested ahead
    Word v[2][2 * NB] = {};
    auto request = [&](int p, Word (&w)[2 * NB]) {
#pragma unroll
      for (int u = 0; u < 2 * NB; ++u)
        if (g + 8 * (u >> 1) < th.nrows && (p < kDownPieces - 1 || last_mine)) w[u] = ld_word(addr(u >> 1, p, u & 1));
    };
    request(0, v[0]);
#pragma unroll
    for (int p = 0; p < kDownPieces; ++p) {
      const bool mine = p < kDownPieces - 1 || last_mine;
      if (p + 1 < kDownPieces) request(p + 1, v[(p + 1) & 1]);
      Piece<F16> T[1] = {};
      if (p >= kPre) load_pieces<MR, F16>(T, 1, rp, true, mine, warp, lane, bad);
      uint32_t pending = 0;
#pragma unroll
      for (int u = 0; u < 2 * NB; ++u)
        if (mine && g + 8 * (u >> 1) < th.nrows) pending |= 1u << u;
      poll_words<2 * NB, false>(
          th.c, [&](int u) { return addr(u >> 1, p, u & 1); }, pending, 0u, v[p & 1], layer * 8 + kPhAct, 2u, bad, true);
      __syncwarp();
      if (mine) {
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
          use(sum[nb], p < kPre ? A[p < kPre ? p : 0] : T[0], v[p & 1][2 * nb], v[p & 1][2 * nb + 1]);
      }
    }
  }
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) store_partial<MR>(red + warp * MR * 16, sum[nb], 8 * nb, lane);
  if (cbar_or(bad)) return 0u;
  finish_residual<MR, F16>(th, red, copy_of(a, sl.x, kXBuf, layer_no), false);
  return pack_pos(rp);
}

// Attention CTA: one (batch row, KV head, split of the context).
__device__ __forceinline__ const half* kv_plane(const PersistArgs& a, const AttnRole& r, int layer, int which) {
  return a.kv + ((((size_t)2 * layer + which) * a.n_slots + r.slot) * kKvHeads + r.kvh) * a.s_max * kHeadDim;
}
// The half tiles of a layer that fit shared memory: warp w's are w and w + 14.
template <int MR, bool F16>
__device__ __forceinline__ void attn_request(const PersistArgs& a, const Th& th, const AttnRole& r, int layer) {
  using L = SL<MR, F16>;
  for (int i = th.warp; i < L::kv_halves; i += kWarps) {
    const int t0 = r.t_lo + kHalf * i;
    if (t0 < r.t_end)
      kv_half_request(smem_u32(smem_base) + i * kHalfBytes, kv_plane(a, r, layer, 0), kv_plane(a, r, layer, 1), t0, r.pos,
                      th.lane);
  }
}

template <int MR, bool F16>
__device__ __forceinline__ bool phase_attention(int layer, uint32_t layer_no) {
  using L = SL<MR, F16>;
  const SmArgs& sa = sm_args<MR, F16>();
  const PersistArgs& a = sa.a;
  const Th th = make_th<MR>(sa);
  const AttnRole& r = sa.role;
  const int tid = th.tid, warp = th.warp, lane = th.lane, g = lane >> 2, t = lane & 3;
  const SyncLayout sl = sync_layout();
  bool bad = false;
  half* qkv_s = SMEM_HALF(L::att_h);  // rows 0..6 q, 7 k, 8 v
  float* att_f = SMEM_F32(L::att_f);
  empty_att(a, th, r.row, r.kvh, r.split, layer_no + 1);
  fence_gpu();
  const bool owner = r.pos >= r.t_lo && r.pos < r.t_end;  // this split holds the step's own token
  const int n_half = (r.t_end - r.t_lo + kHalf - 1) / kHalf;
  const uint32_t first_s = smem_u32(smem_base) + warp * kHalfBytes;
  cp_async_wait_all();
  __syncwarp();
  KvFrags f = {};
  const int own_half = owner ? (r.pos - r.t_lo) / kHalf : -1;
  const bool early = warp < n_half && warp != own_half;
  if (early) load_half(f, first_s, lane);
  if (tid < 72) {
    const int hs = tid >> 3, quarter = (tid >> 1) & 3, w = tid & 1;
    const int head = hs < kGroupHeads ? r.kvh * kGroupHeads + hs : (hs == kGroupHeads ? kHeads + r.kvh : kHeads + kKvHeads + r.kvh);
    Word v[1] = {};
    poll_words<1, false>(
        th.c,
        [&](int) {
          return copy_of(a, sl.qkv, kQkvBuf, layer_no) + ((size_t)r.row * kQkvWords + 2 * (4 * head + quarter) + w) * 16;
        },
        1u, 0u, v, layer * 8 + kPhQkv, 4u, bad);
    *reinterpret_cast<uint4*>(qkv_s + hs * kHeadDim + 8 * quarter + 32 * w) = word_data(v[0]);
  }
  if (cbar_or(bad)) return false;
  uint32_t qb[4][2];  // Q^T fragments: column g = head (column 7 is zero)
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(qkv_s + g * kHeadDim + 16 * ks + 2 * t);
    qb[ks][0] = g < kGroupHeads ? q[0] : 0u;
    qb[ks][1] = g < kGroupHeads ? q[4] : 0u;
  }
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  for (int i = warp; i < n_half; i += kWarps) {
    const int t0 = r.t_lo + kHalf * i;
    uint32_t tile_s = smem_u32(smem_base) + i * kHalfBytes;
    if (i >= L::kv_halves) {  // a context longer than what fits: fetched while the CTA waits for it
      tile_s = first_s;
      __syncwarp();
      kv_half_request(tile_s, kv_plane(a, r, layer, 0), kv_plane(a, r, layer, 1), t0, r.pos, lane);
      cp_async_wait_all();
      __syncwarp();
    }
    if (i == own_half) {
      if (lane < 16) {  // the step's k and v take their row of the tile, and of the cache for later steps
        const int ch = lane & 7;
        const uint4 val = *reinterpret_cast<const uint4*>(qkv_s + (lane < 8 ? kGroupHeads : kGroupHeads + 1) * kHeadDim + 8 * ch);
        const uint32_t dst = tile_s + (lane < 8 ? 0u : (uint32_t)kHalfBytes / 2) + sw128_offset(r.pos - t0, ch);
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(val.x), "r"(val.y), "r"(val.z), "r"(val.w)
                     : "memory");
        half* row = const_cast<half*>(kv_plane(a, r, layer, lane < 8 ? 0 : 1)) + (size_t)r.pos * kHeadDim;
        *reinterpret_cast<uint4*>(row + 8 * ch) = val;
      }
      __syncwarp();
    }
    if (i != warp || !early) load_half(f, tile_s, lane);
    attend_half(f, qb, t0, r.t_end, 0.125f, lane, m, l, o);
  }
  // ---- the warps' results meet: each over its own first half tile, [7][66] floats ----
  const int n_act = n_half < kWarps ? n_half : kWarps;
  float* part = reinterpret_cast<float*>(smem_base + warp * kHalfBytes);
  __syncwarp();
  if (warp < n_act) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
#pragma unroll
      for (int x = 4; x < 32; x <<= 1) l[e] += __shfl_xor_sync(0xffffffffu, l[e], x);
      const int hd = 2 * t + e;
      if (hd < kGroupHeads) {
#pragma unroll
        for (int dt = 0; dt < 4; ++dt) {
          part[hd * 66 + 16 * dt + g] = o[dt][e];
          part[hd * 66 + 16 * dt + 8 + g] = o[dt][2 + e];
        }
        if (g == 0) {
          part[hd * 66 + 64] = m[e];
          part[hd * 66 + 65] = l[e];
        }
      }
    }
  }
  cbar();
  const int h = tid >> 6, d = tid & 63;  // 448 = 7 x 64
  // a lane looks at one warp's maximum and sum, the weights then go round by shuffles
  float mx, num = 0.f, den;
  {
    const float* pw = reinterpret_cast<const float*>(smem_base) + h * 66;
    const float mw = lane < n_act ? pw[lane * (kHalfBytes / 4) + 64] : -INFINITY;
    const float lw = lane < n_act ? pw[lane * (kHalfBytes / 4) + 65] : 0.f;
    float ow[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) ow[w] = w < n_act ? pw[w * (kHalfBytes / 4) + d] : 0.f;
    mx = mw;
#pragma unroll
    for (int x = 1; x < 16; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
    mx = __shfl_sync(0xffffffffu, mx, 0);  // (the warps' results are in lanes 0..15)
    const float e = mw == -INFINITY ? 0.f : __expf(mw - mx);
    den = e * lw;
#pragma unroll
    for (int x = 1; x < 16; x <<= 1) den += __shfl_xor_sync(0xffffffffu, den, x);
    den = __shfl_sync(0xffffffffu, den, 0);
#pragma unroll
    for (int w = 0; w < 4; ++w) num = fmaf(__shfl_sync(0xffffffffu, e, w), ow[w], num);
    if (n_act > 4) {
      float o2[kWarps - 4];
#pragma unroll
      for (int w = 4; w < kWarps; ++w) o2[w - 4] = w < n_act ? pw[w * (kHalfBytes / 4) + d] : 0.f;
#pragma unroll
      for (int w = 4; w < kWarps; ++w) num = fmaf(__shfl_sync(0xffffffffu, e, w), o2[w - 4], num);
    }
  }
  if (a.splits > 1) {  // un-normalised, with maximum and sum: the o_proj CTAs merge the splits
    att_f[h * kHeadDim + d] = num;
    if (d == 0) {
      att_f[kGroupHeads * kHeadDim + 2 * h] = mx;
      att_f[kGroupHeads * kHeadDim + 2 * h + 1] = den;
    }
    cbar();
    if (tid < kPartWords / 2) {
      const int hh = tid / 17, w = tid - 17 * hh;
      unsigned char* dst = copy_of(a, sl.part, kPartBuf, layer_no) +
                           ((size_t)(r.row * a.splits + r.split) * kPartWords + kPartWords / 2 * r.kvh + tid) * 16;
      if (w < 16) {
        const uint4 v = *reinterpret_cast<const uint4*>(att_f + hh * kHeadDim + 4 * w);
        st_word(dst, data_word(v.x, v.y, v.z, v.w));
      } else {
        const float* p = att_f + kGroupHeads * kHeadDim + 2 * hh;
        st_word(dst, data_word(__float_as_uint(p[0]), __float_as_uint(p[1]), 0u, 0u));
      }
    }
  } else {
    half* out = reinterpret_cast<half*>(att_f);
    out[h * kHeadDim + d] = __float2half_rn(den > 0.f ? num / den : 0.f);
    cbar();
    if (tid < kXWords / 2) {
      const uint4 d4 = *reinterpret_cast<const uint4*>(out + 8 * tid);
      st_word(copy_of(a, sl.att, kXBuf, layer_no) + ((size_t)r.row * kXWords + 56 * r.kvh + tid) * 16,
              data_word(d4.x, d4.y, d4.z, d4.w));
    }
  }
  if (layer + 1 < a.n_layers) attn_request<MR, F16>(a, th, r, layer + 1);
  return true;
}

// ---- lm_head ------------------------------------------------------------------------------------
__device__ __forceinline__ u64 cand_key(float v, uint32_t idx) {
  uint32_t u = __float_as_uint(v);
  u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
  return ((u64)u << 32) | (uint32_t)~idx;  // larger logit first, then the lower index
}
// One 16-row tile of the table into this warp's stage.
template <int MR, bool F16>
__device__ __forceinline__ void lm_request(const PersistArgs& a, int tile, int warp, int lane) {
  using L = SL<MR, F16>;
  const uint32_t base = smem_u32(smem_base), bar = base + L::bars + 8 * (2 * L::n_ring + warp);
  const int row = 16 * tile + lane;
  const int rows = a.vocab - 16 * tile < 16 ? a.vocab - 16 * tile : 16;
  if (lane == 0) mbar_expect_tx(bar, (uint32_t)rows * kHidden * 2);
  __syncwarp();
  if (lane < rows)
    bulk_load_stream(base + warp * kLmStage + lane * kLmRow, a.embed + (size_t)row * kHidden, kHidden * 2, bar,
                     evict_first_policy());
}

// Final norm -> tied lm_head -> argmax over all CTAs.
template <int MR, bool F16>
__device__ __forceinline__ bool phase_lm_head(uint32_t last_no) {
  using L = SL<MR, F16>;
  const SmArgs& sa = sm_args<MR, F16>();
  const PersistArgs& a = sa.a;
  const Th th = make_th<MR>(sa);
  constexpr int NB = (MR + 7) / 8;
  const int tid = th.tid, warp = th.warp, lane = th.lane, g = lane >> 2, t = lane & 3;
  const SyncLayout sl = sync_layout();
  const int tiles = (a.vocab + 15) >> 4;
  const int tb = (int)((int64_t)tiles * th.cta / kCtas), te = (int)((int64_t)tiles * (th.cta + 1) / kCtas);
  const uint32_t base = smem_u32(smem_base), bar = base + L::bars + 8 * (2 * L::n_ring + warp);
  bool bad = false;
  uint32_t lm_par = (uint32_t)SMEM_I32(L::state)[49 + (warp < L::n_lm ? warp : 0)];  // parity of the warp's stage
  bool flying = false;  // a copy into this warp's stage has not been waited for
  // (the stages lie over memory that ordinary stores have written: order them before the copies)
  fence_proxy_async();
  cbar();
  if (warp < L::n_lm && tb + warp < te) {
    lm_request<MR, F16>(a, tb + warp, warp, lane);
    flying = true;
  }
  const bool ok = norm_rows<MR, F16>(th.c, copy_of(a, sl.x, kXBuf, last_no), a.ln + (size_t)2 * a.n_layers * kHidden,
                                     th.nrows, a.eps, tid, (a.n_layers * 8 + kPhX) & 0xFF, 4u);
  float bv[NB][2];
  uint32_t bi[NB][2];
#pragma unroll
  for (int nb = 0; nb < NB; ++nb)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      bv[nb][e] = -INFINITY;
      bi[nb][e] = 0x7fffffffu;
    }
  if (warp < L::n_lm) {
    const uint32_t stage = base + warp * kLmStage;
    for (int tile = tb + warp; tile < te; tile += L::n_lm) {
      if (!__all_sync(0xffffffffu, ring_wait<MR, F16>(bar, lm_par))) {
        bad = true;
        break;
      }
      flying = false;
      lm_par ^= 1u;
      float d[NB][2][4];
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int q = 0; q < 2; ++q) d[nb][q][0] = d[nb][q][1] = d[nb][q][2] = d[nb][q][3] = 0.f;
      const uint32_t arow = stage + (lane & 15) * kLmRow + (lane >> 4) * 16;
#pragma unroll 4
      for (int k2 = 0; k2 < kHidden / 32; ++k2) {
        uint32_t A0[4], A1[4];
        ldsm4(A0, arow + k2 * 64);
        ldsm4(A1, arow + k2 * 64 + 32);
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          int r = 8 * nb + (lane & 7);
          r = r < MR ? r : MR - 1;
          uint32_t b[4];
          ldsm4(b, base + L::xs + (uint32_t)(r * kXStride + 32 * k2 + 8 * (lane >> 3)) * 2u);
          mma16816(d[nb][0], A0[0], A0[1], A0[2], A0[3], b[0], b[1]);
          mma16816(d[nb][1], A1[0], A1[1], A1[2], A1[3], b[2], b[3]);
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (tile + L::n_lm < te && ok) {
        lm_request<MR, F16>(a, tile + L::n_lm, warp, lane);
        flying = true;
      }
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const uint32_t row = 16u * tile + g + 8 * hh;
        if (row < (uint32_t)a.vocab) {
#pragma unroll
          for (int nb = 0; nb < NB; ++nb)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const half lh = __float2half_rn(d[nb][0][2 * hh + e] + d[nb][1][2 * hh + e]);
              const float lv = __half2float(lh);
              const int m = 8 * nb + 2 * t + e;
              if (a.logits != nullptr && m < th.nrows) a.logits[(size_t)m * a.vocab + row] = lh;
              if (lv > bv[nb][e]) {
                bv[nb][e] = lv;
                bi[nb][e] = row;
              }
            }
        }
      }
      if (!ok) break;
    }
  }
  if (lane == 0 && warp < L::n_lm) SMEM_I32(L::state)[49 + warp] = (int)lm_par;
  if (flying) ring_wait<MR, F16>(bar, lm_par);  // (only after a wait that ran out)
  // ---- candidates: lanes of a column, warps, CTAs ----
  u64* cand = reinterpret_cast<u64*>(smem_base + L::cand);  // [warp][MR]
#pragma unroll
  for (int nb = 0; nb < NB; ++nb)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      u64 key = cand_key(bv[nb][e], bi[nb][e]);
#pragma unroll
      for (int s = 4; s < 32; s <<= 1) {
        const u64 other = __shfl_xor_sync(0xffffffffu, key, s);
        key = other > key ? other : key;
      }
      const int m = 8 * nb + 2 * t + e;
      if (g == 0 && m < MR && warp < L::n_lm) cand[warp * MR + m] = key;
    }
  __syncwarp();
  if (lane == 0) mbar_arrive(base + L::bars + 8 * (2 * L::n_ring + L::n_lm));
  if (cbar_or(bad || !ok)) return false;
  int* s_tok = SMEM_I32(L::state) + 32;
  for (int m = warp; m < th.nrows; m += kWarps) {
    u64 key = lane < L::n_lm ? cand[lane * MR + m] : 0ull;
#pragma unroll
    for (int s = 1; s < 8; s <<= 1) {
      const u64 other = __shfl_xor_sync(0xffffffffu, key, s);
      key = other > key ? other : key;
    }
    if (lane == 0)
      st_word(a.sync + sl.cand + ((size_t)m * kCtas + th.cta) * 16, word32((uint32_t)key, (uint32_t)(key >> 32), 0u, last_no));
    uint32_t pending = 0;
#pragma unroll
    for (int q = 0; q < 5; ++q)
      if (lane + 32 * q < kCtas) pending |= 1u << q;
    const uint32_t want = pending;
    Word w5[5] = {};
    poll_words<5, true>(
        th.c, [&](int q) { return a.sync + sl.cand + ((size_t)m * kCtas + lane + 32 * q) * 16; }, pending, last_no, w5,
        (a.n_layers * 8 + kPhCand) & 0xFF, 8u, bad);
    __syncwarp();
    key = 0ull;
    if (!bad) {
#pragma unroll
      for (int q = 0; q < 5; ++q)
        if ((want & (1u << q)) && w5[q].lo > key) key = w5[q].lo;
    }
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const u64 other = __shfl_xor_sync(0xffffffffu, key, s);
      key = other > key ? other : key;
    }
    if (lane == 0) {
      const uint32_t idx = ~(uint32_t)key;
      s_tok[m] = idx < (uint32_t)a.vocab ? (int)idx : 0;  // (no logit above -inf: token 0, as the chain)
    }
  }
  return !cbar_or(bad);
}

// ---- the producer: one thread streams the CTA's chunks in the order its phases consume them ------
template <int MR, bool F16>
__device__ __forceinline__ void produce(const PersistArgs& a, int cta, int q0, int qn, bool res, int g0, int gn) {
  using L = SL<MR, F16>;
  using W = Wt<F16>;
  const uint32_t base = smem_u32(smem_base), bars = base + L::bars;
  uint32_t slot = 0, par = 0, issued = 0;
  const u64 policy = evict_first_policy();
  bool go = true;
  // runs of consecutive chunks: first chunk, count, and (down) the bytes of the last piece's chunks
  auto run = [&](const unsigned char* layer, int first, int count, int short_from) {
    for (int i = 0; i < count && go; ++i) {
      if (issued >= (uint32_t)L::n_ring) {
        // (a slot's earlier use was released: one phase behind)
        const uint32_t empty = bars + 8 * (L::n_ring + slot);
        if (!ring_wait<MR, F16>(empty, par ^ 1u)) {
          go = false;
          break;
        }
      }
      const uint32_t bytes = i >= short_from ? (uint32_t)W::last_down : (uint32_t)W::chunk;
      mbar_expect_tx(bars + 8 * slot, bytes);
      bulk_load_stream(base + L::ring + slot * W::chunk, layer + (size_t)(first + i) * W::chunk, bytes, bars + 8 * slot, policy);
      ++issued;
      if (++slot == (uint32_t)L::n_ring) {
        slot = 0;
        par ^= 1u;
      }
    }
  };
  for (int step = 0; step < a.steps && go; ++step) {
    if (step > 0) {  // the ring's memory held lm_head tiles
      if (!ring_wait<MR, F16>(bars + 8 * (2 * L::n_ring + L::n_lm), (uint32_t)(step - 1) & 1u)) break;
    }
    for (int l = 0; l < a.n_layers && go; ++l) {
      const unsigned char* layer = a.chunks + (size_t)l * W::per_layer * W::chunk;
      if (qn > 0) run(layer, q0 * W::per_piece, qn * W::per_piece, 1 << 30);
      if (res) run(layer, W::off_o + cta * W::per_piece, W::per_piece, 1 << 30);
      run(layer, W::off_gu + g0 * W::per_piece, gn * W::per_piece, 1 << 30);
      if (res)
        run(layer, W::off_down + cta * kDownPieces * W::per_piece, kDownPieces * W::per_piece,
            (kDownPieces - 1) * W::per_piece);
    }
  }
  // no copy may be on its way when the CTA ends: the last use of every slot has landed
  for (uint32_t i = 0; i < (uint32_t)L::n_ring && i < issued; ++i) {
    const uint32_t n = issued - 1 - i;  // chunk number
    mbar_wait(bars + 8 * (n % L::n_ring), (n / L::n_ring) & 1u);
  }
}

// Start of a token: the attention CTA's range and its first tiles, the rotation of the QKV CTA's
// tiles at the rows' positions, the residual CTA's elements of the embedding rows.
template <int MR, bool F16>
__device__ __forceinline__ void token_begin() {
  using L = SL<MR, F16>;
  SmArgs& sa = *reinterpret_cast<SmArgs*>(smem_base + L::args);
  const PersistArgs& a = sa.a;
  const Th th = make_th<MR>(sa);
  const int* state = SMEM_I32(L::state);
  if (th.cta >= a.ng) {
    if (th.tid == 0) {
      AttnRole& r = sa.role;
      r.pos = state[r.row];
      // the last split takes the rest: every position belongs to a split, whatever the context hint said
      const int hi = r.split + 1 < a.splits ? r.t_lo + a.chunk_tokens : a.s_max;
      r.t_end = r.slot < 0 ? r.t_lo : (r.pos + 1 < hi ? r.pos + 1 : hi);
      if (r.t_end < r.t_lo) r.t_end = r.t_lo;
    }
    cbar();
    attn_request<MR, F16>(a, th, sa.role, 0);
  }
  float2* rope = reinterpret_cast<float2*>(smem_base + L::rope);
  for (int i = th.tid; i < sa.qn * a.batch * 8; i += kComp) {
    const int d = i & 7, u = i >> 3, tt = u / a.batch, m = u - tt * a.batch;
    int p = state[m];
    p = p < a.max_pos ? p : a.max_pos - 1;
    const size_t at = (size_t)p * 32 + 8 * ((sa.q0 + tt) & 3) + d;
    rope[(tt * MR + m) * 8 + d] = make_float2(__half2float(a.cos_t[at]), __half2float(a.sin_t[at]));
  }
  const int m = 2 * th.warp + (th.lane >> 4), c = (th.lane & 15) < kResCols ? (th.lane & 15) : kResCols - 1;
  if (th.cta < kResCtas && m < a.batch)
    SMEM_HALF(L::resid)[th.tid] = a.embed[(size_t)state[32 + m] * kHidden + kResCols * th.cta + c];
}

// End of a token: CTA 0 writes the slot state, every CTA keeps its own copy of it.
template <int MR, bool F16>
__device__ __forceinline__ void token_end(int step) {
  using L = SL<MR, F16>;
  const SmArgs& sa = sm_args<MR, F16>();
  const PersistArgs& a = sa.a;
  const Th th = make_th<MR>(sa);
  int* state = SMEM_I32(L::state);
  if (th.tid < a.batch) {
    const int slot = state[16 + th.tid], p = state[th.tid] + 1, tk = state[32 + th.tid];
    if (th.cta == 0 && slot >= 0) {
      a.tok[slot] = tk;
      a.pos[slot] = p;
      if (a.out_tokens != nullptr) a.out_tokens[(size_t)((sa.step0 + step) % a.ring) * a.n_slots + slot] = tk;
    }
    state[th.tid] = p < a.s_max ? p : a.s_max - 1;
  }
  if (th.cta == 0 && th.tid == 0 && a.step_counter != nullptr) *a.step_counter = sa.step0 + step + 1;
  cbar();
}

// The status word goes to the host only where it says something: the host's word is zero before the launch, and one that nobody
// waits for may be given back while the kernel runs.
__device__ __forceinline__ void tell_host(const PersistArgs& a, const uint32_t* hdr) {
  const int32_t status = (int32_t)ld_relaxed_u32(hdr + 1);
  if (a.host_status != nullptr && status != 0) *a.host_status = status;
}

template <int MR, bool F16>
__global__ void __launch_bounds__(kThreads, 1) token_kernel(const __grid_constant__ PersistArgs a) {
  using L = SL<MR, F16>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = blockIdx.x;
  const uint32_t bars = smem_u32(smem_base) + L::bars;
  int* state = SMEM_I32(L::state);
  uint32_t* hdr = reinterpret_cast<uint32_t*>(a.sync);
  const bool res = cta < kResCtas, attn = cta >= a.ng;
  const int q0 = (cta - kResCtas) * a.tq;
  const int qn = (!res && cta - kResCtas < a.nq) ? (kQkvTiles - q0 < a.tq ? kQkvTiles - q0 : a.tq) : 0;

  // after a wait that ran out the exchange area holds what it holds, until the status is read and the
  // area cleared by the host
  if (__syncthreads_or(tid == 0 && ld_relaxed_u32(hdr + 1) != 0u)) {
    if (cta == 0 && tid == 0) tell_host(a, hdr);
    return;
  }
  if (tid == 0) {
    for (int i = 0; i < L::n_ring; ++i) {
      mbar_init(bars + 8 * i, 1);
      mbar_init(bars + 8 * (L::n_ring + i), kWarps);
    }
    for (int i = 0; i < L::n_lm; ++i) mbar_init(bars + 8 * (2 * L::n_ring + i), 1);
    mbar_init(bars + 8 * (2 * L::n_ring + L::n_lm), kWarps);
    for (int i = 48; i < 64; ++i) state[i] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < kMaxRows) {
    int slot = -1, p = 0, tk = 0;
    if (tid < a.batch) {
      slot = a.rows[tid];
      if (slot < 0 || slot >= a.n_slots) slot = -1;
      if (slot >= 0) {
        p = __ldcg(a.pos + slot);
        const int64_t f = a.n_feed > 0 ? a.tok + slot - a.feed_dst : -1;
        tk = f >= 0 && f < a.n_feed ? a.feed[f] : __ldcg(a.tok + slot);
      }
      p = p < 0 ? 0 : (p < a.s_max ? p : a.s_max - 1);
      tk = tk < 0 ? 0 : (tk >= a.vocab ? a.vocab - 1 : tk);
    }
    if (cta == 0 && tid < a.n_feed) a.feed_dst[tid] = a.feed[tid];
    // the candidate words keep their last contents and tag, and the tags come round again with the layer numbers
    empty_word(a.sync + sync_layout().cand + ((size_t)tid * kCtas + cta) * 16);
    state[tid] = p;
    state[16 + tid] = slot;
    state[32 + tid] = tk;
  }
  __syncthreads();

  if (warp == kWarps) {  // ---- producer warp ----
    if (lane == 0 && !attn) produce<MR, F16>(a, cta, q0, qn, res, gu_first(a, cta), gu_count(a, cta));
    return;
  }

  SmArgs& sa = *reinterpret_cast<SmArgs*>(smem_base + L::args);
  if (tid == 0) {
    sa.a = a;
    const uint32_t limit = ld_relaxed_u32(hdr + 2);
    sa.poll_limit = limit != 0u ? limit : kPollLimit;
    sa.withhold_layer = (int)ld_relaxed_u32(hdr + 3) - 1;
    sa.no0 = ld_relaxed_u32(hdr) % kNumbers;
    sa.step0 = a.step_counter != nullptr ? __ldcg(a.step_counter) : 0;
    sa.q0 = q0;
    sa.row_magic = (65536u + (uint32_t)a.batch - 1u) / (uint32_t)a.batch;
    sa.qn = qn;
    const int i = attn ? cta - a.ng : 0;
    sa.role.split = i % a.splits;
    sa.role.row = (i / a.splits) >> 1;
    sa.role.kvh = (i / a.splits) & 1;
    sa.role.slot = state[16 + sa.role.row];
    sa.role.t_lo = sa.role.split * a.chunk_tokens;
  }
  cbar();

  uint32_t rp = kAlive;
  for (int step = 0; step < sa.a.steps; ++step) {
    token_begin<MR, F16>();
    for (int layer = 0; layer < sa.a.n_layers; ++layer) {
      const uint32_t no = sa.no0 + (uint32_t)(step * sa.a.n_layers + layer) + 1u;
      if ((int)blockIdx.x >= sa.a.ng) {
        rp = phase_attention<MR, F16>(layer, no) ? rp : 0u;
      } else {
        if (sa.qn > 0) rp = phase_qkv<MR, F16>(rp, layer, no);
        if (rp) rp = phase_mid<MR, F16>(rp, layer, no);
        if (rp && blockIdx.x < kResCtas) rp = phase_down<MR, F16>(rp, layer, no);
      }
      if (rp == 0u) break;
    }
    if (rp == 0u) break;
    if (!phase_lm_head<MR, F16>(sa.no0 + (uint32_t)((step + 1) * sa.a.n_layers))) {
      rp = 0u;
      break;
    }
    token_end<MR, F16>(step);
  }
  if (rp == 0u && threadIdx.x == 0) *reinterpret_cast<volatile int*>(state + 48) = 1;
  cp_async_wait_all();
  if (rp != 0u) {  // everybody has read everything: leave every word empty for the next launch, whatever its rows
    const Th th = make_th<MR>(sa);
    const uint32_t last = sa.no0 + (uint32_t)(sa.a.steps * sa.a.n_layers);
    for (uint32_t no = last - 1u; no <= last; ++no) {
      if (th.cta >= sa.a.ng) {
        empty_att(sa.a, th, sa.role.row, sa.role.kvh, sa.role.split, no);
      } else {
        if (sa.qn > 0) empty_qkv(sa.a, th, sa.q0, sa.qn, no);
        empty_act(sa.a, th, gu_first(sa.a, th.cta), gu_count(sa.a, th.cta), no);
        if (th.cta < kResCtas) empty_residual(sa.a, th, no);
      }
    }
  }
  // The layer numbers that an abandoned burst may have used are spent: their tags must not be met again.
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) {
      hdr[0] = sa.no0 + (uint32_t)(a.steps * a.n_layers);
      tell_host(a, hdr);
    }
    for (int i = threadIdx.x; i < a.n_out; i += kComp) a.host_out[i] = __ldcg(a.out_src + i);
  }
}

// ---- weight stream ------------------------------------------------------------------------------
struct PackArgs {
  quic_w4_t qkv, o, gu, down;
  const half* ln1;
  const half* ln2;
  unsigned char* chunks;  // this layer
  half* ln;               // this layer: [2][896]
  half* bias;             // this layer: [72][16]
};
// Row of the device matrix that row r of a tile holds, or -1.
__device__ __forceinline__ int tile_row(int which, int tile, int r) {
  if (which == 0) {  // rotation partners in rows r and r + 8; a head's columns are stored (0, 32, 1, 33, ..)
    const int dim = 8 * (tile & 3) + (r & 7);
    return (tile >> 2) * kHeadDim + 2 * dim + (r >> 3);
  }
  if (which == 2) return r < 8 ? 8 * tile + r : kInter + 8 * tile + r - 8;
  return r < kResCols ? kResCols * tile + r : -1;
}
__device__ __forceinline__ uint32_t w4_nibble(const quic_w4_t& w, int n, int k) {
  return ((uint32_t)w.qw[(size_t)(k >> 3) * w.n + n] >> (4 * (k & 7))) & 15u;
}
// One block per (tile, piece of 896 k): 72 + 64 + 608 + 64 x 6 blocks of 448 threads.
template <bool F16>
__global__ void __launch_bounds__(kComp) pack_kernel(const PackArgs a) {
  int i = blockIdx.x, which, tile, piece = 0;
  size_t chunk;
  if (i < kQkvTiles) {
    which = 0, tile = i, chunk = (size_t)i * Wt<F16>::per_piece;
  } else if ((i -= kQkvTiles) < kResCtas) {
    which = 1, tile = i, chunk = Wt<F16>::off_o + (size_t)i * Wt<F16>::per_piece;
  } else if ((i -= kResCtas) < kGuTiles) {
    which = 2, tile = i, chunk = Wt<F16>::off_gu + (size_t)i * Wt<F16>::per_piece;
  } else {
    i -= kGuTiles;
    which = 3, tile = i / kDownPieces, piece = i - tile * kDownPieces;
    chunk = Wt<F16>::off_down + (size_t)i * Wt<F16>::per_piece;
  }
  const quic_w4_t& w = which == 0 ? a.qkv : (which == 1 ? a.o : (which == 2 ? a.gu : a.down));
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  unsigned char* dst = a.chunks + chunk * Wt<F16>::chunk;
  for (int j = 0; j < 4; ++j) {
    uint32_t word = 0;
    uint32_t h[4];
    for (int q = 0; q < 4; ++q) {
      const int n = tile_row(which, tile, (lane >> 2) + 8 * (q & 1));
      const int k = 896 * piece + 64 * warp + 16 * (lane & 3) + 4 * j + 2 * (q >> 1);
      const bool ok = n >= 0 && k < w.k;
      if (F16) {
        h[q] = ok ? *reinterpret_cast<const uint32_t*>(reinterpret_cast<const half*>(w.w16) + (size_t)n * w.k + k) : 0u;
      } else if (ok) {
        word |= w4_nibble(w, n, k) << (4 * q);
        word |= w4_nibble(w, n, k + 1) << (4 * (q + 4));
      }
    }
    if (F16)
      *reinterpret_cast<uint4*>(dst + (size_t)j * Wt<F16>::chunk + warp * 512 + lane * 16) = make_uint4(h[0], h[1], h[2], h[3]);
    else
      *reinterpret_cast<uint32_t*>(dst + kScaleBytes + warp * 512 + lane * 16 + 4 * j) = word;
  }
  if (!F16 && lane < 8) {
    const int k = 896 * piece + 64 * warp;
    half s[2];
    uint32_t z[2];
    for (int q = 0; q < 2; ++q) {
      const int n = tile_row(which, tile, lane + 8 * q);
      const bool ok = n >= 0 && k < w.k;
      s[q] = ok ? reinterpret_cast<const half*>(w.sc)[(size_t)(k / kGroup) * w.n + n] : __float2half(0.f);
      z[q] = ok ? ((uint32_t)w.zp[(size_t)(k / kGroup) * (w.n >> 1) + (n >> 1)] >> (4 * (n & 1))) & 15u : 0u;
    }
    uint2 e;
    e.x = (uint32_t)__half_as_ushort(s[0]) | ((uint32_t)__half_as_ushort(s[1]) << 16);
    const half2 zh = __halves2half2(__int2half_rn(1024 + (int)z[0]), __int2half_rn(64 + (int)z[1]));
    e.y = *reinterpret_cast<const uint32_t*>(&zh);
    *reinterpret_cast<uint2*>(dst + warp * 64 + lane * 8) = e;
  }
  if (which == 0 && t < 16)
    a.bias[tile * 16 + t] =
        w.bias ? reinterpret_cast<const half*>(w.bias)[tile_row(0, tile, t)] : __float2half(0.f);
  if (blockIdx.x == 0) {
    for (int i = t; i < kHidden; i += kComp) {
      a.ln[i] = a.ln1[i];
      a.ln[kHidden + i] = a.ln2[i];
    }
  }
}
__global__ void pack_norm_kernel(const half* src, half* out) { out[threadIdx.x] = src[threadIdx.x]; }

inline int64_t bias_offset(int n_layers) { return (int64_t)(2 * n_layers + 1) * kHidden * 2; }
inline int64_t stream_header_bytes(int n_layers) {
  return (bias_offset(n_layers) + (int64_t)n_layers * kQkvTiles * 32 + 255) / 256 * 256;
}
template <bool F16>
inline int64_t stream_bytes(int n_layers) {
  if (n_layers < 1 || n_layers > kMaxLayers) return 0;
  return stream_header_bytes(n_layers) + (int64_t)n_layers * Wt<F16>::per_layer * Wt<F16>::chunk;
}

// Launches of this process on one device follow one another whatever stream they are on: two grids that
// both need every SM must not each hold a part of them.
struct LaunchOrder {
  std::mutex mu;
  cudaEvent_t done = nullptr;
  cudaStream_t last = nullptr;
};
LaunchOrder g_order[64];

// Whether all CTAs can be resident on the device at once (MIG and MPS limits show in its count of SMs).
bool device_holds_kernel(int dev) {
  int sms = 0, coop = 0, smem = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return sms >= kCtas && coop != 0 && smem >= kSmemMax;
}

template <int MR, bool F16>
int launch_token_kernel(const PersistArgs& pa, int dev, cudaStream_t st) {
  static bool configured[64] = {};
  constexpr int smem = SL<MR, F16>::total;
  if (!configured[dev]) {
    QUIC_REQUIRE(device_holds_kernel(dev), QUIC_E_SHAPE,
                 "decode_persist: needs 148 SMs and cooperative launch (every CTA must be resident)");
    QUIC_CUDA(cudaFuncSetAttribute(token_kernel<MR, F16>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    int per_sm = 0;
    QUIC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, token_kernel<MR, F16>, kThreads, smem));
    QUIC_REQUIRE(per_sm >= 1, QUIC_E_SHAPE, "decode_persist: the kernel does not fit an SM");
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kCtas);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  QUIC_CUDA(cudaLaunchKernelEx(&cfg, token_kernel<MR, F16>, pa));
  return QUIC_OK;
}
template <bool F16>
int launch_rows(const PersistArgs& pa, int dev, cudaStream_t st) {
  if (pa.batch <= 1) return launch_token_kernel<1, F16>(pa, dev, st);
  if (pa.batch <= 2) return launch_token_kernel<2, F16>(pa, dev, st);
  if (pa.batch <= 4) return launch_token_kernel<4, F16>(pa, dev, st);
  if (pa.batch <= 8) return launch_token_kernel<8, F16>(pa, dev, st);
  return launch_token_kernel<16, F16>(pa, dev, st);
}

// After a launch that gave up: empties the exchange buffers (nothing else runs on the area meanwhile)
// and then the status word.
inline int clear_sync(void* sync, cudaStream_t st, int rc, int32_t* status_out, int32_t status) {
  unsigned char* base = static_cast<unsigned char*>(sync);
  QUIC_CUDA(cudaMemsetAsync(base + 256, 0, (size_t)(sync_layout().total - 256), st));
  QUIC_CUDA(cudaMemsetAsync(base + 4, 0, 4, st));
  *status_out = status;
  return rc;
}
inline bool dense_model(const quic_model_t* m) { return m->layers[0].qkv.w16 != nullptr; }

}  // namespace
}  // namespace quic

using namespace quic;

extern "C" int32_t quic_persist_max_rows(void) { return kMaxRows; }

extern "C" int32_t quic_persist_device_ok(void) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return device_holds_kernel(dev) ? 1 : 0;
}

extern "C" int64_t quic_persist_stream_bytes(int32_t n_layers) { return stream_bytes<false>(n_layers); }
extern "C" int64_t quic_persist_stream_bytes_f16(int32_t n_layers) { return stream_bytes<true>(n_layers); }

extern "C" int64_t quic_persist_sync_bytes(void) { return sync_layout().total; }

// One split while the context fits a CTA's shared memory: merging splits in the o_proj CTAs costs ~2 us
// a layer, more than the attention of 768 tokens (1.5 us).  Every split is one CTA less for the
// linears; more rows than eight (two row blocks, no room for the merge) take one split, and longer
// splits than fit shared memory fetch their later half tiles within the phase.
extern "C" int32_t quic_persist_pick_splits(int32_t batch, int32_t ctx) {
  if (ctx < 1) ctx = 1;
  if (batch < 1) batch = 1;
  if (batch > kMaxRows) return 1 << 20;
  int most = batch > 8 ? 1 : kMaxParts / (2 * batch);
  if (most > 8) most = 8;
  int s = (ctx + 767) / 768;
  s = s > most ? most : s;
  return (ctx + s - 1) / s > 4096 ? 1 << 20 : s;
}

extern "C" int quic_persist_pack(const quic_model_t* m, void* stream_out, void* stream) {
  QUIC_REQUIRE(m && stream_out, QUIC_E_ARG, "persist_pack: null argument");
  QUIC_REQUIRE(m->n_layers >= 1 && m->n_layers <= kMaxLayers && m->layers, QUIC_E_SHAPE, "persist_pack: 1..64 layers");
  QUIC_REQUIRE((uintptr_t)stream_out % 256 == 0, QUIC_E_ARG, "persist_pack: output must be 256-byte aligned");
  QUIC_REQUIRE(m->final_norm, QUIC_E_ARG, "persist_pack: missing final norm");
  unsigned char* base = static_cast<unsigned char*>(stream_out);
  const int64_t hdr = stream_header_bytes(m->n_layers);
  const bool f16 = dense_model(m);
  half* ln = reinterpret_cast<half*>(base);
  half* bias = reinterpret_cast<half*>(base + bias_offset(m->n_layers));
  cudaStream_t st = (cudaStream_t)stream;
  for (int l = 0; l < m->n_layers; ++l) {
    const quic_layer_t& L = m->layers[l];
    QUIC_REQUIRE(L.qkv.n == kQkvN && L.qkv.k == kHidden && L.o.n == kHidden && L.o.k == kHidden &&
                     L.gate_up.n == 2 * kInter && L.gate_up.k == kHidden && L.down.n == kHidden &&
                     L.down.k == kInter,
                 QUIC_E_SHAPE, "persist_pack: layer shapes are not Qwen2.5-0.5B's");
    if (f16) {
      QUIC_REQUIRE(L.qkv.w16 && L.o.w16 && L.gate_up.w16 && L.down.w16 && L.ln1 && L.ln2, QUIC_E_ARG,
                   "persist_pack: missing layer tensor");
    } else {
      QUIC_REQUIRE(L.qkv.qw && L.o.qw && L.gate_up.qw && L.down.qw && L.ln1 && L.ln2, QUIC_E_ARG,
                   "persist_pack: missing layer tensor");
    }
    PackArgs pa;
    pa.qkv = L.qkv;
    pa.o = L.o;
    pa.gu = L.gate_up;
    pa.down = L.down;
    pa.ln1 = (const half*)L.ln1;
    pa.ln2 = (const half*)L.ln2;
    pa.chunks = base + hdr + (size_t)l * (f16 ? (size_t)Wt<true>::per_layer * Wt<true>::chunk
                                              : (size_t)Wt<false>::per_layer * Wt<false>::chunk);
    pa.ln = ln + (size_t)l * 2 * kHidden;
    pa.bias = bias + (size_t)l * kQkvTiles * 16;
    const int blocks = kQkvTiles + kResCtas + kGuTiles + kResCtas * kDownPieces;
    if (f16) pack_kernel<true><<<blocks, kComp, 0, st>>>(pa);
    else pack_kernel<false><<<blocks, kComp, 0, st>>>(pa);
    QUIC_CUDA(cudaGetLastError());
  }
  pack_norm_kernel<<<1, kHidden, 0, st>>>((const half*)m->final_norm, ln + (size_t)m->n_layers * 2 * kHidden);
  QUIC_CUDA(cudaGetLastError());
  return QUIC_OK;
}

namespace {
// The host-driven form's part of a launch: tokens by value, results to mapped host memory.
struct HostIo {
  const int32_t* in = nullptr;
  int32_t* dev_in = nullptr;
  int32_t n_in = 0;
  const int32_t* dev_out = nullptr;
  int32_t* out = nullptr;
  int32_t n_out = 0;
  int32_t* status = nullptr;
};
int launch_persist(const quic_model_t* m, const quic_decode_t* d, const void* wstream, void* sync, int32_t steps,
                   void* stream, const HostIo& io) {
  QUIC_REQUIRE(m && d && wstream && sync, QUIC_E_ARG, "decode_persist: null argument");
  QUIC_REQUIRE(m->n_layers >= 1 && m->n_layers <= kMaxLayers && m->layers, QUIC_E_SHAPE, "decode_persist: 1..64 layers");
  QUIC_REQUIRE(m->vocab >= 2 * kCtas && m->vocab % 2 == 0, QUIC_E_SHAPE,
               "decode_persist: even vocabulary of at least 296 rows");
  QUIC_REQUIRE(m->embed && m->final_norm && m->rope_cos && m->rope_sin && m->max_pos >= 1, QUIC_E_ARG,
               "decode_persist: missing model tensor");
  QUIC_REQUIRE((uintptr_t)m->embed % 16 == 0 && (uintptr_t)d->kv % 16 == 0, QUIC_E_ARG,
               "decode_persist: embedding and cache must be 16-byte aligned");
  QUIC_REQUIRE(d->kv && d->tok && d->pos && d->rows, QUIC_E_ARG, "decode_persist: missing state tensor");
  QUIC_REQUIRE(d->batch >= 1 && d->batch <= kMaxRows, QUIC_E_LIMIT, "decode_persist: 1..16 batch rows");
  QUIC_REQUIRE(d->n_slots >= 1 && d->s_max >= 1, QUIC_E_SHAPE, "decode_persist: bad cache geometry");
  QUIC_REQUIRE(steps >= 1 && steps <= 4096, QUIC_E_ARG, "decode_persist: 1..4096 steps");
  QUIC_REQUIRE(d->out_tokens == nullptr || (d->ring >= 1 && d->step_counter != nullptr), QUIC_E_ARG,
               "decode_persist: out_tokens needs ring >= 1 and a step counter");
  QUIC_REQUIRE(d->logits == nullptr || steps == 1, QUIC_E_ARG, "decode_persist: logits are kept for one step only");
  QUIC_REQUIRE((uintptr_t)wstream % 256 == 0 && (uintptr_t)sync % 256 == 0, QUIC_E_ARG,
               "decode_persist: stream and sync area must be 256-byte aligned");
  int ctx = d->ctx_hint > 0 ? d->ctx_hint : d->s_max;
  if (ctx > d->s_max) ctx = d->s_max;
  const int splits = d->attn_splits > 0 ? d->attn_splits : quic_persist_pick_splits(d->batch, ctx);
  QUIC_REQUIRE(splits <= 16 && 2 * d->batch * splits <= kMaxAttnCtas && (d->batch <= 8 || splits == 1), QUIC_E_LIMIT,
               "decode_persist: context too long or too many attention splits");
  PersistArgs pa = {};
  const unsigned char* base = static_cast<const unsigned char*>(wstream);
  pa.chunks = base + stream_header_bytes(m->n_layers);
  pa.ln = reinterpret_cast<const half*>(base);
  pa.bias = reinterpret_cast<const half*>(base + bias_offset(m->n_layers));
  pa.embed = (const half*)m->embed;
  pa.cos_t = (const half*)m->rope_cos;
  pa.sin_t = (const half*)m->rope_sin;
  pa.n_layers = m->n_layers;
  pa.vocab = m->vocab;
  pa.max_pos = m->max_pos;
  pa.eps = m->eps;
  pa.kv = (half*)d->kv;
  pa.n_slots = d->n_slots;
  pa.s_max = d->s_max;
  pa.tok = d->tok;
  pa.pos = d->pos;
  pa.rows = d->rows;
  pa.batch = d->batch;
  pa.out_tokens = d->out_tokens;
  pa.ring = d->ring > 0 ? d->ring : 1;
  pa.step_counter = d->step_counter;
  pa.logits = (half*)d->logits;
  pa.sync = static_cast<unsigned char*>(sync);
  pa.steps = steps;
  pa.splits = splits;
  pa.chunk_tokens = ((ctx + splits - 1) / splits + 63) / 64 * 64;
  pa.na = 2 * d->batch * splits;
  pa.ng = kCtas - pa.na;
  const int room = kCtas - kResCtas - pa.na;  // CTAs that can take QKV tiles
  pa.tq = (kQkvTiles + room - 1) / room;
  pa.nq = (kQkvTiles + pa.tq - 1) / pa.tq;
  for (int i = 0; i < io.n_in; ++i) pa.feed[i] = io.in[i];
  pa.feed_dst = io.dev_in;
  pa.n_feed = io.n_in;
  pa.out_src = io.dev_out;
  pa.host_out = io.out;
  pa.n_out = io.n_out;
  pa.host_status = io.status;
  cudaStream_t st = (cudaStream_t)stream;
  int dev = 0;
  QUIC_CUDA(cudaGetDevice(&dev));
  QUIC_REQUIRE(dev >= 0 && dev < 64, QUIC_E_LIMIT, "decode_persist: device index beyond 63");
  LaunchOrder& order = g_order[dev];
  std::lock_guard<std::mutex> hold(order.mu);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  QUIC_CUDA(cudaStreamIsCapturing(st, &capture));
  const bool ordered = capture == cudaStreamCaptureStatusNone;
  if (ordered) {
    if (order.done == nullptr) QUIC_CUDA(cudaEventCreateWithFlags(&order.done, cudaEventDisableTiming));
    else if (order.last != st) QUIC_CUDA(cudaStreamWaitEvent(st, order.done, 0));
  }
  const int rc = dense_model(m) ? launch_rows<true>(pa, dev, st) : launch_rows<false>(pa, dev, st);
  if (rc != QUIC_OK) return rc;
  if (ordered) {
    QUIC_CUDA(cudaEventRecord(order.done, st));
    order.last = st;
  }
  return QUIC_OK;
}
// Device address of page-locked host memory, or nullptr.
template <typename T>
T* mapped(T* host) {
  void* p = nullptr;
  if (host == nullptr || cudaHostGetDevicePointer(&p, host, 0) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  return static_cast<T*>(p);
}
}  // namespace

extern "C" int quic_decode_persist(const quic_model_t* m, const quic_decode_t* d, const void* wstream, void* sync,
                                   int32_t steps, void* stream) {
  return quic_decode_persist_watch(m, d, wstream, sync, steps, stream, nullptr);
}

extern "C" int quic_decode_persist_watch(const quic_model_t* m, const quic_decode_t* d, const void* wstream, void* sync,
                                         int32_t steps, void* stream, int32_t* host_status) {
  HostIo io;
  io.status = mapped(host_status);
  QUIC_REQUIRE(host_status == nullptr || io.status != nullptr, QUIC_E_ARG, "decode_persist: the status word is not page-locked");
  return launch_persist(m, d, wstream, sync, steps, stream, io);
}

extern "C" int quic_decode_persist_status(void* sync, void* stream, int32_t* status_out) {
  QUIC_REQUIRE(sync && status_out, QUIC_E_ARG, "decode_persist_status: null argument");
  cudaStream_t st = (cudaStream_t)stream;
  uint32_t v = 0;
  unsigned char* word = static_cast<unsigned char*>(sync) + 4;
  QUIC_CUDA(cudaMemcpyAsync(&v, word, 4, cudaMemcpyDeviceToHost, st));
  QUIC_CUDA(cudaStreamSynchronize(st));
  if (v != 0) return clear_sync(sync, st, QUIC_OK, status_out, (int32_t)v);
  *status_out = (int32_t)v;
  return QUIC_OK;
}

extern "C" int quic_decode_persist_run_host(const quic_model_t* m, const quic_decode_t* d, const void* wstream,
                                            void* sync, int32_t steps, void* stream, const int32_t* host_in,
                                            int32_t* dev_in, int32_t n_in, const int32_t* dev_out,
                                            int32_t* host_out, int32_t n_out, int32_t* host_status) {
  QUIC_REQUIRE(n_in >= 0 && n_out >= 0, QUIC_E_ARG, "decode_persist_run_host: negative count");
  QUIC_REQUIRE(n_in == 0 || (host_in != nullptr && dev_in != nullptr), QUIC_E_ARG,
               "decode_persist_run_host: null input buffer");
  QUIC_REQUIRE(n_out == 0 || (host_out != nullptr && dev_out != nullptr), QUIC_E_ARG,
               "decode_persist_run_host: null output buffer");
  QUIC_REQUIRE(host_status != nullptr && sync != nullptr, QUIC_E_ARG, "decode_persist_run_host: null status buffer");
  cudaStream_t st = (cudaStream_t)stream;
  // Page-locked buffers (the normal case): the tokens go in with the launch and the kernel stores its
  // results where the host reads them.  Three copy operations less between two tokens.
  HostIo io;
  int32_t* out_dev = n_out > 0 ? mapped(host_out) : nullptr;
  int32_t* status_dev = mapped(host_status);
  if (n_in <= kMaxRows) {
    io.in = host_in;
    io.dev_in = dev_in;
    io.n_in = n_in;
  } else {
    QUIC_CUDA(cudaMemcpyAsync(dev_in, host_in, sizeof(int32_t) * n_in, cudaMemcpyHostToDevice, st));
  }
  if (out_dev != nullptr) {
    io.dev_out = dev_out;
    io.out = out_dev;
    io.n_out = n_out;
  }
  io.status = status_dev;
  *host_status = 0;
  const int rc = launch_persist(m, d, wstream, sync, steps, stream, io);
  if (rc != QUIC_OK) return rc;
  if (n_out > 0 && out_dev == nullptr)
    QUIC_CUDA(cudaMemcpyAsync(host_out, dev_out, sizeof(int32_t) * n_out, cudaMemcpyDeviceToHost, st));
  if (status_dev == nullptr)
    QUIC_CUDA(cudaMemcpyAsync(host_status, static_cast<const unsigned char*>(sync) + 4, 4, cudaMemcpyDeviceToHost, st));
  QUIC_CUDA(cudaStreamSynchronize(st));
  if (*host_status != 0) {
    int32_t ignored = 0;
    const int rc2 = clear_sync(sync, st, QUIC_OK, &ignored, 0);
    if (rc2 != QUIC_OK) return rc2;
    return fail(QUIC_E_TIMEOUT, "decode_persist: a bounded wait inside the kernel gave up; the tokens of this call are invalid");
  }
  return QUIC_OK;
}
