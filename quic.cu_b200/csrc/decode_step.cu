// Host side of the fused decode step: carves the scratch arena, chains the
// kernels of 24 layers + lm_head with programmatic dependent launch, and can
// capture several consecutive steps into one CUDA graph.
//
// One step replaces Engine.step + QUICForCausalLM.forward(seq_len == 1) of the
// reference (src/engine.py:78-107, src/model.py:272-303).  Token ids, positions
// and the row -> slot map live in device memory, so a captured graph is valid
// for any position and consecutive steps need no host round trip.
#include <cstdio>
#include <new>

#include "decode_kernels.cuh"

namespace quic {
namespace {

inline int64_t align256(int64_t v) { return (v + 255) / 256 * 256; }

struct Arena {
  int64_t lm_counter, xres, qbuf, attn_out, act, partial, best_val, best_idx, total;
  int64_t xn, qkv, gu, act16, tcws;
};

int64_t tc_workspace_bytes(int batch) {
  int64_t w = w4a16_gemm_tc_workspace(batch, kQkvN, kHidden);
  const int64_t o = w4a16_gemm_tc_workspace(batch, kHidden, kHidden);
  const int64_t g = w4a16_gemm_tc_workspace(batch, 2 * kInter, kHidden);
  const int64_t d = w4a16_gemm_tc_workspace(batch, kHidden, kInter);
  w = w > o ? w : o;
  w = w > g ? w : g;
  w = w > d ? w : d;
  // the dense fp16 GEMM's split-K planes (same arena slot)
  const int shapes[4][2] = {{kQkvN, kHidden}, {kHidden, kHidden}, {2 * kInter, kHidden}, {kHidden, kInter}};
  for (const auto& s : shapes) {
    const int64_t f = gemm_f16_tc_workspace(batch, s[0], s[1]);
    w = w > f ? w : f;
  }
  return w;
}

// Rows that the chain of rows_chain.cu serves (from g_tensor_min_batch, un-quantised from kF16ChainMaxRows + 1 rows):
// one tile of 128 on the M side of its MMAs.
constexpr int kRowsChainMaxRows = 128;

// What the forms that a batch can take ask for.  The regions that must start zeroed (arrival counters) come first.
Arena carve(int batch, int vocab) {
  Arena a;
  int64_t off = 0;
  a.lm_counter = off;  // arrival counter, then the lm_head's per-row maxima (up to 128 rows)
  off += 256 + 128 * 8;
  a.xres = off;
  off += align256((int64_t)2 * batch * kHidden * 2);
  a.qbuf = off;
  off += align256((int64_t)batch * kHidden * 2);
  a.attn_out = off;
  off += align256((int64_t)batch * kHidden * 2);
  const bool few = batch <= kMmaChainMaxRows, gemms = batch > kRowsChainMaxRows;
  a.act = off;  // partial sums of gate|up, or sums of squares: of the mma.sync chain, of the rows chain
  off += align256((int64_t)batch * (few ? 4 * kInter * 4 : 2 * kRowsSsq * 4));
  a.partial = off;
  if (few) off += align256((int64_t)kDownSplits * batch * kHidden * 4);
  int grid = lm_head_grid(vocab);
  if (lm_head_tc_supported(batch, vocab) && lm_head_tc_tiles(vocab) > grid) grid = lm_head_tc_tiles(vocab);
  a.best_val = off;
  off += align256((int64_t)batch * grid * 4);
  a.best_idx = off;
  off += align256((int64_t)batch * grid * 4);
  a.xn = a.qkv = a.gu = a.act16 = a.tcws = off;
  if (batch >= 2) {  // the mma.sync and rows chains may be selected from batch 2 upwards
    a.xn = off;
    off += align256((int64_t)batch * kHidden * 2);
    a.act16 = off;
    off += align256((int64_t)batch * kInter * 2);
  }
  if (gemms) {
    a.qkv = off;
    off += align256((int64_t)batch * kQkvN * 2);
    a.gu = off;
    off += align256((int64_t)batch * 2 * kInter * 2);
    a.tcws = off;
    off += align256(16384 + tc_workspace_bytes(batch));
  }
  a.total = off;
  return a;
}

int check(const quic_model_t* m, const quic_decode_t* d) {
  QUIC_REQUIRE(m && d, QUIC_E_ARG, "decode_step: null argument");
  QUIC_REQUIRE(m->n_layers >= 1 && m->layers, QUIC_E_ARG, "decode_step: no layers");
  QUIC_REQUIRE(m->vocab >= 2 && m->vocab % 2 == 0, QUIC_E_SHAPE, "decode_step: vocab must be even");
  QUIC_REQUIRE(m->embed && m->final_norm && m->rope_cos && m->rope_sin && m->max_pos >= 1,
               QUIC_E_ARG, "decode_step: missing model tensor");
  QUIC_REQUIRE(d->kv && d->tok && d->pos && d->rows && d->scratch, QUIC_E_ARG,
               "decode_step: missing state tensor");
  QUIC_REQUIRE(d->batch >= 1 && d->batch <= 8 * 65535 && d->n_slots >= 1 && d->s_max >= 1,
               QUIC_E_SHAPE, "decode_step: bad batch / cache geometry");
  QUIC_REQUIRE(d->out_tokens == nullptr || (d->ring >= 1 && d->step_counter != nullptr),
               QUIC_E_ARG, "decode_step: out_tokens needs ring >= 1 and a step counter");
  for (int l = 0; l < m->n_layers; ++l) {
    const quic_layer_t& L = m->layers[l];
    QUIC_REQUIRE(L.qkv.n == kQkvN && L.qkv.k == kHidden && L.o.n == kHidden && L.o.k == kHidden &&
                     L.gate_up.n == 2 * kInter && L.gate_up.k == kHidden && L.down.n == kHidden &&
                     L.down.k == kInter,
                 QUIC_E_SHAPE, "decode_step: layer shapes are not Qwen2.5-0.5B's");
    const bool packed = L.qkv.qw && L.o.qw && L.gate_up.qw && L.down.qw;
    const bool dense = L.qkv.w16 && L.o.w16 && L.gate_up.w16 && L.down.w16;
    QUIC_REQUIRE((packed || dense) && L.ln1 && L.ln2, QUIC_E_ARG, "decode_step: missing layer tensor");
    QUIC_REQUIRE(dense == (m->layers[0].qkv.w16 != nullptr), QUIC_E_ARG,
                 "decode_step: packed and dense layers cannot be mixed");
  }
  return QUIC_OK;
}


int enqueue_step_batched(const quic_model_t* m, const quic_decode_t* d, cudaStream_t st, bool chain_head);
int enqueue_step_rows16(const quic_model_t* m, const quic_decode_t* d, cudaStream_t st, bool chain_head);

// Smallest batch that takes the tensor-core (tcgen05) step (quic_set_tensor_min_batch): 2..17,
// and smallest batch that takes the mma.sync chain (quic_set_mma_chain_min_batch): 2..17.
// Below both, the rows run the GEMV chain (FMA; its cost grows with every row, measured 352,
// 491 and 683 us per step at 1, 2 and 3 rows against 565 and 580 us of the mma.sync chain).
// (us per step of the rows chain / the mma.sync chain: 8 rows of 512 tokens 683 / 646, 12 694 / 709, 15 700 / 747, 16 698 / 764;
// of 3000 tokens 8 rows 810 / 727, 12 780 / 858, 16 792 / 915.  Up to 2560 tokens the persistent kernel serves these rows.)
int g_tensor_min_batch = kMmaChainMaxRows;
int g_mma_chain_min_batch = 3;

int enqueue_step_f16(const quic_model_t* m, const quic_decode_t* d, cudaStream_t st, bool chain_head);
int enqueue_step_batched_f16(const quic_model_t* m, const quic_decode_t* d, cudaStream_t st, bool chain_head);

int enqueue_step_rows(const quic_model_t* m, const quic_decode_t* d, cudaStream_t st, bool chain_head);

// Which attention kernel a step takes.
//   cta     CTAs of 512 tokens, their tiles requested before the dependency wait, clusters beyond: up to 20 rows while the CTAs have
//           an SM each (us per step, cta / flow: 1 x 2100 362 / 395, 5 x 3000 609 / 681, 16 x 1500 718 / 773).
//   stream  one CTA per (row, KV head) with a deep ring (17 rows of 200..1500 tokens: 791 cta, 865 streamed; 24: 963, 872).
//   flow    every row cut into up to eight equal ranges, a cluster each: where the others leave SMs idle or a row is one
//           CTA's walk.  Instead of cta: 16 x 3000 857 -> 814, 20 x 3500 1048 -> 841; instead of stream, from three ranges and 1536 tokens:
//           24 x 2000 871 -> 812, 24 x 5000 1234 -> 1005, 37 x 3000 1010 -> 974 (24 x 900 would be 709 -> 734); and
//           instead of splits merged in global memory, beyond 4096 tokens: 1 x 4200 462 -> 424, 5 x 7000 1140 -> 742, 15 x 8000 1624 -> 1008.
enum AttnForm { kAttnCta = QUIC_ATTN_CTA, kAttnStream = QUIC_ATTN_STREAM, kAttnFlow = QUIC_ATTN_FLOW };
constexpr int kCtaAttnMaxRows = 20, kStreamAnyCtxRows = 48, kFlowMinCtx = 1536;
AttnForm attention_form(int batch, int ctx) {
  const int parts = attn_cta_splits(ctx);
  if (batch <= kCtaAttnMaxRows)
    return parts <= kAttnCtaMaxSplits && (kKvHeads * batch * parts <= 148 || attn_flow_splits(batch, ctx) < 3) ? kAttnCta : kAttnFlow;
  return batch < kStreamAnyCtxRows && ctx > kFlowMinCtx && attn_flow_splits(batch, ctx) >= 3 ? kAttnFlow : kAttnStream;
}

static_assert(kRowsChainMaxRows + 1 >= kStreamAnyCtxRows, "steps that leave the QKV linear to the attention take the form that finishes it");

// a: queries, cache, rows, positions, scale, output.  `fuse` (form stream only): the kernel finishes the QKV linear itself.
int launch_attention(AttnArgs a, const quic_decode_t* d, int ctx, cudaStream_t st, const QkvFinish* fuse = nullptr) {
  const AttnForm form = attention_form(d->batch, ctx);
  QUIC_REQUIRE(fuse == nullptr || form == kAttnStream, QUIC_E_ARG, "decode_step: only the streaming attention finishes the QKV linear");
  a.prefetch = d->step_counter != nullptr ? 1 : 0;
  if (form == kAttnCta) {
    a.splits = attn_cta_splits(ctx);
    a.chunk = 512;
    QUIC_CUDA(launch_attn_cta(a, d->batch, st, true));
    return QUIC_OK;
  }
  if (form == kAttnStream) {
    a.splits = 1;
    a.chunk = ctx;
    return launch_attn_stream(a, fuse, d->batch, d->n_slots, d->s_max, tc_status_words(), st, true);
  }
  a.splits = attn_flow_splits(d->batch, ctx);
  return launch_attn_flow(a, d->batch, tc_status_words(), st, d->n_slots);
}

int enqueue_step(const quic_model_t* m, const quic_decode_t* d, cudaStream_t st, bool chain_head) {
  const int B = d->batch;
  if (B <= kRowsChainMaxRows && B > (m->layers[0].qkv.w16 != nullptr ? kF16ChainMaxRows : g_tensor_min_batch - 1))
    return enqueue_step_rows(m, d, st, chain_head);
  if (m->layers[0].qkv.w16 != nullptr)  // dense fp16 weights
    return B <= kF16ChainMaxRows ? enqueue_step_f16(m, d, st, chain_head) : enqueue_step_batched_f16(m, d, st, chain_head);
  if (B >= g_tensor_min_batch) return enqueue_step_batched(m, d, st, chain_head);
  if (B >= g_mma_chain_min_batch) return enqueue_step_rows16(m, d, st, chain_head);
  const Arena ar = carve(B, m->vocab);
  char* base = static_cast<char*>(d->scratch);
  half* xres[2] = {reinterpret_cast<half*>(base + ar.xres),
                   reinterpret_cast<half*>(base + ar.xres) + (size_t)B * kHidden};
  half* qbuf = reinterpret_cast<half*>(base + ar.qbuf);
  half* attn_out = reinterpret_cast<half*>(base + ar.attn_out);
  float* gu_part = reinterpret_cast<float*>(base + ar.act);
  float* partial = reinterpret_cast<float*>(base + ar.partial);

  const size_t slot_stride = (size_t)kKvHeads * d->s_max * kHeadDim;  // one slot, K or V
  const size_t kv_plane = (size_t)d->n_slots * slot_stride;           // K (or V) of a layer
  int ctx = d->ctx_hint > 0 ? d->ctx_hint : d->s_max;
  if (ctx > d->s_max) ctx = d->s_max;

  RowState rs;
  rs.rows = d->rows;
  rs.tok = d->tok;
  rs.pos = d->pos;
  rs.batch = B;

  for (int l = 0; l < m->n_layers; ++l) {
    const quic_layer_t& L = m->layers[l];
    half* kc = static_cast<half*>(d->kv) + (size_t)(2 * l) * kv_plane;
    half* vc = kc + kv_plane;

    QkvArgs qa = {};
    qa.w = L.qkv;
    qa.ln = (const half*)L.ln1;
    qa.embed = (const half*)m->embed;
    qa.xres_in = xres[1];
    qa.xres_out = xres[0];
    qa.partial = partial;
    qa.rs = rs;
    qa.eps = m->eps;
    qa.first_layer = (l == 0);
    qa.vocab = m->vocab;
    qa.cos_t = (const half*)m->rope_cos;
    qa.sin_t = (const half*)m->rope_sin;
    qa.max_pos = m->max_pos;
    qa.qbuf = qbuf;
    qa.kcache = kc;
    qa.vcache = vc;
    qa.s_max = d->s_max;
    // The first kernel of a sequence starts only after everything enqueued before it has
    // completed (no programmatic overlap), so later kernels of the chain may read the cache
    // before their own dependency wait.
    QUIC_CUDA(launch_qkv(qa, st, !(chain_head && l == 0)));

    AttnArgs aa = {};
    aa.q = qbuf;
    aa.k = kc;
    aa.v = vc;
    aa.stride_b = (int64_t)slot_stride;
    aa.stride_h = (int64_t)d->s_max * kHeadDim;
    aa.rows = d->rows;
    aa.pos = d->pos;
    aa.s_cap = ctx;
    aa.scale = 0.125f;  // 64^-0.5, src/model.py:129
    aa.out = attn_out;
    aa.epoch = d->step_counter;
    const int rc = launch_attention(aa, d, ctx, st);
    if (rc != QUIC_OK) return rc;

    OProjArgs oa = {};
    oa.w = L.o;
    oa.attn = attn_out;
    oa.xres_in = xres[0];
    oa.xres_out = xres[1];
    oa.batch = B;
    QUIC_CUDA(launch_oproj(oa, st, true));

    GateUpArgs ga = {};
    ga.w = L.gate_up;
    ga.ln = (const half*)L.ln2;
    ga.xres = xres[1];
    ga.gu_part = gu_part;
    ga.batch = B;
    ga.eps = m->eps;
    QUIC_CUDA(launch_gateup(ga, st, true));

    DownArgs da = {};
    da.w = L.down;
    da.gu_part = gu_part;
    da.partial = partial;
    da.batch = B;
    QUIC_CUDA(launch_down(da, st, true));
  }

  LmHeadArgs la = {};
  la.embed = (const half*)m->embed;
  la.ln = (const half*)m->final_norm;
  la.xres_in = xres[1];
  la.partial = partial;
  la.batch = B;
  la.vocab = m->vocab;
  la.eps = m->eps;
  la.logits = (half*)d->logits;
  la.best_val = reinterpret_cast<float*>(base + ar.best_val);
  la.best_idx = reinterpret_cast<int32_t*>(base + ar.best_idx);
  la.counter = reinterpret_cast<int32_t*>(base + ar.lm_counter);
  la.keys = reinterpret_cast<unsigned long long*>(base + ar.lm_counter + 256);
  la.rows = d->rows;
  la.tok = d->tok;
  la.pos = d->pos;
  la.out_tokens = d->out_tokens;
  la.n_slots = d->n_slots;
  la.ring = d->ring > 0 ? d->ring : 1;
  la.step_counter = d->step_counter;
  QUIC_CUDA(launch_lm_head(la, lm_head_grid(m->vocab), st, true));
  return QUIC_OK;
}

// 2..16 rows: five launches per layer as for one row, every linear on mma.sync with the rows on
// the M side; each kernel writes a finished fp16 tensor (decode_layers_mma.cu).
int enqueue_step_rows16(const quic_model_t* m, const quic_decode_t* d, cudaStream_t st, bool chain_head) {
  const int B = d->batch;
  const Arena ar = carve(B, m->vocab);
  char* base = static_cast<char*>(d->scratch);
  half* xa = reinterpret_cast<half*>(base + ar.xres);  // residual stream entering a layer
  half* xb = xa + (size_t)B * kHidden;                  // after the attention block
  half* qbuf = reinterpret_cast<half*>(base + ar.qbuf);
  half* attn_out = reinterpret_cast<half*>(base + ar.attn_out);
  half* act = reinterpret_cast<half*>(base + ar.act16);
  half* xn = reinterpret_cast<half*>(base + ar.xn);
  // per-tile sums of squares of the two residual streams ([B][32] fp32 each), the down
  // kernel's K-split planes and its arrival counters (in the arena's zeroed head)
  float* ssq_a = reinterpret_cast<float*>(base + ar.act);
  float* ssq_b = ssq_a + kMmaChainMaxRows * 32;
  float* partial = reinterpret_cast<float*>(base + ar.partial);
  int32_t* down_counters = reinterpret_cast<int32_t*>(base + ar.lm_counter + 128);
  const size_t slot_stride = (size_t)kKvHeads * d->s_max * kHeadDim;
  const size_t kv_plane = (size_t)d->n_slots * slot_stride;
  int ctx = d->ctx_hint > 0 ? d->ctx_hint : d->s_max;
  if (ctx > d->s_max) ctx = d->s_max;
  RowState rs;
  rs.rows = d->rows;
  rs.tok = d->tok;
  rs.pos = d->pos;
  rs.batch = B;
  const half* embed = (const half*)m->embed;

  for (int l = 0; l < m->n_layers; ++l) {
    const quic_layer_t& L = m->layers[l];
    half* kc = static_cast<half*>(d->kv) + (size_t)(2 * l) * kv_plane;
    half* vc = kc + kv_plane;
    // (the head of a sequence starts only after everything enqueued before it has completed)
    QUIC_CUDA(launch_qkv_mma(L.qkv, (const half*)L.ln1, embed, xa, ssq_a, xa, rs, m->eps, l == 0, m->vocab,
                             (const half*)m->rope_cos, (const half*)m->rope_sin, m->max_pos, qbuf, kc, vc, d->s_max,
                             st, !(chain_head && l == 0)));
    AttnArgs aa = {};
    aa.q = qbuf;
    aa.k = kc;
    aa.v = vc;
    aa.stride_b = (int64_t)slot_stride;
    aa.stride_h = (int64_t)d->s_max * kHeadDim;
    aa.rows = d->rows;
    aa.pos = d->pos;
    aa.s_cap = ctx;
    aa.scale = 0.125f;
    aa.out = attn_out;
    aa.epoch = d->step_counter;
    const int rc = launch_attention(aa, d, ctx, st);
    if (rc != QUIC_OK) return rc;
    QUIC_CUDA(launch_oproj_mma(L.o, attn_out, xa, xb, ssq_b, B, st));
    QUIC_CUDA(launch_gateup_mma(L.gate_up, (const half*)L.ln2, xb, ssq_b, act, B, m->eps, st));
    QUIC_CUDA(launch_down_mma(L.down, act, xb, xa, ssq_a, partial, down_counters, B, st));
  }
  LmHeadArgs la = {};
  la.embed = embed;
  la.batch = B;
  la.vocab = m->vocab;
  la.eps = m->eps;
  la.logits = (half*)d->logits;
  la.best_val = reinterpret_cast<float*>(base + ar.best_val);
  la.best_idx = reinterpret_cast<int32_t*>(base + ar.best_idx);
  la.counter = reinterpret_cast<int32_t*>(base + ar.lm_counter);
  la.keys = reinterpret_cast<unsigned long long*>(base + ar.lm_counter + 256);
  la.rows = d->rows;
  la.tok = d->tok;
  la.pos = d->pos;
  la.out_tokens = d->out_tokens;
  la.n_slots = d->n_slots;
  la.ring = d->ring > 0 ? d->ring : 1;
  la.step_counter = d->step_counter;
  if (B > 2 && lm_head_tc_supported(B, m->vocab)) {
    QUIC_CUDA(launch_rmsnorm(xa, nullptr, (const half*)m->final_norm, m->eps, xn, nullptr, B, st));
    la.x_normed = xn;
    return launch_lm_head_tc(la, st);
  }
  // up to two rows (from three the tensor kernel is ahead, 77 -> 50 us): the GEMV form, final norm fused, one launch
  la.ln = (const half*)m->final_norm;
  la.xres_in = xa;
  QUIC_CUDA(launch_lm_head(la, lm_head_grid(m->vocab), st, true));
  return QUIC_OK;
}

// More than kRowsChainMaxRows rows: every linear is the tcgen05 GEMM, norms are
// separate small kernels (at these sizes each kernel does microseconds of real work, so
// the launch chain is no longer what bounds the step).
// `fuse`: the attention kernel finishes the QKV linear itself (the streaming form, which every step of these takes).
int enqueue_attention(const quic_decode_t* d, int ctx, half* qbuf, half* kc, half* vc, half* attn_out, cudaStream_t st,
                      const QkvFinish* fuse = nullptr);

int enqueue_step_batched(const quic_model_t* m, const quic_decode_t* d, cudaStream_t st, bool chain_head) {
  const int B = d->batch;
  const Arena ar = carve(B, m->vocab);
  char* base = static_cast<char*>(d->scratch);
  half* h = reinterpret_cast<half*>(base + ar.xres);        // residual stream
  half* qbuf = reinterpret_cast<half*>(base + ar.qbuf);
  half* attn_out = reinterpret_cast<half*>(base + ar.attn_out);
  half* xn = reinterpret_cast<half*>(base + ar.xn);
  half* act = reinterpret_cast<half*>(base + ar.act16);
  float* ws = reinterpret_cast<float*>(base + ar.tcws);
  const size_t slot_stride = (size_t)kKvHeads * d->s_max * kHeadDim;
  const size_t kv_plane = (size_t)d->n_slots * slot_stride;
  int ctx = d->ctx_hint > 0 ? d->ctx_hint : d->s_max;
  if (ctx > d->s_max) ctx = d->s_max;
  const half* embed = (const half*)m->embed;

  // (the head of a sequence starts only after everything enqueued before it has completed)
  QUIC_CUDA(launch_embed_rows(embed, d->rows, d->tok, m->vocab, h, B, st, !chain_head));
  QUIC_CUDA(launch_rmsnorm(h, nullptr, (const half*)m->layers[0].ln1, m->eps, xn, nullptr, B, st));
  for (int l = 0; l < m->n_layers; ++l) {
    const quic_layer_t& L = m->layers[l];
    half* kc = static_cast<half*>(d->kv) + (size_t)(2 * l) * kv_plane;
    half* vc = kc + kv_plane;
    // linears whose consumer is a small kernel leave split-K partials for it to reduce
    int sp = 1;
    const float* part = ws + 4096;
    int rc = w4a16_gemm_tc(xn, L.qkv, nullptr, B, ws, st, &sp);
    if (rc != QUIC_OK) return rc;
    // the attention CTAs sum the partial sums, rotate and append themselves: one launch less
    // (64 rows of 512 tokens: 934 -> 883 us per step, same bits)
    QkvFinish fin = {part, sp, (const half*)L.qkv.bias, nullptr, (const half*)m->rope_cos, (const half*)m->rope_sin,
                     m->max_pos};
    rc = enqueue_attention(d, ctx, qbuf, kc, vc, attn_out, st, &fin);
    if (rc != QUIC_OK) return rc;
    rc = w4a16_gemm_tc(attn_out, L.o, nullptr, B, ws, st, &sp);
    if (rc != QUIC_OK) return rc;
    QUIC_CUDA(launch_rmsnorm_part(part, sp, h, (const half*)L.ln2, m->eps, xn, h, B, st));
    rc = w4a16_gemm_tc_swiglu(xn, L.gate_up, act, B, st);  // SwiGLU in the GEMM's epilogue
    if (rc != QUIC_OK) return rc;
    rc = w4a16_gemm_tc(act, L.down, nullptr, B, ws, st, &sp);
    if (rc != QUIC_OK) return rc;
    const half* next_ln = (l + 1 < m->n_layers) ? (const half*)m->layers[l + 1].ln1 : (const half*)m->final_norm;
    QUIC_CUDA(launch_rmsnorm_part(part, sp, h, next_ln, m->eps, xn, h, B, st));
  }
  LmHeadArgs la = {};
  la.embed = embed;
  la.x_normed = xn;
  la.batch = B;
  la.vocab = m->vocab;
  la.eps = m->eps;
  la.logits = (half*)d->logits;
  la.best_val = reinterpret_cast<float*>(base + ar.best_val);
  la.best_idx = reinterpret_cast<int32_t*>(base + ar.best_idx);
  la.counter = reinterpret_cast<int32_t*>(base + ar.lm_counter);
  la.keys = reinterpret_cast<unsigned long long*>(base + ar.lm_counter + 256);
  la.rows = d->rows;
  la.tok = d->tok;
  la.pos = d->pos;
  la.out_tokens = d->out_tokens;
  la.n_slots = d->n_slots;
  la.ring = d->ring > 0 ? d->ring : 1;
  la.step_counter = d->step_counter;
  if (lm_head_tc_supported(B, m->vocab)) return launch_lm_head_tc(la, st);
  la.x_normed = xn;
  QUIC_CUDA(launch_lm_head(la, lm_head_grid(m->vocab), st, false));
  return QUIC_OK;
}

// Attention of a decode step with finished fp16 output.
int enqueue_attention(const quic_decode_t* d, int ctx, half* qbuf, half* kc, half* vc, half* attn_out, cudaStream_t st,
                      const QkvFinish* fuse) {
  AttnArgs aa = {};
  aa.q = qbuf;
  aa.k = kc;
  aa.v = vc;
  aa.stride_b = (int64_t)kKvHeads * d->s_max * kHeadDim;
  aa.stride_h = (int64_t)d->s_max * kHeadDim;
  aa.rows = d->rows;
  aa.pos = d->pos;
  aa.s_cap = ctx;
  aa.scale = 0.125f;  // 64^-0.5, src/model.py:129
  aa.out = attn_out;
  aa.epoch = d->step_counter;
  return launch_attention(aa, d, ctx, st, fuse);
}

LmHeadArgs lm_head_args(const quic_model_t* m, const quic_decode_t* d, const Arena& ar);

// 16..128 rows, un-quantised from 3: five launches a layer (rows_chain.cu).
int enqueue_step_rows(const quic_model_t* m, const quic_decode_t* d, cudaStream_t st, bool chain_head) {
  const int B = d->batch;
  const Arena ar = carve(B, m->vocab);
  char* base = static_cast<char*>(d->scratch);
  half* h = reinterpret_cast<half*>(base + ar.xres);  // residual stream
  half* qbuf = reinterpret_cast<half*>(base + ar.qbuf);
  half* attn_out = reinterpret_cast<half*>(base + ar.attn_out);
  half* xn = reinterpret_cast<half*>(base + ar.xn);
  half* act = reinterpret_cast<half*>(base + ar.act16);
  float* ssq = reinterpret_cast<float*>(base + ar.act);  // [B][kRowsSsq], of h after the attention, after the layer
  float* const ssq_mid = ssq;
  float* const ssq_end = ssq + (size_t)B * kRowsSsq;
  const size_t kv_plane = (size_t)d->n_slots * kKvHeads * d->s_max * kHeadDim;
  int ctx = d->ctx_hint > 0 ? d->ctx_hint : d->s_max;
  if (ctx > d->s_max) ctx = d->s_max;
  RowsArgs a = {};
  a.rows = B;
  a.eps = m->eps;
  a.slots = d->rows;
  a.pos = d->pos;
  a.cos_t = (const half*)m->rope_cos;
  a.sin_t = (const half*)m->rope_sin;
  a.max_pos = m->max_pos;
  a.s_max = d->s_max;
  a.n_slots = d->n_slots;
  a.res = h;
  // (the head of a sequence starts only after everything enqueued before it has completed)
  QUIC_CUDA(launch_embed_ssq((const half*)m->embed, d->rows, d->tok, m->vocab, h, ssq_end, B, st, !chain_head));
  int rc;
  for (int l = 0; l < m->n_layers; ++l) {
    const quic_layer_t& L = m->layers[l];
    a.kcache = static_cast<half*>(d->kv) + (size_t)(2 * l) * kv_plane;
    a.vcache = a.kcache + kv_plane;
    a.w = L.qkv;
    a.y = qbuf;
    a.ln = (const half*)L.ln1;
    a.ssq_in = ssq_end;
    a.n_ssq = l == 0 ? 1 : kRowsSsq;
    rows_next(&a, &L.o);  // a launch brings the next linear's weights into L2
    if ((rc = rows_qkv(h, a, st)) != QUIC_OK) return rc;
    if ((rc = enqueue_attention(d, ctx, qbuf, a.kcache, a.vcache, attn_out, st)) != QUIC_OK) return rc;
    a.w = L.o;
    a.y = h;
    a.ssq_out = ssq_mid;
    rows_next(&a, &L.gate_up);
    if ((rc = rows_out(attn_out, a, st)) != QUIC_OK) return rc;
    a.w = L.gate_up;
    a.y = act;
    a.ln = (const half*)L.ln2;
    a.ssq_in = ssq_mid;
    a.n_ssq = kRowsSsq;
    rows_next(&a, &L.down);
    if ((rc = rows_swiglu(h, a, st)) != QUIC_OK) return rc;
    a.w = L.down;
    a.y = h;
    a.ssq_out = ssq_end;
    rows_next(&a, l + 1 < m->n_layers ? &m->layers[l + 1].qkv : nullptr);
    if ((rc = rows_down(act, a, st)) != QUIC_OK) return rc;
  }
  QUIC_CUDA(launch_rmsnorm(h, nullptr, (const half*)m->final_norm, m->eps, xn, nullptr, B, st));
  LmHeadArgs la = lm_head_args(m, d, ar);
  la.x_normed = xn;
  if (lm_head_tc_supported(B, m->vocab)) return launch_lm_head_tc(la, st);
  QUIC_CUDA(launch_lm_head(la, lm_head_grid(m->vocab), st, false));
  return QUIC_OK;
}

LmHeadArgs lm_head_args(const quic_model_t* m, const quic_decode_t* d, const Arena& ar) {
  char* base = static_cast<char*>(d->scratch);
  LmHeadArgs la = {};
  la.embed = (const half*)m->embed;
  la.batch = d->batch;
  la.vocab = m->vocab;
  la.eps = m->eps;
  la.logits = (half*)d->logits;
  la.best_val = reinterpret_cast<float*>(base + ar.best_val);
  la.best_idx = reinterpret_cast<int32_t*>(base + ar.best_idx);
  la.counter = reinterpret_cast<int32_t*>(base + ar.lm_counter);
  la.keys = reinterpret_cast<unsigned long long*>(base + ar.lm_counter + 256);
  la.rows = d->rows;
  la.tok = d->tok;
  la.pos = d->pos;
  la.out_tokens = d->out_tokens;
  la.n_slots = d->n_slots;
  la.ring = d->ring > 0 ? d->ring : 1;
  la.step_counter = d->step_counter;
  return la;
}

// Dense fp16 weights, one or two rows: five kernels per layer (decode_layers_f16.cu) and the GEMV
// lm_head with the final norm fused.
int enqueue_step_f16(const quic_model_t* m, const quic_decode_t* d, cudaStream_t st, bool chain_head) {
  const int B = d->batch;
  const Arena ar = carve(B, m->vocab);
  char* base = static_cast<char*>(d->scratch);
  half* xa = reinterpret_cast<half*>(base + ar.xres);  // residual stream entering a layer
  half* xb = xa + (size_t)B * kHidden;                  // after the attention block
  half* qbuf = reinterpret_cast<half*>(base + ar.qbuf);
  half* attn_out = reinterpret_cast<half*>(base + ar.attn_out);
  half* act = reinterpret_cast<half*>(base + ar.act);
  const size_t kv_plane = (size_t)d->n_slots * kKvHeads * d->s_max * kHeadDim;
  int ctx = d->ctx_hint > 0 ? d->ctx_hint : d->s_max;
  if (ctx > d->s_max) ctx = d->s_max;
  RowState rs;
  rs.rows = d->rows;
  rs.tok = d->tok;
  rs.pos = d->pos;
  rs.batch = B;
  for (int l = 0; l < m->n_layers; ++l) {
    const quic_layer_t& L = m->layers[l];
    half* kc = static_cast<half*>(d->kv) + (size_t)(2 * l) * kv_plane;
    half* vc = kc + kv_plane;
    QUIC_CUDA(launch_qkv_f16(L.qkv, (const half*)L.ln1, (const half*)m->embed, xa, xa, rs, m->eps, l == 0, m->vocab,
                             (const half*)m->rope_cos, (const half*)m->rope_sin, m->max_pos, qbuf, kc, vc, d->s_max,
                             d->n_slots, st, !(chain_head && l == 0)));
    int rc = enqueue_attention(d, ctx, qbuf, kc, vc, attn_out, st);
    if (rc != QUIC_OK) return rc;
    QUIC_CUDA(launch_residual_f16(L.o, attn_out, xa, xb, B, st));
    QUIC_CUDA(launch_gateup_f16(L.gate_up, (const half*)L.ln2, xb, act, B, m->eps, st));
    QUIC_CUDA(launch_residual_f16(L.down, act, xb, xa, B, st));
  }
  LmHeadArgs la = lm_head_args(m, d, ar);
  la.ln = (const half*)m->final_norm;
  la.xres_in = xa;
  QUIC_CUDA(launch_lm_head(la, lm_head_grid(m->vocab), st, true));
  return QUIC_OK;
}

// Dense fp16 weights, more rows: every linear on the tcgen05 fp16 GEMM; norms, RoPE / KV append
// and SwiGLU are the small kernels of the batched W4A16 step.
int enqueue_step_batched_f16(const quic_model_t* m, const quic_decode_t* d, cudaStream_t st, bool chain_head) {
  const int B = d->batch;
  const Arena ar = carve(B, m->vocab);
  char* base = static_cast<char*>(d->scratch);
  half* h = reinterpret_cast<half*>(base + ar.xres);
  half* qbuf = reinterpret_cast<half*>(base + ar.qbuf);
  half* attn_out = reinterpret_cast<half*>(base + ar.attn_out);
  half* xn = reinterpret_cast<half*>(base + ar.xn);
  half* qkv = reinterpret_cast<half*>(base + ar.qkv);  // [B][1152]; also holds a [B][896] linear output
  half* gu = reinterpret_cast<half*>(base + ar.gu);
  half* act = reinterpret_cast<half*>(base + ar.act16);
  float* ws = reinterpret_cast<float*>(base + ar.tcws);  // split-K partials of the small GEMMs
  const size_t kv_plane = (size_t)d->n_slots * kKvHeads * d->s_max * kHeadDim;
  int ctx = d->ctx_hint > 0 ? d->ctx_hint : d->s_max;
  if (ctx > d->s_max) ctx = d->s_max;
  QUIC_CUDA(launch_embed_rows((const half*)m->embed, d->rows, d->tok, m->vocab, h, B, st, !chain_head));
  QUIC_CUDA(launch_rmsnorm(h, nullptr, (const half*)m->layers[0].ln1, m->eps, xn, nullptr, B, st));
  for (int l = 0; l < m->n_layers; ++l) {
    const quic_layer_t& L = m->layers[l];
    half* kc = static_cast<half*>(d->kv) + (size_t)(2 * l) * kv_plane;
    half* vc = kc + kv_plane;
    int rc = gemm_f16_tc(xn, (const half*)L.qkv.w16, (const half*)L.qkv.bias, qkv, B, kQkvN, kHidden, ws, st, true);
    if (rc != QUIC_OK) return rc;
    // the attention CTAs rotate and append themselves
    QkvFinish fin = {nullptr, 0, nullptr, qkv, (const half*)m->rope_cos, (const half*)m->rope_sin, m->max_pos};
    rc = enqueue_attention(d, ctx, qbuf, kc, vc, attn_out, st, &fin);
    if (rc != QUIC_OK) return rc;
    rc = gemm_f16_tc(attn_out, (const half*)L.o.w16, nullptr, qkv, B, kHidden, kHidden, ws, st, true);
    if (rc != QUIC_OK) return rc;
    QUIC_CUDA(launch_rmsnorm(qkv, h, (const half*)L.ln2, m->eps, xn, h, B, st));
    rc = gemm_f16_tc(xn, (const half*)L.gate_up.w16, nullptr, gu, B, 2 * kInter, kHidden, ws, st, true);
    if (rc != QUIC_OK) return rc;
    QUIC_CUDA(launch_swiglu_fused(gu, act, B, st));
    rc = gemm_f16_tc(act, (const half*)L.down.w16, nullptr, qkv, B, kHidden, kInter, ws, st, true);
    if (rc != QUIC_OK) return rc;
    const half* next_ln = (l + 1 < m->n_layers) ? (const half*)m->layers[l + 1].ln1 : (const half*)m->final_norm;
    QUIC_CUDA(launch_rmsnorm(qkv, h, next_ln, m->eps, xn, h, B, st));
  }
  LmHeadArgs la = lm_head_args(m, d, ar);
  la.x_normed = xn;
  if (lm_head_tc_supported(B, m->vocab)) return launch_lm_head_tc(la, st);
  QUIC_CUDA(launch_lm_head(la, lm_head_grid(m->vocab), st, false));
  return QUIC_OK;
}

struct Graph {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int32_t* words = nullptr;  // where its kernels' bounded waits report
  bool own_words = false;
};

}  // namespace
}  // namespace quic

using namespace quic;

extern "C" void quic_set_tensor_min_batch(int32_t batch) {
  g_tensor_min_batch = batch < 2 ? 2 : (batch > kMmaChainMaxRows + 1 ? kMmaChainMaxRows + 1 : batch);
}

extern "C" void quic_set_mma_chain_min_batch(int32_t batch) {
  g_mma_chain_min_batch = batch < 2 ? 2 : (batch > kMmaChainMaxRows + 1 ? kMmaChainMaxRows + 1 : batch);
}

extern "C" int32_t quic_decode_attention_form(int32_t batch, int32_t ctx) {
  return attention_form(batch < 1 ? 1 : batch, ctx < 1 ? 1 : ctx);
}

extern "C" int32_t quic_decode_pick_splits(int32_t batch, int32_t ctx) {
  if (batch < 1) batch = 1;
  if (ctx < 1) ctx = 1;
  // (no step's attention merges splits in global memory any more: the number is for callers that ask for it)
  if (ctx <= 2048) return (ctx + 63) / 64;
  const int by_len = (ctx + 127) / 128, most = batch >= g_tensor_min_batch ? 1184 / (batch * kKvHeads) : 64;
  const int s = by_len < most ? by_len : most;
  return s < 1 ? 1 : s > 64 ? 64 : s;
}

extern "C" int64_t quic_decode_scratch_bytes(int32_t batch, int32_t vocab, int32_t attn_splits) {
  if (batch < 1 || vocab < 2 || attn_splits < 1) return 0;
  return carve(batch, vocab).total;
}

extern "C" int32_t quic_decode_launch_count(const quic_model_t* m, const quic_decode_t* d) {
  if (!m) return 0;
  if (d && m->layers && d->batch <= kRowsChainMaxRows &&
      d->batch > (m->layers[0].qkv.w16 != nullptr ? kF16ChainMaxRows : g_tensor_min_batch - 1))
    return 5 * m->n_layers + 3;
  if (m->layers && m->layers[0].qkv.w16 != nullptr) {
    if (d && d->batch > kF16ChainMaxRows) return 8 * m->n_layers + 3;
    return 5 * m->n_layers + 1;
  }
  if (d && d->batch >= g_tensor_min_batch) return 7 * m->n_layers + 3;  // the streamed attention finishes the QKV linear
  if (d && d->batch >= g_mma_chain_min_batch) return 5 * m->n_layers + ((d->batch > 2 && lm_head_tc_supported(d->batch, m->vocab)) ? 2 : 1);
  return 5 * m->n_layers + 1;
}

extern "C" int quic_decode_step(const quic_model_t* m, const quic_decode_t* d, void* stream) {
  int rc = check(m, d);
  if (rc != QUIC_OK) return rc;
  return enqueue_step(m, d, (cudaStream_t)stream, true);
}

extern "C" int quic_graph_destroy(void* graph) {
  if (graph == nullptr) return QUIC_OK;
  Graph* g = static_cast<Graph*>(graph);
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  if (g->own_words) quic_error_words_free(g->words);
  delete g;
  return QUIC_OK;
}

extern "C" int quic_decode_graph_create_watch(const quic_model_t* m, const quic_decode_t* d, int32_t steps, void* stream,
                                              int32_t* error_words, void** graph_out) {
  int rc = check(m, d);
  if (rc != QUIC_OK) return rc;
  QUIC_REQUIRE(graph_out != nullptr && steps >= 1 && steps <= 4096, QUIC_E_ARG,
               "decode_graph_create: bad steps / output pointer");
  cudaStream_t st = (cudaStream_t)stream;
  QUIC_REQUIRE(st != nullptr, QUIC_E_ARG,
               "decode_graph_create: capture needs a non-default stream");
  Graph* g = new (std::nothrow) Graph();
  QUIC_REQUIRE(g != nullptr, QUIC_E_ARG, "decode_graph_create: out of host memory");
  g->own_words = error_words == nullptr;
  g->words = g->own_words ? quic_error_words_new() : error_words;
  StatusScope scope(g->words);
  if (g->words == nullptr || !scope.ok) {
    quic_graph_destroy(g);
    return fail(QUIC_E_CUDA, "decode_graph_create: no page-locked error words");
  }
  cudaError_t e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) {
    quic_graph_destroy(g);
    return fail(QUIC_E_CUDA, cudaGetErrorString(e));
  }
  for (int s = 0; s < steps && rc == QUIC_OK; ++s) rc = enqueue_step(m, d, st, s == 0);
  e = cudaStreamEndCapture(st, &g->graph);
  if (rc == QUIC_OK && e != cudaSuccess) rc = fail(QUIC_E_CUDA, cudaGetErrorString(e));
  if (rc == QUIC_OK) {
    e = cudaGraphInstantiate(&g->exec, g->graph, 0);
    if (e != cudaSuccess) rc = fail(QUIC_E_CUDA, cudaGetErrorString(e));
  }
  if (rc != QUIC_OK) {
    quic_graph_destroy(g);
    cudaGetLastError();
    return rc;
  }
  *graph_out = g;
  return QUIC_OK;
}

extern "C" int quic_decode_graph_create(const quic_model_t* m, const quic_decode_t* d,
                                        int32_t steps, void* stream, void** graph_out) {
  return quic_decode_graph_create_watch(m, d, steps, stream, nullptr, graph_out);
}

extern "C" int quic_graph_launch(void* graph, void* stream) {
  QUIC_REQUIRE(graph != nullptr, QUIC_E_ARG, "graph_launch: null graph");
  Graph* g = static_cast<Graph*>(graph);
  QUIC_CUDA(cudaGraphLaunch(g->exec, (cudaStream_t)stream));
  return QUIC_OK;
}

extern "C" int quic_graph_run_host(void* graph, void* stream, const int32_t* host_in, int32_t* dev_in,
                                   int32_t n_in, const int32_t* dev_out, int32_t* host_out, int32_t n_out) {
  QUIC_REQUIRE(graph != nullptr, QUIC_E_ARG, "graph_run_host: null graph");
  QUIC_REQUIRE(n_in >= 0 && n_out >= 0, QUIC_E_ARG, "graph_run_host: negative count");
  QUIC_REQUIRE(n_in == 0 || (host_in != nullptr && dev_in != nullptr), QUIC_E_ARG,
               "graph_run_host: null input buffer");
  QUIC_REQUIRE(n_out == 0 || (host_out != nullptr && dev_out != nullptr), QUIC_E_ARG,
               "graph_run_host: null output buffer");
  Graph* g = static_cast<Graph*>(graph);
  cudaStream_t st = (cudaStream_t)stream;
  if (n_in > 0) QUIC_CUDA(cudaMemcpyAsync(dev_in, host_in, sizeof(int32_t) * n_in, cudaMemcpyHostToDevice, st));
  QUIC_CUDA(cudaGraphLaunch(g->exec, st));
  if (n_out > 0)
    QUIC_CUDA(cudaMemcpyAsync(host_out, dev_out, sizeof(int32_t) * n_out, cudaMemcpyDeviceToHost, st));
  QUIC_CUDA(cudaStreamSynchronize(st));
  const int32_t word = error_words_take(g->words);
  if (word != 0) {
    char msg[160];
    snprintf(msg, sizeof(msg),
             "decode: a bounded wait of a tensor-core kernel gave up (status 0x%x); the tokens of this call are invalid",
             (unsigned)word);
    return fail(QUIC_E_TIMEOUT, msg);
  }
  return QUIC_OK;
}
