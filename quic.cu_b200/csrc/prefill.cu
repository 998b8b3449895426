// Fused prefill: every admitted prompt through the whole model in one library call (no host
// framework ops between the kernels).  It chains the stand-alone entry points of this
// library -- W4A16 linear, RMSNorm (+ residual), quic_qkv_rope_append, quic_attn_prefill,
// quic_swiglu_fused, tied lm_head + argmax -- over activations in a caller-provided scratch
// arena, plus three small kernels of its own (embedding gather, last-row gather, slot state).
#include "decode_kernels.cuh"

namespace quic {
namespace {

// Rows from which a layer's linears run on SM pairs over fp16 weights (gemm_pair.cu).  Packed weights are
// unpacked for it once per call and layer, 8 us: 1 x 600 tokens 1848 -> 2196 us, 1 x 768 2190 -> 2179,
// 1 x 1000 2728 -> 2515, 16 x 2048 42.0 -> 33.1 ms.  Dense weights are read as they are: 1 x 130 tokens 1578 -> 1690 us,
// 1 x 200 1768 -> 1747, 1 x 500 2426 -> 2041, 2 x 1024 5826 -> 3196.
constexpr int kPairRows = 768, kDensePairRows = 192;
// Rows up to which a layer runs on the chain of rows_chain.cu: one tile of 128 rows of packed weights (us, GEMMs / chain: 2 rows
// 746 / 708, 40 867 / 747, 87 1069 / 913, 128 1116 / 1004, 129 1347 / 1370, 256 1358 / 1508), which it unpacks again for every
// tile; un-quantised ones it reads again (40 1079 / 696, 128 1424 / 979, 256 1685 / 1413, 300 1913 / 1678; the line was drawn at
// 1903 / 1902 for 384 rows, which are 1909 / 1786 now).
constexpr int kRowsChain = 128, kDenseRowsChain = 320;
constexpr int64_t kLayerWeights = (int64_t)(kQkvN + kHidden + 2 * kInter) * kHidden + (int64_t)kHidden * kInter;

inline int64_t align256(int64_t v) { return (v + 255) / 256 * 256; }

struct PrefillArena {
  int64_t lm, h, xn, tmp, qkv, q, attn, gu, act, xlast, ssq, ws, w16, total;
};

int64_t linear_ws(int rows) {
  if (rows >= kPairRows) return (int64_t)gemm_pair_splits(rows, kHidden, kInter) * rows * kHidden * 4;
  const int m = rows;
  int64_t w = quic_w4a16_workspace_bytes(m, kQkvN, kHidden);
  const int64_t o = quic_w4a16_workspace_bytes(m, kHidden, kHidden);
  const int64_t g = quic_w4a16_workspace_bytes(m, 2 * kInter, kHidden);
  const int64_t d = quic_w4a16_workspace_bytes(m, kHidden, kInter);
  w = w > o ? w : o;
  w = w > g ? w : g;
  return w > d ? w : d;
}

// The lm_head scratch (whose arrival counter must start zeroed) comes first.
PrefillArena carve_prefill(int rows, int n_seq, int vocab) {
  PrefillArena a;
  int64_t off = 0;
  a.lm = off;
  off += align256(quic_lm_head_scratch_bytes(n_seq, vocab));
  a.h = off;
  off += align256((int64_t)rows * kHidden * 2);
  a.xn = off;
  off += align256((int64_t)rows * kHidden * 2);
  a.tmp = off;
  off += align256((int64_t)rows * kHidden * 2);
  a.qkv = off;
  off += align256((int64_t)rows * kQkvN * 2);
  a.q = off;
  off += align256((int64_t)rows * kHidden * 2);
  a.attn = off;
  off += align256((int64_t)rows * kHidden * 2);
  a.gu = off;
  // gate|up is materialised by the one-row fallback and by dense weights below kDensePairRows rows
  off += align256((int64_t)(rows < kPairRows ? rows : 1) * 2 * kInter * 2);
  a.act = off;
  off += align256((int64_t)rows * kInter * 2);
  a.xlast = off;
  off += align256((int64_t)n_seq * kHidden * 2);
  a.ssq = a.qkv;  // sums of squares of the residual stream's rows, twice: on the rows chain, which leaves no qkv there
  static_assert(2 * kRowsSsq * 4 <= kQkvN * 2, "the sums fit in the place of the qkv rows");
  a.ws = off;
  off += align256(linear_ws(rows));
  a.w16 = off;  // fp16 copies of one layer's packed weights
  if (rows >= kPairRows) off += kLayerWeights * 2;
  a.total = off;
  return a;
}

// x[r] = embed[ids[r]] (ids clamped into the table), 224 threads x 8 bytes per row.
__global__ void __launch_bounds__(224) embed_tokens_kernel(const half* __restrict__ embed,
                                                           const int32_t* __restrict__ ids, int vocab,
                                                           half* __restrict__ x) {
  const int r = blockIdx.x, t = threadIdx.x;
  int id = ids[r];
  id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
  reinterpret_cast<uint2*>(x + (size_t)r * kHidden)[t] =
      reinterpret_cast<const uint2*>(embed + (size_t)id * kHidden)[t];
}

// y[i] = x[seq_start[i] + seq_len[i] - 1]: the last position of every sequence.
__global__ void __launch_bounds__(224) gather_last_kernel(const half* __restrict__ x,
                                                          const int32_t* __restrict__ seq_start,
                                                          const int32_t* __restrict__ seq_len,
                                                          half* __restrict__ y) {
  const int i = blockIdx.x, t = threadIdx.x;
  const int r = seq_start[i] + seq_len[i] - 1;
  reinterpret_cast<uint2*>(y + (size_t)i * kHidden)[t] = reinterpret_cast<const uint2*>(x + (size_t)r * kHidden)[t];
}

// tok[slot] = first generated token, pos[slot] = prompt length.
__global__ void set_slot_state_kernel(const int64_t* __restrict__ first, const int32_t* __restrict__ seq_len,
                                      const int32_t* __restrict__ seq_slot, const int32_t* __restrict__ seq_off,
                                      int n_seq, int n_slots, int32_t* __restrict__ tok, int32_t* __restrict__ pos) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_seq) return;
  const int slot = seq_slot[i];
  if (slot < 0 || slot >= n_slots) return;
  tok[slot] = (int32_t)first[i];
  pos[slot] = seq_len[i] + (seq_off != nullptr ? seq_off[i] : 0);
}

bool layer_pairs(const quic_layer_t& L, int rows) {
  const bool dense = L.qkv.w16 != nullptr && L.o.w16 != nullptr && L.gate_up.w16 != nullptr && L.down.w16 != nullptr;
  return rows >= (dense ? kDensePairRows : kPairRows);
}

// The linear for a consumer that sums K splits itself: with packed weights
// *splits > 1 fp32 partials stay in the workspace and y is not written; else y holds the result.
// (A finish kernel of its own costs a small prefill 2 us, three times a layer: 1 x 87 rows
// 1120 -> 1055 us.)
int linear_parts(const half* x, const quic_w4_t& w, half* y, int rows, void* ws, cudaStream_t st, int* splits,
                 bool adds_bias = false) {
  *splits = 0;
  if (w.w16 == nullptr && rows >= 2 && (adds_bias || w.bias == nullptr) &&
      w4a16_gemm_tc_workspace(rows, w.n, w.k) > 0)
    return w4a16_gemm_tc(x, w, nullptr, rows, static_cast<float*>(ws), st, splits);
  return quic_w4a16_linear(x, &w, y, rows, 1, ws, st);
}

// xn holds the finally normalised rows: lm_head + argmax on the last one of every sequence
int prefill_finish(const quic_model_t* m, const quic_prefill_t* p, const PrefillArena& ar, cudaStream_t st) {
  char* base = static_cast<char*>(p->scratch);
  const half* xn = reinterpret_cast<const half*>(base + ar.xn);
  half* xlast = reinterpret_cast<half*>(base + ar.xlast);
  gather_last_kernel<<<p->n_seq, 224, 0, st>>>(xn, p->seq_start, p->seq_len, xlast);
  QUIC_CUDA(cudaGetLastError());
  const int rc = quic_lm_head_argmax(xlast, nullptr, m->eps, m->embed, m->vocab, p->n_seq, p->logits, p->first_tokens, base + ar.lm, st);
  if (rc != QUIC_OK) return rc;
  set_slot_state_kernel<<<(p->n_seq + 127) / 128, 128, 0, st>>>(p->first_tokens, p->seq_len, p->seq_slot, p->seq_off,
                                                               p->n_seq, p->n_slots, p->tok, p->pos);
  QUIC_CUDA(cudaGetLastError());
  return QUIC_OK;
}

// Few rows: five launches a layer (rows_chain.cu and the attention).
int prefill_rows(const quic_model_t* m, const quic_prefill_t* p, const PrefillArena& ar, cudaStream_t st) {
  char* base = static_cast<char*>(p->scratch);
  half* h = reinterpret_cast<half*>(base + ar.h);
  half* q = reinterpret_cast<half*>(base + ar.q);
  half* attn = reinterpret_cast<half*>(base + ar.attn);
  half* act = reinterpret_cast<half*>(base + ar.act);
  float* const ssq_mid = reinterpret_cast<float*>(base + ar.ssq);
  float* const ssq_end = ssq_mid + (size_t)p->rows * kRowsSsq;
  const size_t kv_plane = (size_t)p->n_slots * kKvHeads * p->s_max * kHeadDim;
  RowsArgs a = {};
  a.rows = p->rows;
  a.eps = m->eps;
  a.slots = p->row_slot;
  a.row_pos = p->row_pos;
  a.cos_t = (const half*)m->rope_cos;
  a.sin_t = (const half*)m->rope_sin;
  a.max_pos = m->max_pos;
  a.s_max = p->s_max;
  a.n_slots = p->n_slots;
  a.head_major = 1;
  a.res = h;
  QUIC_CUDA(launch_embed_ssq((const half*)m->embed, nullptr, p->ids, m->vocab, h, ssq_end, p->rows, st, false));
  int rc;
  for (int l = 0; l < m->n_layers; ++l) {
    const quic_layer_t& L = m->layers[l];
    a.kcache = static_cast<half*>(p->kv) + (size_t)(2 * l) * kv_plane;
    a.vcache = a.kcache + kv_plane;
    a.w = L.qkv;
    a.y = q;
    a.ln = (const half*)L.ln1;
    a.ssq_in = ssq_end;
    a.n_ssq = l == 0 ? 1 : kRowsSsq;
    rows_next(&a, &L.o);
    if ((rc = rows_qkv(h, a, st)) != QUIC_OK) return rc;
    if ((rc = attn_prefill_launch(q, a.kcache, a.vcache, p->seq_start, p->seq_len, p->seq_slot, p->seq_off, p->n_seq, p->max_len, p->rows,
                                  p->s_max, p->n_slots, 0.125f /* 64^-0.5, src/model.py:129 */, attn, st, true)) != QUIC_OK)
      return rc;
    a.w = L.o;
    a.y = h;
    a.ssq_out = ssq_mid;
    rows_next(&a, &L.gate_up);
    if ((rc = rows_out(attn, a, st)) != QUIC_OK) return rc;
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
  QUIC_CUDA(launch_rmsnorm(h, nullptr, (const half*)m->final_norm, m->eps, reinterpret_cast<half*>(base + ar.xn), nullptr, p->rows, st));
  return QUIC_OK;
}

}  // namespace
}  // namespace quic

using namespace quic;

extern "C" int64_t quic_prefill_scratch_bytes(int32_t rows, int32_t n_seq, int32_t vocab) {
  if (rows < 1 || n_seq < 1 || vocab < 2) return 0;
  return carve_prefill(rows, n_seq, vocab).total;
}

extern "C" int quic_prefill(const quic_model_t* m, const quic_prefill_t* p, void* stream) {
  return quic_prefill_watch(m, p, nullptr, stream);
}

extern "C" int quic_prefill_watch(const quic_model_t* m, const quic_prefill_t* p, int32_t* error_words, void* stream) {
  QUIC_REQUIRE(m && p && m->layers && m->embed && m->final_norm && m->rope_cos && m->rope_sin, QUIC_E_ARG,
               "prefill: null model");
  QUIC_REQUIRE(p->ids && p->row_slot && p->row_pos && p->seq_start && p->seq_len && p->seq_slot && p->kv && p->tok &&
                   p->pos && p->first_tokens && p->scratch,
               QUIC_E_ARG, "prefill: null tensor");
  QUIC_REQUIRE(p->rows >= 1 && p->n_seq >= 1 && p->n_seq <= p->rows && p->n_seq <= 65535 && p->max_len >= 1 &&
                   p->max_len <= p->s_max && p->max_len <= m->max_pos && p->n_slots >= 1,
               QUIC_E_SHAPE, "prefill: bad row / sequence counts or a prompt longer than a KV slot");
  const StatusScope scope(error_words);
  QUIC_REQUIRE(scope.ok, QUIC_E_ARG, "prefill: the error words are not page-locked");
  cudaStream_t st = (cudaStream_t)stream;
  const int rows = p->rows;
  const PrefillArena ar = carve_prefill(rows, p->n_seq, m->vocab);
  char* base = static_cast<char*>(p->scratch);
  half* h = reinterpret_cast<half*>(base + ar.h);       // residual stream
  half* xn = reinterpret_cast<half*>(base + ar.xn);     // normalised input of the next linear
  half* tmp = reinterpret_cast<half*>(base + ar.tmp);   // o_proj / down output
  half* qkv = reinterpret_cast<half*>(base + ar.qkv);
  half* q = reinterpret_cast<half*>(base + ar.q);
  half* attn = reinterpret_cast<half*>(base + ar.attn);
  half* gu = reinterpret_cast<half*>(base + ar.gu);
  half* act = reinterpret_cast<half*>(base + ar.act);
  void* ws = base + ar.ws;
  half* const w16[4] = {reinterpret_cast<half*>(base + ar.w16), reinterpret_cast<half*>(base + ar.w16) + kQkvN * kHidden,
                        reinterpret_cast<half*>(base + ar.w16) + (kQkvN + kHidden) * kHidden,
                        reinterpret_cast<half*>(base + ar.w16) + (kQkvN + kHidden + 2 * kInter) * kHidden};
  const size_t slot_stride = (size_t)kKvHeads * p->s_max * kHeadDim;
  const size_t kv_plane = (size_t)p->n_slots * slot_stride;

  int rc = QUIC_OK, sp = 0;
  if (rows >= 2 && rows <= (m->layers[0].qkv.w16 != nullptr ? kDenseRowsChain : kRowsChain)) {
    if ((rc = prefill_rows(m, p, ar, st)) != QUIC_OK) return rc;
    return prefill_finish(m, p, ar, st);
  }
  embed_tokens_kernel<<<rows, 224, 0, st>>>((const half*)m->embed, p->ids, m->vocab, h);
  QUIC_CUDA(cudaGetLastError());
  // From here on the kernels are chained with programmatic dependent launch: each one does
  // its set-up (and the GEMMs request their weight tiles) while its predecessor drains.
  QUIC_CUDA(launch_rmsnorm(h, nullptr, (const half*)m->layers[0].ln1, m->eps, xn, nullptr, rows, st));
  const float* part = static_cast<const float*>(ws) + 4096;  // (behind the workspace's 16 KB head)
  for (int l = 0; l < m->n_layers; ++l) {
    const quic_layer_t& L = m->layers[l];
    half* kc = static_cast<half*>(p->kv) + (size_t)(2 * l) * kv_plane;
    half* vc = kc + kv_plane;
    if (layer_pairs(L, rows)) {
      const quic_w4_t* const w[4] = {&L.qkv, &L.o, &L.gate_up, &L.down};
      const half* f[4];
      int packed = 0;
      for (int i = 0; i < 4; ++i) {
        f[i] = w[i]->w16 != nullptr ? (const half*)w[i]->w16 : w16[i];
        packed += w[i]->w16 == nullptr;
      }
      if (packed > 0 && (rc = w4_unpack(w, w16, 4, st)) != QUIC_OK) return rc;
      const PairRope rope = {p->row_slot, p->row_pos, (const half*)m->rope_cos, (const half*)m->rope_sin, q, kc, vc,
                             m->max_pos, p->s_max, p->n_slots};
      if ((rc = gemm_pair_qkv(xn, f[0], (const half*)L.qkv.bias, rows, rope, st)) != QUIC_OK) return rc;
      if ((rc = attn_prefill_launch(q, kc, vc, p->seq_start, p->seq_len, p->seq_slot, p->seq_off, p->n_seq, p->max_len,
                                    rows, p->s_max, p->n_slots, 0.125f, attn, st, true)) != QUIC_OK)
        return rc;
      if ((rc = gemm_pair(attn, f[1], (const half*)L.o.bias, tmp, rows, kHidden, kHidden, false, st)) != QUIC_OK) return rc;
      QUIC_CUDA(launch_rmsnorm(tmp, h, (const half*)L.ln2, m->eps, xn, h, rows, st));
      if ((rc = gemm_pair(xn, f[2], nullptr, act, rows, 2 * kInter, kHidden, true, st)) != QUIC_OK) return rc;
      if ((rc = gemm_pair(act, f[3], (const half*)L.down.bias, tmp, rows, kHidden, kInter, false, st,
                          L.down.bias == nullptr ? static_cast<float*>(ws) : nullptr, &sp)) != QUIC_OK)
        return rc;
      const void* next_ln = (l + 1 < m->n_layers) ? m->layers[l + 1].ln1 : m->final_norm;
      QUIC_CUDA(sp > 0 ? launch_rmsnorm_part(static_cast<const float*>(ws), sp, h, (const half*)next_ln, m->eps, xn, h, rows, st)
                       : launch_rmsnorm(tmp, h, (const half*)next_ln, m->eps, xn, h, rows, st));
      continue;
    }
    if ((rc = linear_parts(xn, L.qkv, qkv, rows, ws, st, &sp, true)) != QUIC_OK) return rc;
    QUIC_CUDA(launch_qkv_rope_append(qkv, p->row_slot, p->row_pos, (const half*)m->rope_cos, (const half*)m->rope_sin,
                                     m->max_pos, q, kc, vc, p->s_max, p->n_slots, rows, st, true, sp > 0 ? part : nullptr, sp,
                                     (const half*)L.qkv.bias));
    if ((rc = attn_prefill_launch(q, kc, vc, p->seq_start, p->seq_len, p->seq_slot, p->seq_off, p->n_seq, p->max_len,
                                  rows, p->s_max, p->n_slots, 0.125f /* 64^-0.5, src/model.py:129 */, attn, st, true)) != QUIC_OK)
      return rc;
    if ((rc = linear_parts(attn, L.o, tmp, rows, ws, st, &sp)) != QUIC_OK) return rc;
    // h += o ; xn = norm(h)
    QUIC_CUDA(sp > 0 ? launch_rmsnorm_part(part, sp, h, (const half*)L.ln2, m->eps, xn, h, rows, st)
                     : launch_rmsnorm(tmp, h, (const half*)L.ln2, m->eps, xn, h, rows, st));
    if (L.gate_up.w16 == nullptr && rows >= 2) {
      // gate|up GEMM with SwiGLU in its epilogue: the [rows, 9728] intermediate never exists
      if ((rc = w4a16_gemm_tc_swiglu(xn, L.gate_up, act, rows, st)) != QUIC_OK) return rc;
    } else {
      if ((rc = quic_w4a16_linear(xn, &L.gate_up, gu, rows, 1, ws, stream)) != QUIC_OK) return rc;
      QUIC_CUDA(launch_swiglu_fused(gu, act, rows, st));
    }
    if ((rc = linear_parts(act, L.down, tmp, rows, ws, st, &sp)) != QUIC_OK) return rc;
    const void* next_ln = (l + 1 < m->n_layers) ? m->layers[l + 1].ln1 : m->final_norm;
    QUIC_CUDA(sp > 0 ? launch_rmsnorm_part(part, sp, h, (const half*)next_ln, m->eps, xn, h, rows, st)
                     : launch_rmsnorm(tmp, h, (const half*)next_ln, m->eps, xn, h, rows, st));
  }
  return prefill_finish(m, p, ar, st);
}
