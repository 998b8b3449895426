// One warp's 64-token tile of decode attention from swizzled shared memory, with the tokens (first
// product) or the head dims (second) on the M side of mma.sync and the seven heads of a KV head on its N side:
// seven of eight columns are used, where heads on M leave nine of sixteen rows empty.  Shared
// by attn_decode_flow.cu and attn_decode_stream.cu.
#pragma once
#include "attn_warp.cuh"
#include "tc_common.cuh"

namespace quic {

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void ldsm4_trans(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
  uint32_t d;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}

// running softmax of the warp's tiles: columns 2t, 2t + 1 (t = lane & 3) are heads; o: dims g + 8 .. of them
struct FlowState {
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[4][4] = {};
};

// the tile's fragments and scores; K and V of the stage are in registers afterwards
__device__ __forceinline__ void flow_scores(uint32_t k_s, uint32_t v_s, const uint32_t (&qb)[4][2], int lane, uint32_t (&V)[4][4][4],
                                            float (&sc)[4][4]) {
  const int mi = lane >> 3, mr = lane & 7;
  uint32_t K[4][4][4];
#pragma unroll
  for (int ks = 0; ks < 4; ++ks)
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) ldsm4(K[mt][ks], k_s + sw128_offset(16 * mt + 8 * (mi & 1) + mr, 2 * ks + (mi >> 1)));
#pragma unroll
  for (int ks = 0; ks < 4; ++ks)
#pragma unroll
    for (int dt = 0; dt < 4; ++dt)
      ldsm4_trans(V[dt][ks], v_s + sw128_offset(16 * ks + 8 * (mi >> 1) + mr, 2 * dt + (mi & 1)));
#pragma unroll
  for (int mt = 0; mt < 4; ++mt) sc[mt][0] = sc[mt][1] = sc[mt][2] = sc[mt][3] = 0.f;
#pragma unroll
  for (int ks = 0; ks < 4; ++ks)
#pragma unroll
    for (int mt = 0; mt < 4; ++mt)
      mma16816(sc[mt], K[mt][ks][0], K[mt][ks][1], K[mt][ks][2], K[mt][ks][3], qb[ks][0], qb[ks][1]);
}

// softmax over the tokens [t_begin, t_end) of the tile at t0, and the second product
__device__ __forceinline__ void flow_attend(FlowState& st, uint32_t (&V)[4][4][4], float (&sc)[4][4], int t0, int t_begin, int t_end,
                                            float scale, int lane) {
  const int g = lane >> 2, t = lane & 3;
  float (&m)[2] = st.m, (&l)[2] = st.l, (&o)[4][4] = st.o;
  const bool edge = t0 < t_begin || t0 + kWarpChunk > t_end;
  if (edge) {  // values outside the row's tokens may be anything, 0 x NaN included
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int tok = t0 + 16 * ks + 8 * hh + 2 * t;
        const uint32_t keep_v = (tok >= t_begin && tok < t_end ? 0xffffu : 0u) |
                                (tok + 1 >= t_begin && tok + 1 < t_end ? 0xffff0000u : 0u);
#pragma unroll
        for (int dt = 0; dt < 4; ++dt) {
          V[dt][ks][2 * hh] &= keep_v;
          V[dt][ks][2 * hh + 1] &= keep_v;
        }
      }
  }
  float mx[2] = {m[0], m[1]};
#pragma unroll
  for (int mt = 0; mt < 4; ++mt)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float s = sc[mt][e] * scale;
      if (edge) {
        const int tok = t0 + 16 * mt + g + 8 * (e >> 1);
        s = tok >= t_begin && tok < t_end ? s : -INFINITY;
      }
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
  uint32_t pb[4][2];
#pragma unroll
  for (int mt = 0; mt < 4; ++mt)
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
  for (int ks = 0; ks < 4; ++ks)
#pragma unroll
    for (int dt = 0; dt < 4; ++dt)
      mma16816(o[dt], V[dt][ks][0], V[dt][ks][1], V[dt][ks][2], V[dt][ks][3], pb[ks][0], pb[ks][1]);
}

// the warp's state -> shared memory: maxima, sums and unnormalised outputs of its heads
__device__ __forceinline__ void flow_store(FlowState& st, float (&m_w)[8], float (&l_w)[8], float (&o_w)[kHeads / kKvHeads][kHeadDim],
                                           int lane) {
  const int g = lane >> 2, t = lane & 3;
  float (&m)[2] = st.m, (&l)[2] = st.l, (&o)[4][4] = st.o;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
#pragma unroll
    for (int x = 4; x < 32; x <<= 1) l[e] += __shfl_xor_sync(0xffffffffu, l[e], x);
    const int hd = 2 * t + e;
    if (hd < kHeads / kKvHeads) {
#pragma unroll
      for (int dt = 0; dt < 4; ++dt) {
        o_w[hd][16 * dt + g] = o[dt][e];
        o_w[hd][16 * dt + 8 + g] = o[dt][2 + e];
      }
      if (g == 0) {
        m_w[hd] = m[e];
        l_w[hd] = l[e];
      }
    }
  }
}

}  // namespace quic
