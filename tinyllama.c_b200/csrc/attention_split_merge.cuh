// The merge of the splits of single-token attention, run by the last block of a (row, key/value
// head) to finish: softmax statistics (maximum, sum) and unnormalised partial outputs of every
// split become the normalised output (CodeClaper/tinyllama.c cpu_op.c:1010-1062 computes the same softmax
// in one piece).  All in 32-bit.
#pragma once
#include "common.cuh"

// part_o [T, H, n_splits, HD], part_ml [T, H, n_splits, 2]; out: rows of out_ld elements, head h at h * HD;
// sh: the block's dynamic shared memory of smem_floats floats (free by now); NT threads.  All threads of
// the block call it.  A split without keys has a sum of 0 and no outputs; any other sum counts, NaN among them.  head_gate: see tlc_head_gate.  sink: one more split of maximum 0 (or sink_values[head]) and sum 1 that carries no values.
template <int HD, int NT>
__device__ __forceinline__ void attention_merge_splits(const float* part_o, const float* part_ml, __nv_bfloat16* out,
                                                       float* sh, int smem_floats, int t, int g, int G, int H,
                                                       int n_splits, int out_ld, int sink = 0,
                                                       const float* sink_values = nullptr, const float* head_gate = nullptr,
                                                       int gate_ld = 0) {
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  constexpr int NW = NT / 32;
  if (2 * G * n_splits <= smem_floats) {
    // statistics of all heads and splits into shared memory (one round trip), weights from them,
    // then the weighted sum with the loads of a thread in flight together
    for (int idx = tid; idx < G * n_splits; idx += NT) {
      const int hg = idx / n_splits, s = idx % n_splits;
      const float2 v = __ldcg(reinterpret_cast<const float2*>(part_ml + (((size_t)t * H + (size_t)g * G + hg) * n_splits + s) * 2));
      sh[2 * idx] = v.x;
      sh[2 * idx + 1] = v.y;
    }
    __syncthreads();
    for (int hg = wp; hg < G; hg += NW) {
      float* e = sh + (size_t)2 * hg * n_splits;
      float m = -INFINITY;
      for (int s = lane; s < n_splits; s += 32) m = fmaxf(m, e[2 * s]);
      m = warp_max(m);
      const float sv = (sink && sink_values) ? sink_values[g * G + hg] : 0.f;    // the sink's score: 0, or the head's own
      if (sink) m = fmaxf(m, sv);
      float l = 0.f;
      for (int s = lane; s < n_splits; s += 32) if (e[2 * s + 1] != 0.f) l += e[2 * s + 1] * expf(e[2 * s] - m);
      l = warp_sum(l);
      if (sink) l += expf(sv - m);
      const float inv = tlc_head_gate(head_gate, gate_ld, t, g * G + hg) / l;
      for (int s = lane; s < n_splits; s += 32) e[2 * s] = e[2 * s + 1] != 0.f ? expf(e[2 * s] - m) * inv : 0.f;
    }
    __syncthreads();
    // four outputs of a thread at a time, eight splits of each: 32 loads in flight, all unconditional (past the last split or
    // output they read the last one, with weight 0); one output after the other, 32 splits were 16 trips to memory in a row
    // (a step of the 1.5B sizes after 3,700 tokens: one sequence 1108 -> 1090 us, two 1161 -> 1131, four 1186 -> 1160)
    constexpr int NI = 4, NS = 8;
    for (int base = tid; base < G * HD; base += NI * NT) {
      const float* po[NI];
      const float* e[NI];
      float acc[NI];
#pragma unroll
      for (int i = 0; i < NI; i++) {
        const int idx = min(base + i * NT, G * HD - 1), hg = idx / HD;
        po[i] = part_o + ((size_t)t * H + (size_t)g * G + hg) * n_splits * HD + idx % HD;
        e[i] = sh + (size_t)2 * hg * n_splits;
        acc[i] = 0.f;
      }
      for (int s0 = 0; s0 < n_splits; s0 += NS) {
        float v[NI][NS];
#pragma unroll
        for (int u = 0; u < NS; u++)
#pragma unroll
          for (int i = 0; i < NI; i++) v[i][u] = __ldcg(po[i] + (size_t)min(s0 + u, n_splits - 1) * HD);
#pragma unroll
        for (int u = 0; u < NS; u++)
#pragma unroll
          for (int i = 0; i < NI; i++) {
            const float w = s0 + u < n_splits ? e[i][2 * (s0 + u)] : 0.f;
            acc[i] = w != 0.f ? fmaf(v[i][u], w, acc[i]) : acc[i];
          }
      }
#pragma unroll
      for (int i = 0; i < NI; i++) {
        const int idx = base + i * NT;
        if (idx < G * HD) out[(size_t)t * out_ld + (size_t)g * G * HD + idx] = __float2bfloat16_rn(acc[i]);
      }
    }
    return;
  }
  // more splits than shared memory holds statistics for: one head after the other from global memory
  for (int hg = 0; hg < G; hg++) {
    const size_t th = (size_t)t * H + (size_t)g * G + hg;
    const float* mlh = part_ml + th * n_splits * 2;
    float m = -INFINITY;
    for (int s = 0; s < n_splits; s++) m = fmaxf(m, __ldcg(mlh + 2 * s));
    const float sv = (sink && sink_values) ? sink_values[g * G + hg] : 0.f;
    if (sink) m = fmaxf(m, sv);
    float l = sink ? expf(sv - m) : 0.f;
    for (int s = 0; s < n_splits; s++) {
      const float ls = __ldcg(mlh + 2 * s + 1);
      if (ls != 0.f) l += ls * expf(__ldcg(mlh + 2 * s) - m);
    }
    const float inv = tlc_head_gate(head_gate, gate_ld, t, g * G + hg) / l;
    for (int d = tid; d < HD; d += NT) {
      float acc = 0.f;
      for (int s = 0; s < n_splits; s++)
        if (__ldcg(mlh + 2 * s + 1) != 0.f)
          acc = fmaf(__ldcg(part_o + (th * n_splits + s) * HD + d), expf(__ldcg(mlh + 2 * s) - m), acc);
      out[(size_t)t * out_ld + ((size_t)g * G + hg) * HD + d] = __float2bfloat16_rn(acc * inv);
    }
  }
}
