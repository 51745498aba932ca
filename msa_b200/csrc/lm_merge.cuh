// Merge of the partial results of a split decode attention: weights e^(m_i - m), a sink, an output gate.
#pragma once
#include "lm_common.cuh"

namespace msa {

struct MergeParams {
  const float *part_o, *part_ml;     // [rows, splits, cols], [rows, splits, 2] (maximum in log2 units, sum)
  int heads, splits, cols;
  int sink;                          // one more entry with score 0 and no value
  const __nv_bfloat16* gate; long long gate_row;   // null, or a logit per (sequence, head)
  __nv_bfloat16* out; long long out_row;           // row stride of a sequence; heads are cols apart
};

// One block per (sequence, head).  Launched behind the attention, not early: an SM takes on another split of shared memory and L1 only
// when it is empty, and blocks that join the attention's, with the product that starts early behind them, keep its small L1, which is
// too small for the loads such a product has in flight.  Behind 8 sequences' attention a gated product of 12288 x 2048 took 10.4 us
// instead of 17, the next one of 2048 x 8192 8 instead of 13, and the merge itself, no longer beside that product's loads, 4.6.
static __global__ void __launch_bounds__(128) merge_partials_kernel(const MergeParams p) {
  let_product_start((int)(gridDim.x / (unsigned)p.heads));
  const long long row = blockIdx.x;
  const int b = (int)(row / p.heads), h = (int)(row % p.heads);
  const int c = threadIdx.x * 4, splits = p.splits, cols = p.cols;
  const float g = p.gate ? sigmoid_f(__bfloat162float(p.gate[b * p.gate_row + h])) : 1.f;
  float m = p.sink ? 0.f : -INFINITY, l = p.sink ? 1.f : 0.f;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s0 = 0; s0 < splits; s0 += 8) {               // eight partial results in flight; an empty one has weight 0
    float4 v[8];
    float2 ml[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const bool on = s0 + i < splits;
      ml[i] = on ? *reinterpret_cast<const float2*>(p.part_ml + (row * splits + s0 + i) * 2) : make_float2(-INFINITY, 0.f);
      v[i] = on && c < cols ? load4(p.part_o + (row * splits + s0 + i) * cols + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float mx = m;
#pragma unroll
    for (int i = 0; i < 8; ++i) mx = fmaxf(mx, ml[i].x);
    const float f = m == -INFINITY ? 0.f : exp2f(m - mx);
    l *= f; a.x *= f; a.y *= f; a.z *= f; a.w *= f;
    m = mx;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float w = ml[i].x == -INFINITY ? 0.f : exp2f(ml[i].x - m);
      l = fmaf(w, ml[i].y, l);
      a.x = fmaf(w, v[i].x, a.x); a.y = fmaf(w, v[i].y, a.y); a.z = fmaf(w, v[i].z, a.z); a.w = fmaf(w, v[i].w, a.w);
    }
  }
  const float inv = g / l;
  if (c < cols) store4(p.out + b * p.out_row + (long long)h * cols + c, make_float4(a.x * inv, a.y * inv, a.z * inv, a.w * inv));
}

inline int launch_merge(const MergeParams& p, int n, cudaStream_t stream) {
  merge_partials_kernel<<<dim3((unsigned)(n * p.heads)), 128, 0, stream>>>(p);
  MSA_CUDA_OK(cudaGetLastError());
  return MSA_OK;
}

}  // namespace msa
