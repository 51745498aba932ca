// The elementwise work between the GEMMs of the memory model (bf16): head norm + rotation, residual add + RMSNorm,
// silu(gate) * up, rotation tables.  The reference's modules (Qwen3RMSNorm, apply_rotary_pos_emb, residual adds, SiLU * up;
// transformers' modeling_qwen3 as used by src/msa/model.py:67-135) issue some forty elementwise kernels per layer: over a
// block of documents they move every activation about ten times, in a decode step they are forty launches over a few KB.
// Here each reads its inputs once, computes in fp32 and rounds once.
//
// All are bound by HBM on a block of documents and by launch latency in a decode step.
//
// Quotients, roots and exponentials are the fast ones (a few 2^-23 of themselves, subnormals flushed) where the eager modules take
// the exact ones: the results are rounded to 8 bits once, the modules' two to four times, and that outweighs it.  silu(gate) * up over
// every finite bf16 gate from -87 on and four values of up, against 64 bits: at most 1.00 x 2^-8 of the result and 0.43 x 2^-8 in the mean (root of
// squares); silu and product as two modules 1.61 and 0.45.  Below -87 the sum 1 + e^-gate passes 2^126 and the result, 3e-36 at
// most in size, is 0.  No choice between discrete things hangs on last bits here (the layered decoders' experts, which do, take exact ones).
#include "common.cuh"

namespace msa {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
struct HeadsNormRope {
  const __nv_bfloat16 *q, *k;                 // [rows, heads * 128]
  long long q_stride, k_stride;
  int n_rows, n_q, n_kv, cos_rows;
  const __nv_bfloat16 *q_w, *k_w, *cos_t, *sin_t;
  __nv_bfloat16 *q_out, *k_out;               // contiguous
  float eps;
};

// RMS-normalise every q and k head of a row (weight per dimension), rotate by the row's cos / sin (first and second half of a
// head form the planes).  head_dim = 128: 64 / V lanes share a head, lane l holds dimensions V*l .. and 64 + V*l .. , so both
// members of a plane are in one thread and no value crosses lanes but the sum of squares.  V = 8 where rows are 16-byte
// aligned, else 4.  A warp takes PER rounds of heads of one row with all their loads in flight: 8 heads under one row's angles
// where there are rows enough, one round where a decode step's few rows have to spread over the SMs.
// 32,002 rows of 32 + 8 heads (655 MB): 135 us = 4.9 TB/s; V = 4 175 us; the eager modules about 2.7 ms.
template <int V> struct Half;
template <> struct Half<4> { using type = uint2; };
template <> struct Half<8> { using type = uint4; };
template <int V>
__device__ __forceinline__ void widen_half(const typename Half<V>::type& r, float (&f)[V]) {
#pragma unroll
  for (int i = 0; i < V / 2; ++i) {
    const float2 a = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&r)[i]);
    f[2 * i] = a.x; f[2 * i + 1] = a.y;
  }
}
template <int V>
__device__ __forceinline__ void store_half(__nv_bfloat16* p, const float (&f)[V]) {
  typename Half<V>::type r;
#pragma unroll
  for (int i = 0; i < V / 2; ++i) reinterpret_cast<__nv_bfloat162*>(&r)[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<typename Half<V>::type*>(p) = r;
}

template <int V, int PER>
__global__ void __launch_bounds__(256) heads_norm_rope_kernel(const HeadsNormRope p) {
  using R = typename Half<V>::type;
  constexpr int kLanes = 64 / V, kHeads = 32 / kLanes;      // lanes of a head, heads of a round
  const int lane = threadIdx.x & 31, sub = lane / kLanes, l = lane % kLanes;
  const int heads = p.n_q + p.n_kv, groups = (heads + kHeads * PER - 1) / (kHeads * PER);
  const unsigned unit = blockIdx.x * 8u + (threadIdx.x >> 5);
  const unsigned row = unit / (unsigned)groups;
  if (row >= (unsigned)p.n_rows) return;
  const int h0 = (int)(unit - row * groups) * kHeads * PER + sub;
  R lo[PER], hi[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int h = h0 + kHeads * i;
    lo[i] = hi[i] = R{};
    if (h >= heads) continue;
    const __nv_bfloat16* src = h < p.n_q ? p.q + row * p.q_stride + (long long)h * 128 : p.k + row * p.k_stride + (long long)(h - p.n_q) * 128;
    lo[i] = *reinterpret_cast<const R*>(src + V * l);
    hi[i] = *reinterpret_cast<const R*>(src + 64 + V * l);
  }
  const long long at = (long long)(row % (unsigned)p.cos_rows) * 128 + V * l;
  float cl[V], ch[V], sl[V], sh[V];
  widen_half<V>(*reinterpret_cast<const R*>(p.cos_t + at), cl);
  widen_half<V>(*reinterpret_cast<const R*>(p.cos_t + at + 64), ch);
  widen_half<V>(*reinterpret_cast<const R*>(p.sin_t + at), sl);
  widen_half<V>(*reinterpret_cast<const R*>(p.sin_t + at + 64), sh);
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int h = h0 + kHeads * i;
    float a[V], b[V], wa[V], wb[V], ss = 0.f;
    widen_half<V>(lo[i], a);
    widen_half<V>(hi[i], b);
#pragma unroll
    for (int j = 0; j < V; ++j) ss += a[j] * a[j] + b[j] * b[j];
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (h >= heads) continue;
    const float inv = rsqrtf(ss * (1.f / 128.f) + p.eps);
    const __nv_bfloat16* w = h < p.n_q ? p.q_w : p.k_w;
    widen_half<V>(*reinterpret_cast<const R*>(w + V * l), wa);
    widen_half<V>(*reinterpret_cast<const R*>(w + 64 + V * l), wb);
    __nv_bfloat16* dst = h < p.n_q ? p.q_out + ((long long)row * p.n_q + h) * 128 : p.k_out + ((long long)row * p.n_kv + h - p.n_q) * 128;
    float oa[V], ob[V];
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const float x = a[j] * (inv * wa[j]), y = b[j] * (inv * wb[j]);
      oa[j] = x * cl[j] - y * sl[j];
      ob[j] = y * ch[j] + x * sh[j];
    }
    store_half<V>(dst + V * l, oa);
    store_half<V>(dst + 64 + V * l, ob);
  }
}

// x_out = x + y (y may be null; the sum is rounded to bf16, as the residual stream is stored), h_out = rmsnorm(x_out) * w.
// T threads share a row and keep it in registers, NV 16-byte vectors each, all in flight at once: a warp per row needs no
// block-wide step and suits many rows, a block per row brings the few rows of a decode step in with one round of loads.
// 32,002 rows of 2560 (four streams, 655 MB): 98 us = 6.7 TB/s (eager modules 0.6 ms); 32 rows: 2.8 us.
template <int T, int NV>
__global__ void __launch_bounds__(256)
add_rmsnorm_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ w,
                   float eps, int n_rows, int hidden, __nv_bfloat16* __restrict__ x_out, __nv_bfloat16* __restrict__ h_out) {
  const long long row = (long long)blockIdx.x * (256 / T) + threadIdx.x / T;
  if (row >= n_rows) return;                      // whole warps (T = 32) or never (T = 256)
  const int t = threadIdx.x % T, vecs = hidden / 8;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * hidden);
  const uint4* yr = reinterpret_cast<const uint4*>(y + row * hidden);
  uint4 v[NV], u[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) if (t + i * T < vecs) v[i] = xr[t + i * T];
  if (y) {
#pragma unroll
    for (int i = 0; i < NV; ++i) if (t + i * T < vecs) u[i] = yr[t + i * T];
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (t + i * T >= vecs) continue;
    __nv_bfloat162* a = reinterpret_cast<__nv_bfloat162*>(&v[i]);
    const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u[i]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 f = __bfloat1622float2(a[j]);
      if (y) {
        const float2 g = __bfloat1622float2(b[j]);
        a[j] = __floats2bfloat162_rn(f.x + g.x, f.y + g.y);
        f = __bfloat1622float2(a[j]);
      }
      ss += f.x * f.x + f.y * f.y;
    }
    if (y && x_out) reinterpret_cast<uint4*>(x_out + row * hidden)[t + i * T] = v[i];
  }
  ss = warp_sum(ss);
  if (T > 32) {
    __shared__ float part[8];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
    __syncthreads();
    ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += part[i];
  }
  const float inv = rsqrtf(ss / (float)hidden + eps);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (t + i * T >= vecs) continue;
    const uint4 wr = reinterpret_cast<const uint4*>(w)[t + i * T];
    const __nv_bfloat162* a = reinterpret_cast<const __nv_bfloat162*>(&v[i]);
    const __nv_bfloat162* g = reinterpret_cast<const __nv_bfloat162*>(&wr);
    uint4 o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(a[j]), s = __bfloat1622float2(g[j]);
      reinterpret_cast<__nv_bfloat162*>(&o)[j] = __floats2bfloat162_rn(f.x * inv * s.x, f.y * inv * s.y);
    }
    reinterpret_cast<uint4*>(h_out + row * hidden)[t + i * T] = o;
  }
}

// The same for rows that are no whole number of aligned 16-byte vectors, or wider than the registers above hold.
__global__ void __launch_bounds__(256)
add_rmsnorm_pairs_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ y,
                         const __nv_bfloat16* __restrict__ w, float eps, int hidden, __nv_bfloat16* __restrict__ x_out,
                         __nv_bfloat16* __restrict__ h_out) {
  extern __shared__ float s_row[];   // [hidden]
  __shared__ float s_part[8];
  const long long base = (long long)blockIdx.x * hidden;
  float ss = 0.f;
  for (int i = threadIdx.x * 2; i < hidden; i += 512) {
    float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(x + base + i));
    if (y) {
      const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(y + base + i));
      a.x = Elem<__nv_bfloat16>::round(a.x + b.x);
      a.y = Elem<__nv_bfloat16>::round(a.y + b.y);
      if (x_out) *reinterpret_cast<__nv_bfloat162*>(x_out + base + i) = __floats2bfloat162_rn(a.x, a.y);
    }
    s_row[i] = a.x;
    s_row[i + 1] = a.y;
    ss += a.x * a.x + a.y * a.y;
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += s_part[i];
  const float inv = rsqrtf(tot / (float)hidden + eps);
  for (int i = threadIdx.x * 2; i < hidden; i += 512) {
    const float2 wv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(w + i));
    *reinterpret_cast<__nv_bfloat162*>(h_out + base + i) = __floats2bfloat162_rn(s_row[i] * inv * wv.x, s_row[i + 1] * inv * wv.y);
  }
}

__device__ __forceinline__ float silu_times(float g, float u) { return g / (1.f + __expf(-g)) * u; }

// out[r, j] = silu(gate[r, j]) * up[r, j]; V elements per access (8 where everything is 16-byte aligned, else 2), four
// accesses of each operand in flight per thread.  32,002 rows of 9728 (1.87 GB): 272 us = 6.9 TB/s (two eager kernels 546 us).
template <int V> struct Pack;
template <> struct Pack<8> { using type = uint4; };
template <> struct Pack<2> { using type = uint32_t; };
template <int V>
__global__ void __launch_bounds__(256)
silu_mul_kernel(const __nv_bfloat16* __restrict__ gate, long long gate_stride, const __nv_bfloat16* __restrict__ up, long long up_stride,
                int ffn, int n_rows, __nv_bfloat16* __restrict__ out) {
  using P = typename Pack<V>::type;
  const int per_row = ffn / V;
  const long long total = (long long)n_rows * per_row;
  const long long first = (long long)blockIdx.x * 1024 + threadIdx.x;
  P g[4], u[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const long long i = first + k * 256;
    if (i >= total) continue;
    const long long r = i / per_row;
    const int j = (int)(i - r * per_row) * V;
    g[k] = __ldcs(reinterpret_cast<const P*>(gate + r * gate_stride + j));
    u[k] = __ldcs(reinterpret_cast<const P*>(up + r * up_stride + j));
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const long long i = first + k * 256;
    if (i >= total) continue;
    P o;
#pragma unroll
    for (int e = 0; e < V / 2; ++e) {
      const float2 a = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&g[k])[e]);
      const float2 b = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&u[k])[e]);
      reinterpret_cast<__nv_bfloat162*>(&o)[e] = __floats2bfloat162_rn(silu_times(a.x, b.x), silu_times(a.y, b.y));
    }
    reinterpret_cast<P*>(out)[i] = o;             // rows of out are contiguous
  }
}

// cos / sin [n, 2 * half] of pos * inv_freq (the product in fp32, as the reference's rotary module forms it; the angle's
// functions in 64 bits, so that large positions keep their phase), both halves alike, scaled and rounded to bf16.
__global__ void __launch_bounds__(256)
rope_table_kernel(const int64_t* __restrict__ pos, const float* __restrict__ inv_freq, int n, int half, float scaling,
                  __nv_bfloat16* __restrict__ cos_t, __nv_bfloat16* __restrict__ sin_t) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)n * half) return;
  const long long r = i / half;
  const int j = (int)(i - r * half);
  double s, c;
  sincos((double)__fmul_rn((float)pos[r], inv_freq[j]), &s, &c);
  const __nv_bfloat16 cb = __float2bfloat16_rn((float)c * scaling), sb = __float2bfloat16_rn((float)s * scaling);
  const long long at = r * 2 * half + j;
  cos_t[at] = cos_t[at + half] = cb;
  sin_t[at] = sin_t[at + half] = sb;
}

static bool aligned4(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 3u) == 0; }
static bool aligned8(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 7u) == 0; }

// Eight heads per warp once that fills the GPU's warp slots (64 an SM), else one round of heads.
static int launch_heads_norm_rope(const HeadsNormRope& p, void* stream) {
  const int heads = p.n_q + p.n_kv;
  const bool wide = aligned16(p.q) && aligned16(p.k) && aligned16(p.q_w) && aligned16(p.k_w) && aligned16(p.cos_t) && aligned16(p.sin_t) &&
                    aligned16(p.q_out) && aligned16(p.k_out) && p.q_stride % 8 == 0 && p.k_stride % 8 == 0;
  int n_sm = 0;
  MSA_OK_OR_RETURN(device_sm_count(&n_sm));
  const bool many = (long long)p.n_rows * ((heads + 7) / 8) >= 64ll * n_sm;
  const int per_warp = many ? 8 : wide ? 4 : 2;
  const unsigned grid = (unsigned)(((long long)p.n_rows * ((heads + per_warp - 1) / per_warp) + 7) / 8);
  cudaStream_t st = (cudaStream_t)stream;
  if (wide && many) heads_norm_rope_kernel<8, 2><<<grid, 256, 0, st>>>(p);
  else if (wide) heads_norm_rope_kernel<8, 1><<<grid, 256, 0, st>>>(p);
  else if (many) heads_norm_rope_kernel<4, 4><<<grid, 256, 0, st>>>(p);
  else heads_norm_rope_kernel<4, 1><<<grid, 256, 0, st>>>(p);
  MSA_LAUNCH_OK("heads_norm_rope_kernel");
  return MSA_OK;
}

template <int T, int NV>
static void launch_add_rmsnorm(const void* x, const void* y, const void* w, float eps, int n_rows, int hidden, void* x_out, void* h_out,
                               void* stream) {
  add_rmsnorm_kernel<T, NV><<<(n_rows + 256 / T - 1) / (256 / T), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)x, (const __nv_bfloat16*)y, (const __nv_bfloat16*)w, eps, n_rows, hidden, (__nv_bfloat16*)x_out, (__nv_bfloat16*)h_out);
}

}  // namespace msa

using namespace msa;

extern "C" int msa_heads_norm_rope(const void* q, int64_t q_stride, const void* k, int64_t k_stride, int32_t n_rows, int32_t n_q_heads,
                                   int32_t n_kv_heads, int32_t head_dim, const void* q_weight, const void* k_weight, float eps,
                                   const void* cos_table, const void* sin_table, int32_t table_rows, void* q_out, void* k_out,
                                   void* stream) {
  MSA_REQUIRE(q && k && q_weight && k_weight && cos_table && sin_table && q_out && k_out, "heads_norm_rope: null pointer");
  MSA_REQUIRE(head_dim == 128, "heads_norm_rope: head_dim must be 128");
  MSA_REQUIRE(n_rows >= 0 && n_q_heads > 0 && n_kv_heads > 0 && q_stride % 4 == 0 && k_stride % 4 == 0, "heads_norm_rope: bad sizes");
  MSA_REQUIRE(table_rows > 0 && n_rows % table_rows == 0, "heads_norm_rope: the rows must be a multiple of the tables' rows");
  MSA_REQUIRE(aligned8(q) && aligned8(k) && aligned8(q_weight) && aligned8(k_weight) && aligned8(q_out) && aligned8(k_out) &&
                  aligned8(cos_table) && aligned8(sin_table), "heads_norm_rope: pointers must be 8-byte aligned");
  MSA_REQUIRE((long long)n_rows * (n_q_heads + n_kv_heads) < (1ll << 31), "heads_norm_rope: too many rows");
  if (n_rows == 0) return MSA_OK;
  const HeadsNormRope p = {(const __nv_bfloat16*)q, (const __nv_bfloat16*)k, q_stride, k_stride, n_rows, n_q_heads, n_kv_heads, table_rows,
                           (const __nv_bfloat16*)q_weight, (const __nv_bfloat16*)k_weight, (const __nv_bfloat16*)cos_table,
                           (const __nv_bfloat16*)sin_table, (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_out, eps};
  return launch_heads_norm_rope(p, stream);
}

extern "C" int msa_qk_norm_rope(const void* qkv, int64_t row_stride, int32_t n_seq, int32_t n_q_heads,
                                int32_t n_kv_heads, int32_t head_dim, const void* q_weight, const void* k_weight,
                                float eps, const void* cos_table, const void* sin_table, void* q_out, void* k_out,
                                void* stream) {
  MSA_REQUIRE(qkv, "qk_norm_rope: null pointer");
  MSA_REQUIRE(n_seq >= 0 && n_q_heads > 0, "qk_norm_rope: bad sizes");
  return msa_heads_norm_rope(qkv, row_stride, (const __nv_bfloat16*)qkv + (long long)n_q_heads * 128, row_stride, n_seq, n_q_heads, n_kv_heads,
                             head_dim, q_weight, k_weight, eps, cos_table, sin_table, n_seq > 0 ? n_seq : 1, q_out, k_out, stream);
}

extern "C" int msa_add_rmsnorm(const void* x, const void* y, const void* weight, float eps, int32_t n_rows,
                               int32_t hidden, void* x_out, void* h_out, void* stream) {
  MSA_REQUIRE(x && weight && h_out, "add_rmsnorm: null pointer");
  MSA_REQUIRE(n_rows >= 0 && hidden > 0 && hidden % 2 == 0 && hidden <= 12288, "add_rmsnorm: hidden must be even and <= 12288");
  MSA_REQUIRE(aligned4(x) && aligned4(y) && aligned4(weight) && aligned4(x_out) && aligned4(h_out), "add_rmsnorm: pointers must be 4-byte aligned");
  if (n_rows == 0) return MSA_OK;
  const bool vec = hidden % 8 == 0 && aligned16(x) && aligned16(y) && aligned16(weight) && aligned16(x_out) && aligned16(h_out);
  // A warp per row from the row count on that gives every SM eight of them.
  int n_sm = 0;
  MSA_OK_OR_RETURN(device_sm_count(&n_sm));
  const bool many = n_rows >= 8 * n_sm;
#define MSA_ADD_RMSNORM(T, NV) launch_add_rmsnorm<T, NV>(x, y, weight, eps, n_rows, hidden, x_out, h_out, stream)
  if (vec && many && hidden <= 4096) {
    if (hidden <= 1024) MSA_ADD_RMSNORM(32, 4);
    else if (hidden <= 2048) MSA_ADD_RMSNORM(32, 8);
    else if (hidden <= 2560) MSA_ADD_RMSNORM(32, 10);
    else if (hidden <= 3072) MSA_ADD_RMSNORM(32, 12);
    else MSA_ADD_RMSNORM(32, 16);
  } else if (vec) {
    if (hidden <= 2048) MSA_ADD_RMSNORM(256, 1);
    else if (hidden <= 4096) MSA_ADD_RMSNORM(256, 2);
    else if (hidden <= 8192) MSA_ADD_RMSNORM(256, 4);
    else MSA_ADD_RMSNORM(256, 6);
  } else {
    add_rmsnorm_pairs_kernel<<<n_rows, 256, hidden * sizeof(float), (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)x, (const __nv_bfloat16*)y, (const __nv_bfloat16*)weight, eps, hidden, (__nv_bfloat16*)x_out,
        (__nv_bfloat16*)h_out);
  }
#undef MSA_ADD_RMSNORM
  MSA_LAUNCH_OK("add_rmsnorm_kernel");
  return MSA_OK;
}

extern "C" int msa_silu_mul_parts(const void* gate, int64_t gate_stride, const void* up, int64_t up_stride, int32_t n_rows, int32_t ffn,
                                  void* out, void* stream) {
  MSA_REQUIRE(gate && up && out, "silu_mul: null pointer");
  MSA_REQUIRE(n_rows >= 0 && ffn > 0 && ffn % 2 == 0 && gate_stride % 2 == 0 && up_stride % 2 == 0, "silu_mul: ffn and the row strides must be even");
  MSA_REQUIRE(aligned4(gate) && aligned4(up) && aligned4(out), "silu_mul: pointers must be 4-byte aligned");
  if (n_rows == 0) return MSA_OK;
  const bool vec = ffn % 8 == 0 && gate_stride % 8 == 0 && up_stride % 8 == 0 && aligned16(gate) && aligned16(up) && aligned16(out);
  const long long grid = ((long long)n_rows * (ffn / (vec ? 8 : 2)) + 1023) / 1024;
  MSA_REQUIRE(grid < (1ll << 31), "silu_mul: too many rows");
  auto launch = [&](auto kernel) {
    kernel<<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)gate, gate_stride, (const __nv_bfloat16*)up, up_stride, ffn,
                                                             n_rows, (__nv_bfloat16*)out);
  };
  if (vec) launch(silu_mul_kernel<8>);
  else launch(silu_mul_kernel<2>);
  MSA_LAUNCH_OK("silu_mul_kernel");
  return MSA_OK;
}

extern "C" int msa_silu_mul(const void* gate_up, int64_t row_stride, int32_t n_rows, int32_t ffn, void* out, void* stream) {
  MSA_REQUIRE(gate_up && ffn > 0, "silu_mul: null pointer or bad sizes");
  return msa_silu_mul_parts(gate_up, row_stride, (const __nv_bfloat16*)gate_up + ffn, row_stride, n_rows, ffn, out, stream);
}

extern "C" int msa_rope_table(const int64_t* positions, const float* inv_freq, int32_t n, int32_t half, float scaling, void* cos_table,
                              void* sin_table, void* stream) {
  MSA_REQUIRE(positions && inv_freq && cos_table && sin_table, "rope_table: null pointer");
  MSA_REQUIRE(n >= 0 && half > 0, "rope_table: bad sizes");
  if (n == 0) return MSA_OK;
  const long long grid = ((long long)n * half + 255) / 256;
  MSA_REQUIRE(grid < (1ll << 31), "rope_table: too many positions");
  rope_table_kernel<<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(positions, inv_freq, n, half, scaling, (__nv_bfloat16*)cos_table,
                                                                      (__nv_bfloat16*)sin_table);
  MSA_LAUNCH_OK("rope_table_kernel");
  return MSA_OK;
}
