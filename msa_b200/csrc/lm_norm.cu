// Residual stream (fp32), the norms on either side of a sublayer, the embedding (with a hashed bigram table), the dense
// feed-forward's gate and the cap of the logits.  One launch between two matrix products: branch norm, residual add, next
// norm (two of them where two branches read the same stream), rounding for the next product.
#include <climits>

#include "lm_common.cuh"

namespace msa {

struct ResNormParams {
  const float* base; long long base_stride;
  const void* y; int32_t y_dtype; long long y_stride;
  const int32_t* inv; const float* mix; int32_t top;
  const float* w_branch; const float* w_next; float eps;
  const int32_t* rows; int32_t width;
  float* x_out; void* h_out; void* cat_out; long long cat_stride;
  const float* add;                            // further rows [n, width] that join the stream (null: none)
  const float* w_next2; void* h_out2;          // a second norm of the same stream
};

template <typename TY>
__device__ __forceinline__ float4 branch4(const ResNormParams& p, long long r, int i) {
  const TY* y = reinterpret_cast<const TY*>(p.y);
  if (!p.inv) return load4(y + r * p.y_stride + i);
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k = 0; k < p.top; ++k) {
    const float w = p.mix[r * p.top + k];
    const float4 v = load4(y + (long long)p.inv[r * p.top + k] * p.y_stride + i);
    a.x = fmaf(w, v.x, a.x); a.y = fmaf(w, v.y, a.y); a.z = fmaf(w, v.z, a.z); a.w = fmaf(w, v.w, a.w);
  }
  return a;
}
template <typename TY>
__device__ __forceinline__ float branch1(const ResNormParams& p, long long r, int i) {
  const TY* y = reinterpret_cast<const TY*>(p.y);
  if (!p.inv) return to_f(y[r * p.y_stride + i]);
  float a = 0.f;
  for (int k = 0; k < p.top; ++k)
    a = fmaf(p.mix[r * p.top + k], to_f(y[(long long)p.inv[r * p.top + k] * p.y_stride + i]), a);
  return a;
}

// Rows above 4096 columns and odd ones.  V = 4: every row pointer is 4-element aligned and width % 4 == 0; V = 1: any width.
template <typename T, typename TY, int V>
__global__ void residual_norm_kernel(const ResNormParams p) {
  extern __shared__ float s_row[];   // [width]
  __shared__ float s_part[32];
  const long long r = blockIdx.x;
  const long long rb = p.rows ? p.rows[r] : r;
  const int nt = blockDim.x;
  T* h_out = reinterpret_cast<T*>(p.h_out);
  T* h_out2 = reinterpret_cast<T*>(p.h_out2);
  T* cat = reinterpret_cast<T*>(p.cat_out);
  float scale_b = 1.f;
  if (p.y && p.w_branch) {
    float ss = 0.f;
    for (int i = threadIdx.x * V; i < p.width; i += nt * V) {
      if constexpr (V == 4) {
        const float4 b = branch4<TY>(p, r, i);
        store4(s_row + i, b);
        ss += b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w;
      } else {
        const float b = branch1<TY>(p, r, i);
        s_row[i] = b;
        ss += b * b;
      }
    }
    scale_b = 1.f / sqrtf(block_sum(ss, s_part) / (float)p.width + p.eps);
  }
  float ss = 0.f;
  for (int i = threadIdx.x * V; i < p.width; i += nt * V) {   // every thread revisits the elements it stored above
    if constexpr (V == 4) {
      float4 x = p.base ? load4(p.base + rb * p.base_stride + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      if (p.y) {
        if (p.w_branch) {
          const float4 b = load4(s_row + i), w = load4(p.w_branch + i);
          x.x += b.x * scale_b * w.x; x.y += b.y * scale_b * w.y; x.z += b.z * scale_b * w.z; x.w += b.w * scale_b * w.w;
        } else {
          const float4 b = branch4<TY>(p, r, i);
          x.x += b.x; x.y += b.y; x.z += b.z; x.w += b.w;
        }
      }
      if (p.add) {
        const float4 b = load4(p.add + r * p.width + i);
        x.x += b.x; x.y += b.y; x.z += b.z; x.w += b.w;
      }
      if (p.x_out) store4(p.x_out + r * p.width + i, x);
      if (cat) store4(cat + r * p.cat_stride + i, x);
      store4(s_row + i, x);
      ss += x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
    } else {
      float x = p.base ? p.base[rb * p.base_stride + i] : 0.f;
      if (p.y) x += p.w_branch ? s_row[i] * scale_b * p.w_branch[i] : branch1<TY>(p, r, i);
      if (p.add) x += p.add[r * p.width + i];
      if (p.x_out) p.x_out[r * p.width + i] = x;
      if (cat) cat[r * p.cat_stride + i] = from_f<T>(x);
      s_row[i] = x;
      ss += x * x;
    }
  }
  if (!h_out) return;
  const float inv = 1.f / sqrtf(block_sum(ss, s_part) / (float)p.width + p.eps);
  for (int i = threadIdx.x * V; i < p.width; i += nt * V) {
    if constexpr (V == 4) {
      const float4 x = load4(s_row + i), w = load4(p.w_next + i);
      store4(h_out + r * p.width + i, make_float4(x.x * inv * w.x, x.y * inv * w.y, x.z * inv * w.z, x.w * inv * w.w));
      if (h_out2) {
        const float4 w2 = load4(p.w_next2 + i);
        store4(h_out2 + r * p.width + i, make_float4(x.x * inv * w2.x, x.y * inv * w2.y, x.z * inv * w2.z, x.w * inv * w2.w));
      }
    } else {
      h_out[r * p.width + i] = from_f<T>(s_row[i] * inv * p.w_next[i]);
      if (h_out2) h_out2[r * p.width + i] = from_f<T>(s_row[i] * inv * p.w_next2[i]);
    }
  }
}

// The same for rows that a block of width / 4 threads covers in one pass (everything in registers, all loads in flight
// before the first reduction): a decode step has few rows and waits for latency, not for bandwidth.
template <typename T, typename TY>
__global__ void __launch_bounds__(1024) residual_norm_once_kernel(const ResNormParams p) {
  let_product_start(gridDim.x);
  grid_dependency_wait();
  __shared__ float s_part[32];
  const long long r = blockIdx.x;
  const long long rb = p.rows ? p.rows[r] : r;
  const int i = threadIdx.x * 4;
  const bool on = i < p.width;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 x = on && p.base ? load4(p.base + rb * p.base_stride + i) : zero;
  const float4 wb = on && p.w_branch ? load4(p.w_branch + i) : zero;
  const float4 wn = on && p.h_out ? load4(p.w_next + i) : zero;
  const float4 wn2 = on && p.h_out2 ? load4(p.w_next2 + i) : zero;
  const float4 more = on && p.add ? load4(p.add + r * p.width + i) : zero;
  float4 b = zero;
  if (p.y && on) {
    const TY* y = reinterpret_cast<const TY*>(p.y);
    if (p.inv) {
      for (int k0 = 0; k0 < p.top; k0 += 4) {
        float4 v[4];
        float w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const bool in = k0 + k < p.top;
          w[k] = in ? p.mix[r * p.top + k0 + k] : 0.f;
          v[k] = in ? load4(y + (long long)p.inv[r * p.top + k0 + k] * p.y_stride + i) : zero;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          b.x = fmaf(w[k], v[k].x, b.x); b.y = fmaf(w[k], v[k].y, b.y); b.z = fmaf(w[k], v[k].z, b.z); b.w = fmaf(w[k], v[k].w, b.w);
        }
      }
    } else {
      b = load4(y + r * p.y_stride + i);
    }
  }
  if (p.y && p.w_branch) {
    const float sc = 1.f / sqrtf(block_sum(b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w, s_part) / (float)p.width + p.eps);
    x.x += b.x * sc * wb.x; x.y += b.y * sc * wb.y; x.z += b.z * sc * wb.z; x.w += b.w * sc * wb.w;
  } else {
    x.x += b.x; x.y += b.y; x.z += b.z; x.w += b.w;
  }
  x.x += more.x; x.y += more.y; x.z += more.z; x.w += more.w;
  if (on && p.x_out) store4(p.x_out + r * p.width + i, x);
  if (on && p.cat_out) store4(reinterpret_cast<T*>(p.cat_out) + r * p.cat_stride + i, x);
  if (!p.h_out) return;
  const float inv = 1.f / sqrtf(block_sum(x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w, s_part) / (float)p.width + p.eps);
  if (on) store4(reinterpret_cast<T*>(p.h_out) + r * p.width + i, make_float4(x.x * inv * wn.x, x.y * inv * wn.y, x.z * inv * wn.z, x.w * inv * wn.w));
  if (on && p.h_out2)
    store4(reinterpret_cast<T*>(p.h_out2) + r * p.width + i, make_float4(x.x * inv * wn2.x, x.y * inv * wn2.y, x.z * inv * wn2.z, x.w * inv * wn2.w));
}

// The same for many rows, E vectors per thread in registers, all of a row's loads in flight before the first reduction.  12 bytes per
// element (base and stream in 32 bits, branch and norm in 16).  One vector at a time through shared memory took 47.1 us for 6236 x 2048
// from a cold L2, this takes 39.9; the bytes alone take 24 at HBM's rate.  What bounds it is the issue of instructions (63 % of the slots, DRAM
// 36 %): two sums over the block per row and four conversions per vector.
// Threads and order of the sums are those of residual_norm_kernel above, bit for bit.  That holds from 513 rows on: up to 512 rows
// residual_norm_once_kernel sums in another order, and products of up to 8 rows (rows_gemm_kernel) do too, so the last bits
// of a position, and its experts where two of them tie, do depend on the number of rows beside it.
template <typename T, typename TY, int E>
__global__ void __launch_bounds__(256) residual_norm_rows_kernel(const ResNormParams p) {
  __shared__ float s_part[2][32];
  const long long r = blockIdx.x;
  const long long rb = p.rows ? p.rows[r] : r;
  const int nt = blockDim.x, lane = threadIdx.x & 31, warps = nt >> 5;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto at = [&](int e) { return (e * nt + (int)threadIdx.x) * 4; };
  auto sum = [&](float v, float* part) {             // block_sum with a buffer for each of the two reductions
    v = warp_sum_f(v);
    if (lane == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = 0.f;
    for (int i = 0; i < warps; ++i) t += part[i];
    return t;
  };
  float4 x[E], b[E];
#pragma unroll
  for (int e = 0; e < E; ++e) x[e] = p.base && at(e) < p.width ? load4(p.base + rb * p.base_stride + at(e)) : zero;
  if (p.y) {
#pragma unroll
    for (int e = 0; e < E; ++e) b[e] = at(e) < p.width ? branch4<TY>(p, r, at(e)) : zero;
    if (p.w_branch) {
      float ss = 0.f;
#pragma unroll
      for (int e = 0; e < E; ++e) ss += b[e].x * b[e].x + b[e].y * b[e].y + b[e].z * b[e].z + b[e].w * b[e].w;
      const float sc = 1.f / sqrtf(sum(ss, s_part[0]) / (float)p.width + p.eps);
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const float4 w = at(e) < p.width ? load4(p.w_branch + at(e)) : zero;
        x[e].x += b[e].x * sc * w.x; x[e].y += b[e].y * sc * w.y; x[e].z += b[e].z * sc * w.z; x[e].w += b[e].w * sc * w.w;
      }
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) { x[e].x += b[e].x; x[e].y += b[e].y; x[e].z += b[e].z; x[e].w += b[e].w; }
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    if (at(e) >= p.width) continue;
    if (p.add) {
      const float4 a = load4(p.add + r * p.width + at(e));
      x[e].x += a.x; x[e].y += a.y; x[e].z += a.z; x[e].w += a.w;
    }
    if (p.x_out) store4(p.x_out + r * p.width + at(e), x[e]);
    if (p.cat_out) store4(reinterpret_cast<T*>(p.cat_out) + r * p.cat_stride + at(e), x[e]);
    ss += x[e].x * x[e].x + x[e].y * x[e].y + x[e].z * x[e].z + x[e].w * x[e].w;
  }
  if (!p.h_out) return;
  const float inv = 1.f / sqrtf(sum(ss, s_part[1]) / (float)p.width + p.eps);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    if (at(e) >= p.width) continue;
    const float4 w = load4(p.w_next + at(e));
    store4(reinterpret_cast<T*>(p.h_out) + r * p.width + at(e), make_float4(x[e].x * inv * w.x, x[e].y * inv * w.y, x[e].z * inv * w.z, x[e].w * inv * w.w));
    if (p.h_out2) {
      const float4 w2 = load4(p.w_next2 + at(e));
      store4(reinterpret_cast<T*>(p.h_out2) + r * p.width + at(e),
             make_float4(x[e].x * inv * w2.x, x[e].y * inv * w2.y, x[e].z * inv * w2.z, x[e].w * inv * w2.w));
    }
  }
}

// V = 4: rows and pointers are 4-element aligned; V = 1: any width.
template <typename T, int V>
__global__ void embed_kernel(const msa_lm_embed_args a) {
  let_product_start(gridDim.x);
  extern __shared__ float s_row[];
  __shared__ float s_part[32];
  const long long r = blockIdx.x;
  const int width = a.width;
  int tok = a.token[r];
  if (tok < 0 || tok >= a.vocab) {
    if (threadIdx.x == 0 && a.status) atomicAdd(a.status + 2, 1);
    tok = 0;
  }
  const T* src = reinterpret_cast<const T*>(a.table) + (long long)tok * width;
  const T* pair = nullptr;
  if (a.pair_table) {
    const int s = a.tok_seq[r], t = (int)r - a.cu[s], slot = a.slot[s];
    long long row = a.buckets;
    if (t > 0 || a.start[s] > 0) {
      int prev = t > 0 ? a.token[r - 1] : a.last_token[slot];
      if (prev < 0 || prev >= a.vocab) prev = 0;
      row = ((long long)prev * a.mul_prev + (long long)tok * a.mul_cur) % a.buckets;
      if (row < 0) row += a.buckets;
    }
    pair = reinterpret_cast<const T*>(a.pair_table) + row * width;
    __syncthreads();                             // every thread has read the sequence's previous token
    if (t == 0 && threadIdx.x == 0) a.last_token[slot] = a.token[a.cu[s + 1] - 1];
  }
  T* cat0 = reinterpret_cast<T*>(a.cat0);
  T* cat1 = reinterpret_cast<T*>(a.cat1);
  float ss = 0.f;
  for (int i = threadIdx.x * V; i < width; i += blockDim.x * V) {
    if constexpr (V == 4) {
      float4 x = load4(src + i);
      if (pair) { const float4 y = load4(pair + i); x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w; }
      store4(a.x_out + r * width + i, x);
      if (a.x_copy) store4(a.x_copy + r * width + i, x);
      if (cat0) store4(cat0 + r * a.cat_stride + i, x);
      if (cat1) store4(cat1 + r * a.cat_stride + i, x);
      store4(s_row + i, x);
      ss += x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
    } else {
      float x = to_f(src[i]);
      if (pair) x += to_f(pair[i]);
      a.x_out[r * width + i] = x;
      if (a.x_copy) a.x_copy[r * width + i] = x;
      if (cat0) cat0[r * a.cat_stride + i] = from_f<T>(x);
      if (cat1) cat1[r * a.cat_stride + i] = from_f<T>(x);
      s_row[i] = x;
      ss += x * x;
    }
  }
  if (!a.h_out) return;
  T* h = reinterpret_cast<T*>(a.h_out);
  T* h2 = reinterpret_cast<T*>(a.h_out2);
  const float inv = 1.f / sqrtf(block_sum(ss, s_part) / (float)width + a.eps);
  for (int i = threadIdx.x * V; i < width; i += blockDim.x * V) {
    if constexpr (V == 4) {
      const float4 x = load4(s_row + i), w = load4(a.w_next + i);
      store4(h + r * width + i, make_float4(x.x * inv * w.x, x.y * inv * w.y, x.z * inv * w.z, x.w * inv * w.w));
      if (h2) {
        const float4 w2 = load4(a.w_next2 + i);
        store4(h2 + r * width + i, make_float4(x.x * inv * w2.x, x.y * inv * w2.y, x.z * inv * w2.z, x.w * inv * w2.w));
      }
    } else {
      h[r * width + i] = from_f<T>(s_row[i] * inv * a.w_next[i]);
      if (h2) h2[r * width + i] = from_f<T>(s_row[i] * inv * a.w_next2[i]);
    }
  }
}

// x = cap * tanh(x / cap), in place.
__global__ void __launch_bounds__(256) softcap_kernel(float* x, long long n, float cap) {
  grid_dependency_wait();
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) x[i] = cap * tanhf(x[i] / cap);
}

// Place of the largest entry of a row (NaN counts as the largest, equals go to the lowest place).  One block per row, eight
// 16-byte loads in flight per thread: bound by what one SM draws from L2 (8 x 32768: 5.3 us; a general reduction and the
// conversion of its 64-bit places took 12.3 us).
__device__ __forceinline__ bool larger(float a, int ia, float b, int ib) {
  const bool na = a != a, nb = b != b;
  if (na != nb) return na;
  return a > b || ((a == b || na) && ia < ib);
}
__global__ void __launch_bounds__(1024) argmax_kernel(const float* __restrict__ x, long long stride, int cols, bool vec, int32_t* __restrict__ out) {
  __shared__ float s_v[32];
  __shared__ int s_i[32];
  const float* row = x + blockIdx.x * stride;
  float best = -INFINITY;
  int at = INT_MAX;                                    // nothing yet: loses to every entry
  auto take = [&](float v, int i) { if (larger(v, i, best, at)) { best = v; at = i; } };
  int done = 0;
  if (vec) {
    done = cols & ~3;
    int i = threadIdx.x * 4;
    for (; i + 7 * 4096 < done; i += 8 * 4096) {
      float4 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = load4(row + i + k * 4096);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int c = i + k * 4096;
        take(v[k].x, c); take(v[k].y, c + 1); take(v[k].z, c + 2); take(v[k].w, c + 3);
      }
    }
    for (; i < done; i += 4096) {
      const float4 v = load4(row + i);
      take(v.x, i); take(v.y, i + 1); take(v.z, i + 2); take(v.w, i + 3);
    }
  }
  for (int i = done + threadIdx.x; i < cols; i += 1024) take(row[i], i);
  auto reduce = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float v = __shfl_xor_sync(0xffffffffu, best, o);
      const int i = __shfl_xor_sync(0xffffffffu, at, o);
      take(v, i);
    }
  };
  reduce();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { s_v[warp] = best; s_i[warp] = at; }
  __syncthreads();
  if (warp != 0) return;
  best = s_v[lane];
  at = s_i[lane];
  reduce();
  if (lane == 0) out[blockIdx.x] = at;
}

// out[r, part * cols + c] = part-th share of tanh(x[r, c]): with two parts the bf16 rounding and what it leaves behind,
// so that a product over both keeps 16 significant bits.
template <typename T>
__global__ void __launch_bounds__(256) tanh_split_kernel(const float* x, int cols, int parts, long long n, T* __restrict__ out) {
  if (n <= (long long)kEarlyRows * cols) grid_launch_dependents();
  grid_dependency_wait();
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
    const long long r = i / cols;
    const int c = (int)(i - r * cols);
    float v = tanhf(x[i]);
    for (int k = 0; k < parts; ++k) {
      const T part = from_f<T>(v);
      out[(r * parts + k) * cols + c] = part;
      v -= to_f(part);
    }
  }
}

// Row r of h beside row r-1 of its sequence (of the previous step: from `shift`): out[m, r] = h + (before - h) * mu[m].
// The block of a sequence's first row hands the step's last row over to `shift`.
template <typename T, int V>
__global__ void token_shift_kernel(const T* __restrict__ h, const float* __restrict__ mu, int n_mix, int n_tok, int width,
                                   const int32_t* __restrict__ tok_seq, const int32_t* __restrict__ slot,
                                   const int32_t* __restrict__ start, const int32_t* __restrict__ cu, T* shift, T* __restrict__ out) {
  let_product_start(gridDim.x);
  const long long r = blockIdx.x;
  const int s = tok_seq[r], t = (int)r - cu[s];
  T* state = shift + (long long)slot[s] * width;
  const bool from_state = t == 0, none = from_state && start[s] == 0;
  const T* before = from_state ? state : h + (r - 1) * width;
  const T* last = h + (long long)(cu[s + 1] - 1) * width;
  for (int i = (blockIdx.y * blockDim.x + threadIdx.x) * V; i < width; i += gridDim.y * blockDim.x * V) {
    if constexpr (V == 4) {
      const float4 x = load4(h + r * width + i);
      float4 d = none ? make_float4(0.f, 0.f, 0.f, 0.f) : load4(before + i);
      if (from_state) store4(state + i, load4(last + i));
      d.x -= x.x; d.y -= x.y; d.z -= x.z; d.w -= x.w;
      for (int m = 0; m < n_mix; ++m) {
        const float4 w = load4(mu + (long long)m * width + i);
        store4(out + ((long long)m * n_tok + r) * width + i,
               make_float4(fmaf(d.x, w.x, x.x), fmaf(d.y, w.y, x.y), fmaf(d.z, w.z, x.z), fmaf(d.w, w.w, x.w)));
      }
    } else {
      const float x = to_f(h[r * width + i]), d = (none ? 0.f : to_f(before[i])) - x;
      if (from_state) state[i] = last[i];
      for (int m = 0; m < n_mix; ++m) out[((long long)m * n_tok + r) * width + i] = from_f<T>(fmaf(d, mu[(long long)m * width + i], x));
    }
  }
}

// V = 8: 16-byte loads (bf16); V = 4: 8- or 16-byte ones; V = 1: any alignment.  A block takes 256 * V columns of a row.  Bound by the issue of
// instructions (74 % of the slots, DRAM 61 %): the exponential and the quotient are exact.  With 8-byte loads and an index division
// by a run-time number 6236 x 6144 took 57.5 us from a cold L2, now 40.2; the bytes alone take 35.6 at HBM's rate.  (A chain of such
// launches from a graph.)  Approximate exponentials gave 2 us more, but their last bits decide between experts that tie.
template <typename T, int V>
__global__ void __launch_bounds__(256)
lm_silu_mul_kernel(const T* __restrict__ gu, long long stride, int ff, T* __restrict__ out, long long out_stride) {
  const int j = (blockIdx.x * 256 + threadIdx.x) * V;
  if (j >= ff) return;
  const T *g = gu + blockIdx.y * stride + j, *u = g + ff;
  T* o = out + blockIdx.y * out_stride + j;
  if constexpr (V == 8) {
    const uint4 gv = *reinterpret_cast<const uint4*>(g), uv = *reinterpret_cast<const uint4*>(u);
    const __nv_bfloat162 *a = reinterpret_cast<const __nv_bfloat162*>(&gv), *b = reinterpret_cast<const __nv_bfloat162*>(&uv);
    uint4 ov;
    __nv_bfloat162* c = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = __bfloat1622float2(a[i]), y = __bfloat1622float2(b[i]);
      c[i] = __floats2bfloat162_rn(silu_f(x.x) * y.x, silu_f(x.y) * y.y);
    }
    *reinterpret_cast<uint4*>(o) = ov;
  } else if constexpr (V == 4) {
    const float4 x = load4(g), y = load4(u);
    store4(o, make_float4(silu_f(x.x) * y.x, silu_f(x.y) * y.y, silu_f(x.z) * y.z, silu_f(x.w) * y.w));
  } else {
    *o = from_f<T>(silu_f(to_f(*g)) * to_f(*u));
  }
}

inline int row_threads(int width) { return width >= 2048 ? 256 : (width >= 512 ? 128 : 64); }
inline bool vec4_ok(const void* p, int elem) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) % (4 * elem)) == 0; }

}  // namespace msa

using namespace msa;

extern "C" int msa_lm_residual_norm(const float* base, int64_t base_stride, const void* y, int32_t y_dtype,
                                    int64_t y_stride, const int32_t* inv, const float* mix, int32_t top,
                                    const float* w_branch, const float* w_next, float eps, const int32_t* rows,
                                    int32_t n_rows, int32_t width, float* x_out, void* h_out, void* cat_out,
                                    int64_t cat_stride, const float* add, const float* w_next2, void* h_out2, int32_t dtype,
                                    void* stream) {
  MSA_REQUIRE(dtype_ok(dtype) && (!y || dtype_ok(y_dtype)), "residual_norm: bad dtype");
  MSA_REQUIRE(n_rows >= 0 && width > 0 && width <= 12000, "residual_norm: width must be 1..12000");
  MSA_REQUIRE(base || y, "residual_norm: neither base nor branch");
  MSA_REQUIRE(!h_out || w_next, "residual_norm: h_out needs w_next");
  MSA_REQUIRE(!h_out2 || (h_out && w_next2), "residual_norm: h_out2 needs h_out and w_next2");
  MSA_REQUIRE(!inv || (mix && top > 0 && y), "residual_norm: a mixture needs weights and top > 0");
  if (n_rows == 0) return MSA_OK;
  ResNormParams p{base, base_stride, y, y_dtype, y_stride, inv, mix, top, w_branch, w_next, eps, rows, width, x_out, h_out,
                  cat_out, cat_stride, add, w_next2, h_out2};
  const int e = (int)dtype_size(dtype), ey = (int)dtype_size(y_dtype);
  const bool v4 = width % 4 == 0 && base_stride % 4 == 0 && (!y || y_stride % 4 == 0) && (!cat_out || cat_stride % 4 == 0) &&
                  vec4_ok(base, 4) && vec4_ok(y, ey) && vec4_ok(w_branch, 4) && vec4_ok(w_next, 4) && vec4_ok(x_out, 4) &&
                  vec4_ok(h_out, e) && vec4_ok(cat_out, e) && vec4_ok(add, 4) && vec4_ok(w_next2, 4) && vec4_ok(h_out2, e);
  cudaStream_t st = (cudaStream_t)stream;
  if (v4 && width <= 4096 && n_rows <= 512) {
    const int once = (width / 4 + 31) / 32 * 32;
    MSA_LM_DISPATCH(dtype, {
      auto kernel = y && y_dtype == MSA_BF16 ? residual_norm_once_kernel<T, __nv_bfloat16> : residual_norm_once_kernel<T, float>;
      MSA_CUDA_OK(launch_kernel_pdl(kernel, dim3(n_rows), dim3(once), 0, st, n_rows <= kEarlyRows && !inv, p));   // inv: behind the experts
    });
    MSA_LAUNCH_OK("residual_norm_once_kernel");
    return MSA_OK;
  }
  const int threads = row_threads(width);
  const int vectors = (width / 4 + threads - 1) / threads;
  if (v4 && vectors <= 4) {                            // beyond, the registers leave too few rows in flight (8192: 33.8 us against 20.5)
    MSA_LM_DISPATCH(dtype, {
      const bool half = y && y_dtype == MSA_BF16;
      auto launch = [&](auto with_half, auto with_float) { half ? with_half<<<n_rows, threads, 0, st>>>(p) : with_float<<<n_rows, threads, 0, st>>>(p); };
      if (vectors <= 2) launch(residual_norm_rows_kernel<T, __nv_bfloat16, 2>, residual_norm_rows_kernel<T, float, 2>);
      else launch(residual_norm_rows_kernel<T, __nv_bfloat16, 4>, residual_norm_rows_kernel<T, float, 4>);
    });
    MSA_LAUNCH_OK("residual_norm_rows_kernel");
    return MSA_OK;
  }
  const size_t smem = (size_t)width * 4;
  MSA_LM_DISPATCH(dtype, {
    if (y && y_dtype == MSA_BF16) {
      if (v4) residual_norm_kernel<T, __nv_bfloat16, 4><<<n_rows, threads, smem, st>>>(p);
      else residual_norm_kernel<T, __nv_bfloat16, 1><<<n_rows, threads, smem, st>>>(p);
    } else {
      if (v4) residual_norm_kernel<T, float, 4><<<n_rows, threads, smem, st>>>(p);
      else residual_norm_kernel<T, float, 1><<<n_rows, threads, smem, st>>>(p);
    }
  });
  MSA_LAUNCH_OK("residual_norm_kernel");
  return MSA_OK;
}

extern "C" int msa_lm_embed(const msa_lm_embed_args* args, void* stream) {
  MSA_REQUIRE(args, "embed: null arguments");
  const msa_lm_embed_args a = *args;
  MSA_REQUIRE(dtype_ok(a.dtype) && a.table && a.token && a.x_out, "embed: bad arguments");
  MSA_REQUIRE(a.n_rows >= 0 && a.width > 0 && a.width <= 12000 && a.vocab > 0, "embed: bad sizes");
  MSA_REQUIRE((!a.h_out || a.w_next) && (!a.h_out2 || (a.h_out && a.w_next2)), "embed: a norm needs its weight");
  MSA_REQUIRE(!a.pair_table || (a.buckets > 0 && a.last_token && a.tok_seq && a.slot && a.start && a.cu), "embed: a pair table needs the step's tables");
  if (a.n_rows == 0) return MSA_OK;
  const int e = (int)dtype_size(a.dtype);
  const bool v4 = a.width % 4 == 0 && a.cat_stride % 4 == 0 && vec4_ok(a.table, e) && vec4_ok(a.pair_table, e) && vec4_ok(a.x_out, 4) &&
                  vec4_ok(a.x_copy, 4) && vec4_ok(a.h_out, e) && vec4_ok(a.h_out2, e) && vec4_ok(a.cat0, e) && vec4_ok(a.cat1, e) &&
                  vec4_ok(a.w_next, 4) && vec4_ok(a.w_next2, 4);
  const size_t smem = (size_t)a.width * 4;
  MSA_LM_DISPATCH(a.dtype, {
    if (v4) embed_kernel<T, 4><<<a.n_rows, row_threads(a.width), smem, (cudaStream_t)stream>>>(a);
    else embed_kernel<T, 1><<<a.n_rows, row_threads(a.width), smem, (cudaStream_t)stream>>>(a);
  });
  MSA_LAUNCH_OK("embed_kernel");
  return MSA_OK;
}

namespace {
inline int flat_grid(long long n) { return (int)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16); }
}  // namespace

extern "C" int msa_lm_softcap(float* x, int64_t n, float cap, void* stream) {
  MSA_REQUIRE(x && n >= 0 && cap > 0.f, "softcap: bad arguments");
  if (n == 0) return MSA_OK;
  MSA_CUDA_OK(launch_kernel_pdl(softcap_kernel, dim3(flat_grid(n)), dim3(256), 0, (cudaStream_t)stream, true, x, (long long)n, cap));
  MSA_LAUNCH_OK("softcap_kernel");
  return MSA_OK;
}

extern "C" int msa_lm_argmax(const float* x, int64_t stride, int32_t n_rows, int32_t cols, int32_t* out, void* stream) {
  MSA_REQUIRE(x && out && n_rows >= 0 && cols > 0, "argmax: bad arguments");
  if (n_rows == 0) return MSA_OK;
  argmax_kernel<<<n_rows, 1024, 0, (cudaStream_t)stream>>>(x, stride, cols, aligned16(x) && stride % 4 == 0, out);
  MSA_LAUNCH_OK("argmax_kernel");
  return MSA_OK;
}

extern "C" int msa_lm_tanh_split(const float* x, int32_t n_rows, int32_t cols, int32_t parts, void* out, int32_t dtype, void* stream) {
  MSA_REQUIRE(dtype_ok(dtype) && x && out && n_rows >= 0 && cols > 0 && parts >= 1, "tanh_split: bad arguments");
  const long long n = (long long)n_rows * cols;
  if (n == 0) return MSA_OK;
  MSA_LM_DISPATCH(dtype, {
    MSA_CUDA_OK(launch_kernel_pdl(tanh_split_kernel<T>, dim3(flat_grid(n)), dim3(256), 0, (cudaStream_t)stream, n <= (long long)kEarlyRows * cols,
                                  x, cols, parts, (long long)n, (T*)out));
  });
  MSA_LAUNCH_OK("tanh_split_kernel");
  return MSA_OK;
}

extern "C" int msa_lm_token_shift(const void* h, const float* mu, int32_t n_mix, int32_t n_tok, int32_t width, const int32_t* tok_seq,
                                  const int32_t* slot, const int32_t* start, const int32_t* cu, void* shift, void* out, int32_t dtype,
                                  void* stream) {
  MSA_REQUIRE(dtype_ok(dtype) && h && mu && tok_seq && slot && start && cu && shift && out, "token_shift: null pointer or bad dtype");
  MSA_REQUIRE(n_mix > 0 && n_tok >= 0 && width > 0, "token_shift: bad sizes");
  if (n_tok == 0) return MSA_OK;
  const int e = (int)dtype_size(dtype);
  const bool v4 = width % 4 == 0 && vec4_ok(h, e) && vec4_ok(mu, 4) && vec4_ok(shift, e) && vec4_ok(out, e);
  const int per = v4 ? width / 4 : width, threads = per >= 256 ? 256 : (per + 31) / 32 * 32;
  const dim3 grid((unsigned)n_tok, n_tok <= 256 ? (unsigned)((per + threads - 1) / threads) : 1u);   // few rows: spread the columns
  MSA_LM_DISPATCH(dtype, {
    if (v4) token_shift_kernel<T, 4><<<grid, threads, 0, (cudaStream_t)stream>>>((const T*)h, mu, n_mix, n_tok, width, tok_seq, slot, start, cu, (T*)shift, (T*)out);
    else token_shift_kernel<T, 1><<<grid, threads, 0, (cudaStream_t)stream>>>((const T*)h, mu, n_mix, n_tok, width, tok_seq, slot, start, cu, (T*)shift, (T*)out);
  });
  MSA_LAUNCH_OK("token_shift_kernel");
  return MSA_OK;
}

template <int V, typename T>
static void launch_silu_mul(const T* gu, int64_t gu_stride, int n_rows, int ff, T* out, int64_t out_stride, cudaStream_t stream) {
  for (int64_t r = 0; r < n_rows; r += 65535) {        // the second axis of a grid ends there
    const unsigned rows = (unsigned)(n_rows - r < 65535 ? n_rows - r : 65535);
    lm_silu_mul_kernel<T, V><<<dim3((unsigned)((ff + 256 * V - 1) / (256 * V)), rows), 256, 0, stream>>>(
        gu + r * gu_stride, gu_stride, ff, out + r * out_stride, out_stride);
  }
}

extern "C" int msa_lm_silu_mul(const void* gu, int64_t gu_stride, int32_t n_rows, int32_t ff, void* out, int64_t out_stride,
                               int32_t dtype, void* stream) {
  MSA_REQUIRE(dtype_ok(dtype) && gu && out && n_rows >= 0 && ff > 0, "lm_silu_mul: bad arguments");
  if (n_rows == 0) return MSA_OK;
  const int e = (int)dtype_size(dtype);
  const bool v4 = ff % 4 == 0 && gu_stride % 4 == 0 && out_stride % 4 == 0 && vec4_ok(gu, e) && vec4_ok(out, e);
  const bool v8 = dtype == MSA_BF16 && ff % 8 == 0 && gu_stride % 8 == 0 && out_stride % 8 == 0 && aligned16(gu) && aligned16(out);
  cudaStream_t st = (cudaStream_t)stream;
  int n_sm = 0;
  MSA_OK_OR_RETURN(device_sm_count(&n_sm));
  // Eight elements a thread where that still makes four blocks for every SM, else four: 32 x 3072 3.1 and 2.8 us, 512 x 3072 (768 blocks)
  // 5.1 both, 1055 x 6144 9.5 and 11.3.
  const bool many = (long long)n_rows * ((ff + 2047) / 2048) >= 4ll * n_sm;
  MSA_LM_DISPATCH(dtype, {
    const T* from = (const T*)gu;
    T* to = (T*)out;
    if constexpr (sizeof(T) == 2) {
      if (v8 && many) { launch_silu_mul<8>(from, gu_stride, n_rows, ff, to, out_stride, st); break; }
    }
    if (v4) launch_silu_mul<4>(from, gu_stride, n_rows, ff, to, out_stride, st);
    else launch_silu_mul<1>(from, gu_stride, n_rows, ff, to, out_stride, st);
  });
  MSA_LAUNCH_OK("lm_silu_mul_kernel");
  return MSA_OK;
}
