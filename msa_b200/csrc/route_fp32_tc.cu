// Routing of fp32 queries and keys on the 5th-generation tensor cores (tcgen05 + TMEM + TMA).
//
// Every 32-bit number is the exact sum of three bf16 numbers (8 bits each, rounded to nearest: x = h + m + l), so
//     q.k = qh.kh + (qh.km + qm.kh) + (qh.kl + qm.km + ql.kh)  + terms below 2^-25 of |q||k|,
// six bf16 products with fp32 accumulation.  The tensor core cuts off what it aligns away while it accumulates; the leading
// product is therefore summed over 64 channels at a time and the parts are added in registers, rounded to nearest; the five small
// ones go over all channels, two rows' planes side by side where the key's plane is the same (a product costs some 70 cycles,
// whatever its columns: four per 16 channels, not six).  Against 64 bits (16,000 chunks x 64 rows x 1024) that is no further off than chains of fp32
// multiply-adds.  Rows and chunks with a number for which the split is not exact or a part could overflow (not finite, 2^60 and more, below
// 2^-100 but not zero) get their scores from such chains (redo_odd); rows without a token are not looked at.
//
// 128 chunks (TMEM lanes) x up to 64 query rows per block, warps by role: 0-3 and 4-7 turn the keys' 32-channel boxes (TMA ring)
// into three planes of bf16 in TMEM, where the products read them as their A operand; 8-10 turn the query rows into planes in shared
// memory (B); 11 fetches boxes and issues the products; 12-15 add up the parts and publish.
//
// Bound by the conversions (6.5 instructions per element of 128 x 1024 keys and 64 x 1024 rows per block) and the latency of the chain
// box -> planes -> products, with one block per SM; the keys at HBM rate would take 10 us.  64 rows x 16,000 chunks x 1024: 29.6 us,
// 76.4 with fp32 multiply-adds on the CUDA cores (whose floor is 29); the error against 64 bits 1.0e-7 where that had 3.0e-7.
#include <cuda.h>

#include "common.cuh"
#include "route.cuh"
#include "tc_attn_common.cuh"

namespace msa {

constexpr int kRfChunks = 128, kRfRows = 64, kRfStages = 8, kRfBox = kRfChunks * 128;       // a box: 32 channels of 128 chunks
constexpr int kRfThreads = 16 * 32, kRfQThreads = 3 * 32, kRfSmem = kRfStages * kRfBox + 2 * 3 * kRfRows * 128 + 1024;
constexpr uint32_t kRfLead = 0, kRfSmall = 2 * kRfRows, kRfLast = 4 * kRfRows, kRfPlanes = 5 * kRfRows;      // TMEM columns
// redo_odd: channels at a time, floats of their row (16-byte reads without conflicts), of one buffer
constexpr int kRfSlab = 64, kRfPitch = kRfSlab + 4, kRfSlabFloats = (kRfChunks + kRfRows) * kRfPitch;
static_assert((2 * kRfSlabFloats + kRfRows * kRfChunks) * 4 <= kRfSmem - 1024, "redo_odd's memory");
constexpr float kRfTop = 0x1p60f, kRfLow = 0x1p-100f;

struct RouteFp32Params {
  const float* qf; const float* row_bias;
  const float* rk; long long rk_stride;
  const int32_t* chunk_doc;
  int n_rows, s_pad, bn, n_chunks, kdim, n_docs;
  int first_row;                                            // of this launch: a grid has 65535 tiles of rows at most
  float alpha;
  uint32_t* keys; long long table_stride;
  int32_t* status;
};

// Two numbers to three packed pairs.
__device__ __forceinline__ void split3(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack2_bf16(x, y);
  x -= __uint_as_float(h << 16);
  y -= __uint_as_float(h & 0xffff0000u);
  m = pack2_bf16(x, y);
  x -= __uint_as_float(m << 16);
  y -= __uint_as_float(m & 0xffff0000u);
  l = pack2_bf16(x, y);
}
// Denormal operands count (the file is compiled with them flushed), in fma_f32x2 too.
__device__ __forceinline__ void add_exact(float& c, float a) { asm("add.rn.f32 %0, %0, %1;" : "+f"(c) : "f"(a)); }
// Whether some of the numbers is outside what split3 takes.
template <int N>
__device__ __forceinline__ bool outside(const float (&x)[N]) {
  float top = fabsf(x[0]), low = top;
#pragma unroll
  for (int i = 1; i < N; ++i) {
    asm("max.NaN.f32 %0, %0, %1;" : "+f"(top) : "f"(fabsf(x[i])));
    low = fminf(low, fabsf(x[i]));
  }
  bool bad = !(top < kRfTop);
  if (low < kRfLow) {                                       // zeros, mostly
#pragma unroll
    for (int i = 0; i < N; ++i) bad |= fabsf(x[i]) < kRfLow && (__float_as_uint(x[i]) & 0x7fffffffu) != 0;
  }
  return bad;
}

// Four rows and the 32s of chunks I0 .. I1 - 1 of redo_odd; sums over the even and the odd channels.
template <int I0, int I1>
__device__ __forceinline__ void redo_add(unsigned long long (&sum)[4][4], const float* key, const float* row) {
#pragma unroll 2
  for (int k = 0; k < kRfSlab; k += 4) {
    ulonglong2 q[4], c[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) q[j] = *reinterpret_cast<const ulonglong2*>(row + j * kRfPitch + k);
#pragma unroll
    for (int i = I0; i < I1; ++i) c[i] = *reinterpret_cast<const ulonglong2*>(key + i * 32 * kRfPitch + k);
#pragma unroll
    for (int i = I0; i < I1; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[i][j] = fma_f32x2(c[i].x, q[j].x, sum[i][j]);
#pragma unroll
    for (int i = I0; i < I1; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[i][j] = fma_f32x2(c[i].y, q[j].y, sum[i][j]);
  }
}
// Scores of the rows and chunks with a number that split3 does not take, as two chains of fp32 multiply-adds in the order of the channels: 64
// channels of the block's 128 chunks and 64 rows at a time through shared memory, the next ones on their way, four rows per warp, four
// chunks per lane.  A warp works on 32 chunks only where one of its rows or one of those chunks is such; the others' scores stay as the
// products gave them.  Bound by the latency of its steps: 64 rows x 16,000 chunks x 1024 from a cold L2, table reset included, take 43 us, 84
// with one such row, 105 with one such chunk, 135 with nothing but such rows (84 with multiply-adds throughout, and 2120 for any of them
// when a thread per chunk read its key from memory row after row).
__device__ __forceinline__ void redo_odd(const RouteFp32Params& p, int c0, int r0, float* tiles, float* scores, unsigned long long odd_rows,
                                         const uint32_t* odd_chunks) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, n_steps = (p.kdim + kRfSlab - 1) / kRfSlab;
  const uint32_t mine = (uint32_t)(odd_rows >> (4 * warp)) & 15u;
  uint32_t groups = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) groups |= mine || odd_chunks[i] ? 1u << i : 0u;
  unsigned long long sum[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) sum[i][j] = 0ull;
  auto fetch = [&](int step) {
    constexpr int kVecs = kRfSlab / 4;
    const uint32_t dst = smem_u32(tiles + step % 2 * kRfSlabFloats);
    for (int item = threadIdx.x; item < (kRfChunks + kRfRows) * kVecs; item += kRfThreads) {
      const int r = item / kVecs, v = item % kVecs, k = step * kRfSlab + v * 4, row = r0 + r - kRfChunks;
      const bool on = k < p.kdim && (r < kRfChunks ? c0 + r < p.n_chunks : r - kRfChunks < p.bn && row < p.n_rows);
      const float* src = r < kRfChunks ? p.rk + (long long)(c0 + r) * p.rk_stride + k : p.qf + (long long)row * p.kdim + k;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (r * kRfPitch + v * 4) * 4), "l"(on ? src : p.qf), "r"(on ? 16u : 0u)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0);
  for (int step = 0; step < n_steps; ++step) {
    if (step + 1 < n_steps) {
      fetch(step + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const float* key = tiles + step % 2 * kRfSlabFloats + lane * kRfPitch;
    const float* row = tiles + step % 2 * kRfSlabFloats + (kRfChunks + 4 * warp) * kRfPitch;
    if (groups == 15u) {
      redo_add<0, 4>(sum, key, row);
    } else {
      if (groups & 1u) redo_add<0, 1>(sum, key, row);
      if (groups & 2u) redo_add<1, 2>(sum, key, row);
      if (groups & 4u) redo_add<2, 3>(sum, key, row);
      if (groups & 8u) redo_add<3, 4>(sum, key, row);
    }
    __syncthreads();                                        // read before the step after the next lands there
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if ((mine >> j & 1u) || (odd_chunks[i] >> lane & 1u)) {
        float even, odd;
        f32x2_split(sum[i][j], even, odd);
        add_exact(even, odd);
        scores[(4 * warp + j) * kRfChunks + 32 * i + lane] = even;
      }
  __syncthreads();
}

__global__ void __launch_bounds__(kRfThreads, 1)
route_fp32_kernel(const __grid_constant__ CUtensorMap tmap_k, const RouteFp32Params p) {
  extern __shared__ unsigned char smem_dyn[];
  __shared__ uint64_t s_full[kRfStages], s_t_full[2], s_t_empty[2], s_b_full[2], s_b_empty[2], s_d_full[2], s_d_empty[2], s_drain;
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;
  __shared__ unsigned long long s_odd_rows;                 // query rows and chunks with a number that split3 does not take
  __shared__ uint32_t s_odd_chunks[kRfChunks / 32];
  __shared__ float s_bias[kRfRows];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int c0 = blockIdx.x * kRfChunks, r0 = p.first_row + blockIdx.y * p.bn;
  unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  unsigned char* planes = ring + kRfStages * kRfBox;
  const int b_bytes = 3 * p.bn * 128;
  volatile int* abort_flag = &s_abort;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kRfStages; ++i) mbar_init(&s_full[i], 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_t_full[i], 4); mbar_init(&s_t_empty[i], 1);
      mbar_init(&s_b_full[i], kRfQThreads / 32); mbar_init(&s_b_empty[i], 1);
      mbar_init(&s_d_full[i], 1); mbar_init(&s_d_empty[i], 4);
    }
    mbar_init(&s_drain, 1);
    s_abort = 0;
    s_odd_rows = 0ull;
    for (int i = 0; i < kRfChunks / 32; ++i) s_odd_chunks[i] = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 11) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  bool mine = false;
  if (threadIdx.x < kRfRows) {
    const float bias = (int)threadIdx.x < p.bn && r0 + (int)threadIdx.x < p.n_rows ? p.row_bias[r0 + threadIdx.x] : -INFINITY;
    s_bias[threadIdx.x] = bias;
    mine = bias != -INFINITY;
  }
  tc_fence_before();
  const bool live = __syncthreads_or(mine);                 // rows without a token have no scores
  tc_fence_after();
  const uint32_t tmem = s_tmem_base;
  const int n_kb = live ? (p.kdim + 63) / 64 : 0, n_box = 2 * n_kb;
  float acc[kRfRows];

  if (warp < 8) {
    // ---- keys: box after box, the two groups in turn; thread = chunk
    const int group = warp / 4, row = threadIdx.x % kRfChunks;
    const uint32_t dst = tmem + ((uint32_t)(warp % 4 * 32) << 16) + kRfPlanes + group * 48;
    bool bad = false;
    for (int box = group, n = 0; box < n_box; box += 2, ++n) {
      const int st = box % kRfStages;
      bool ok = mbar_wait(&s_full[st], (box / kRfStages) & 1u, abort_flag, p.status, 21);
      if (!__all_sync(0xffffffffu, ok)) break;
      const unsigned char* src = ring + st * kRfBox + row * 128;
      float x[32];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 v = *reinterpret_cast<const float4*>(src + ((j ^ (row & 7)) * 16));
        x[4 * j] = v.x; x[4 * j + 1] = v.y; x[4 * j + 2] = v.z; x[4 * j + 3] = v.w;
      }
      bad |= outside(x);
      uint32_t h[16], m[16], l[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) split3(x[2 * i], x[2 * i + 1], h[i], m[i], l[i]);
      ok = mbar_wait(&s_t_empty[group], (n & 1u) ^ 1u, abort_flag, p.status, 22);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      tmem_st16(dst, h);
      tmem_st16(dst + 16, m);
      tmem_st16(dst + 32, l);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_t_full[group]);
    }
    if (bad) atomicOr(&s_odd_chunks[row / 32], 1u << (row % 32));
  } else if (warp < 11) {
    // ---- query rows: 64 channels at a time, eight per item
    const int t = threadIdx.x - 256, n_items = p.bn * 8;
    constexpr int kItems = (kRfRows * 8 + kRfQThreads - 1) / kRfQThreads;
    float x[kItems][8];
    uint32_t bad = 0u;                                      // by item: its row is the same throughout
    auto load = [&](int kb) {
#pragma unroll
      for (int i = 0; i < kItems; ++i) {
        const int item = t + i * kRfQThreads, r = item / 8, k = kb * 64 + item % 8 * 8;
        const float* src = p.qf + (long long)(r0 + r) * p.kdim + k;
        const bool on = item < n_items && r0 + r < p.n_rows;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 a = on && k < p.kdim ? *reinterpret_cast<const float4*>(src) : zero;
        const float4 b = on && k + 4 < p.kdim ? *reinterpret_cast<const float4*>(src + 4) : zero;
        x[i][0] = a.x; x[i][1] = a.y; x[i][2] = a.z; x[i][3] = a.w;
        x[i][4] = b.x; x[i][5] = b.y; x[i][6] = b.z; x[i][7] = b.w;
      }
    };
    if (n_kb > 0) load(0);
    for (int kb = 0; kb < n_kb; ++kb) {
      const bool ok = mbar_wait(&s_b_empty[kb & 1], ((kb >> 1) & 1u) ^ 1u, abort_flag, p.status, 23);
      if (!__all_sync(0xffffffffu, ok)) break;
      unsigned char* dst = planes + (kb & 1) * b_bytes;
#pragma unroll
      for (int i = 0; i < kItems; ++i) {
        const int item = t + i * kRfQThreads, r = item / 8, c = item % 8;
        if (item >= n_items) break;
        bad |= (uint32_t)outside(x[i]) << i;
        uint4 h, m, l;
        split3(x[i][0], x[i][1], h.x, m.x, l.x);
        split3(x[i][2], x[i][3], h.y, m.y, l.y);
        split3(x[i][4], x[i][5], h.z, m.z, l.z);
        split3(x[i][6], x[i][7], h.w, m.w, l.w);
        unsigned char* d = dst + r * 128 + ((c ^ (r & 7)) * 16);
        *reinterpret_cast<uint4*>(d) = h;
        *reinterpret_cast<uint4*>(d + p.bn * 128) = m;
        *reinterpret_cast<uint4*>(d + 2 * p.bn * 128) = l;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_b_full[kb & 1]);
      if (kb + 1 < n_kb) load(kb + 1);
    }
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      const int r = (t + i * kRfQThreads) / 8;
      if ((bad >> i & 1u) && s_bias[r] != -INFINITY) atomicOr(&s_odd_rows, 1ull << r);       // what stands in a row without a token is not asked for
    }
  } else if (warp == 11) {
    if (lane == 0) {
      auto fetch = [&](int box) {
        mbar_expect_tx(&s_full[box % kRfStages], kRfBox);
        tma_load_2d(ring + box % kRfStages * kRfBox, &tmap_k, box * 32, c0, &s_full[box % kRfStages]);
      };
      for (int box = 0; box < min(n_box, kRfStages); ++box) fetch(box);
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.bn >> 3) << 17) | ((uint32_t)(kRfChunks >> 4) << 24);
      const uint32_t idesc2 = idesc + ((uint32_t)(p.bn >> 3) << 17);          // two planes of the rows at once
      bool ok = true;
      for (int kb = 0; kb < n_kb && ok; ++kb) {
        const int b = kb & 1;
        const uint32_t ph = (kb >> 1) & 1u, lead = tmem + kRfLead + b * kRfRows, small = tmem + kRfSmall, last = tmem + kRfLast;
        if (!(ok = mbar_wait(&s_b_full[b], ph, abort_flag, p.status, 26))) break;
        if (!(ok = mbar_wait(&s_d_empty[b], ph ^ 1u, abort_flag, p.status, 27))) break;
        const uint64_t q = make_smem_desc(smem_u32(planes) + b * b_bytes);
        const uint64_t plane = (uint64_t)(p.bn * 128 / 16);
        for (int half = 0; half < 2; ++half) {
          if (!(ok = mbar_wait(&s_t_full[half], kb & 1u, abort_flag, p.status, 28))) break;
          if (2 * kb + half + kRfStages < n_box) fetch(2 * kb + half + kRfStages);      // the box in this place has been read
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const uint32_t a = tmem + kRfPlanes + half * 48 + k * 8;
            const uint64_t qh = q + (uint64_t)(2 * (2 * half + k)), qm = qh + plane;
            tc_mma_bf16_ts(lead, a, qh, idesc, (half | k) ? 1u : 0u);
            tc_mma_bf16_ts(small, a, qm, idesc2, (kb | half | k) ? 1u : 0u);          // kh qm | kh ql
            tc_mma_bf16_ts(small, a + 16, qh, idesc2, 1u);                            // km qh | km qm
            tc_mma_bf16_ts(last, a + 32, qh, idesc, (kb | half | k) ? 1u : 0u);       // kl qh
          }
          tc_commit(&s_t_empty[half]);
        }
        if (!ok) break;
        tc_commit(&s_b_empty[b]);
        tc_commit(&s_d_full[b]);
      }
      tc_commit(&s_drain);
      unsigned long long w0 = global_ns();
      while (!mbar_try_wait(&s_drain, 0) && global_ns() - w0 < kWaitLimitNs) {}
      if (!ok) {                                             // copies in flight land before the block's memory goes
        w0 = global_ns();
        while (global_ns() - w0 < 1000000ull) {}
      }
    }
  } else {
    // ---- sums of the leading product's parts; thread = chunk
    const uint32_t src = tmem + ((uint32_t)(warp % 4 * 32) << 16);
#pragma unroll
    for (int j = 0; j < kRfRows; ++j) acc[j] = 0.f;
    auto add = [&](uint32_t col) {
#pragma unroll
      for (int j = 0; j < kRfRows; j += 16) {
        if (j < p.bn) {
          uint32_t v[16];
          tmem_ld16(src + col + j, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) acc[j + i] += __uint_as_float(v[i]);
        }
      }
    };
    bool ok = true;
    for (int kb = 0; kb < n_kb && ok; ++kb) {
      ok = mbar_wait(&s_d_full[kb & 1], (kb >> 1) & 1u, abort_flag, p.status, 24);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      add(kRfLead + (kb & 1) * kRfRows);
      if (kb + 1 == n_kb) { add(kRfSmall); add(kRfSmall + p.bn); add(kRfLast); }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_d_empty[kb & 1]);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 11) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  if (s_abort) return;
  const bool some = s_odd_rows || s_odd_chunks[0] || s_odd_chunks[1] || s_odd_chunks[2] || s_odd_chunks[3];
  float* scores = reinterpret_cast<float*>(ring) + 2 * kRfSlabFloats;                  // [row][chunk]
  if (some) {
    if (warp >= 12) {
#pragma unroll
      for (int j = 0; j < kRfRows; ++j) scores[j * kRfChunks + threadIdx.x - 384] = acc[j];
    }
    redo_odd(p, c0, r0, reinterpret_cast<float*>(ring), scores, s_odd_rows, s_odd_chunks);
  }
  if (warp < 12) return;
  const int in_block = (warp - 12) * 32 + lane, chunk = c0 + in_block;
  if (chunk >= p.n_chunks) return;
  if (some) {
#pragma unroll
    for (int j = 0; j < kRfRows; ++j) acc[j] = scores[j * kRfChunks + in_block];
  }
  const int doc = p.chunk_doc[chunk];
  const bool known = doc >= 1 && doc <= p.n_docs;
  float best = -INFINITY;
#pragma unroll
  for (int j = 0; j < kRfRows; j += 16) {                    // a block of 16 rows is one sequence's
    if (j >= p.bn || r0 + j >= p.n_rows) break;
#pragma unroll
    for (int i = 0; i < 16; ++i) best = fmaxf(best, acc[j + i] + s_bias[j + i]);
    const int seq = (r0 + j) / p.s_pad;
    if (j + 16 < p.bn && r0 + j + 16 < p.n_rows && (r0 + j + 16) / p.s_pad == seq) continue;
    if (known) atomicMax(p.keys + seq * p.table_stride + doc, float_to_key(best * p.alpha));
    else atomicAdd(p.status + 2, 1);                         // an id outside the table: counted, never used as a column
    best = -INFINITY;
  }
}

int launch_route_fp32(const float* qf, const float* row_bias, int n_rows, int s_pad, const float* rk, int64_t rk_stride, int n_chunks, int kdim,
                      const int32_t* chunk_doc, int n_docs, float alpha, uint32_t* keys, int64_t table_stride, int32_t* status, cudaStream_t stream) {
  EncodeTiledFn enc = get_encode_fn();
  MSA_REQUIRE(enc, "cuTensorMapEncodeTiled is not available from the driver");
  CUtensorMap map;
  cuuint64_t dims[2] = {(cuuint64_t)kdim, (cuuint64_t)n_chunks}, strides[1] = {(cuuint64_t)rk_stride * 4};
  cuuint32_t box[2] = {32, kRfChunks}, estr[2] = {1, 1};
  const CUresult r = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(rk), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  MSA_REQUIRE(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed with code %d", (int)r);
  const int blocks = n_rows / 16, tiles = (blocks + kRfRows / 16 - 1) / (kRfRows / 16), bn = (blocks + tiles - 1) / tiles * 16;
  static DeviceSmem state{};
  MSA_OK_OR_RETURN(ensure_dynamic_smem(route_fp32_kernel, kRfSmem, state));
  RouteFp32Params p{qf, row_bias, rk, rk_stride, chunk_doc, n_rows, s_pad, bn, n_chunks, kdim, n_docs, 0, alpha, keys, table_stride, status};
  for (long long first = 0; first < n_rows; first += 65535ll * bn) {
    p.first_row = (int)first;
    const long long left = (n_rows - first + bn - 1) / bn;
    route_fp32_kernel<<<dim3((n_chunks + kRfChunks - 1) / kRfChunks, (unsigned)(left < 65535 ? left : 65535)), kRfThreads, kRfSmem, stream>>>(map, p);
    MSA_LAUNCH_OK("route_fp32_kernel");
  }
  return MSA_OK;
}

}  // namespace msa
