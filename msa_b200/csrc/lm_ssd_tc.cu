// The state-space recurrence over prompt portions (lm_linear_chunk.cu) on the 5th-generation tensor cores: one block walks the chunks
// of 64 tokens of a portion with the states of two heads of a group in TMEM, so that no chunk state passes through memory.
//
// Transposed, a thread's TMEM lane is a value column; two heads of 64 make the 128 lanes.  With the chunk's keys B and queries C (one
// set per group), its values X, steps dt and running log2 decays G (per head):
//     scores = C B^T                          P_h = scores * 2^(G_t - G_i) dt_i below the diagonal, hi / lo planes in shared memory
//     R^T = S^T C^T                           O_h^T = 2^G R^T + X^T P_h^T  (for both heads' lanes; each reads its own)
//     dS^T = (w X)^T B, w_i = dt_i 2^(G_C - G_i)     S' = fma(2^(G_C), S, dS)
//     y = (O + skip x) silu(gate)
// 32-bit operands (state, scores with their decays, weighted values) enter as hi / lo pairs of bf16; sums are fp32.  Every sum runs as in the
// kernels over all chunks at once (running decays in 64 bits, the same products in the same order) and the bits are theirs, so that a
// sequence does not depend on what else is in a step.  In particular no sum on the tensor core, which cuts off what it aligns away, goes
// on over chunks: the state is rounded to nearest once a chunk.
//
// The scores come twice, in the lower and the upper 64 lanes (C lies in shared memory twice), so that 128 threads make the two heads' P.
//
// Warps by role: 0-7 scores -> P, 8-11 states and the values (weighted as TMEM planes, transposed in shared memory), 12-19 outputs,
// 20-22 fetch (two chunks' buffers) and sum up the decays, 23 issues the products.
// What bounds it: instructions of the conversions (their latencies, with five or six warps per scheduler), 56 products of some 70 cycles
// each, whatever their columns, and the chains scores -> P -> outputs and state -> read-out -> outputs.  Portions of 2048, 1500, 1911 and 777
// tokens, 64 heads, from a cold L2: 187 us, where the three kernels over all chunks at once take 425 (chunk states through HBM four
// times, products on mma.sync).  With the state as the tensor core's accumulator and its read-out added to the outputs at the end it took 172.
#include "lm_linear.cuh"
#include "mma_helpers.cuh"
#include "tc_attn_common.cuh"

namespace msa {

constexpr int kStRows = 64, kStN = 128, kStV = 64, kStThreads = 768;
constexpr int kStPlane = kStRows * 128;                                            // 64 rows of 128 bytes
constexpr int kStC = 0, kStB = 4 * kStPlane, kStX = kStB + 2 * kStPlane, kStBuf = kStX + 2 * kStPlane;   // C twice per 64 columns
// per head hi, lo; values transposed (two chunks').  The gates come where the values were, once those are transposed.
constexpr int kStP = 2 * kStBuf, kStXt = kStP + 4 * kStPlane;
constexpr size_t kStSmem = kStXt + 4 * kStPlane + 1024;
// TMEM columns: states; what the chunk adds to them, 16 columns at a time replaced by the new state's planes (8 hi, 8 lo); scores; planes of the
// weighted values; outputs of head 0 and of head 1
constexpr uint32_t kStS = 0, kStD = 128, kStZ = 256, kStWh = 320, kStWl = 352, kStO1 = 384, kStO2 = 448;

struct SsdTcParams {
  msa_lm_ssd_args a;
  const __nv_bfloat16* xbc;      // [rows, inner | groups * n_state | groups * n_state]
  const float* dt;               // [rows, heads]
  int32_t* status;
};
struct SsdTcBars { uint64_t full[2], free[2], g_full[2], z_done, p_ready, s_ready, x_ready, s_done, r_done, r_ready, h_done, o_done, o_free, drain; };
struct __align__(16) SsdTcDecay {              // of a chunk, per head; g is read two at a time
  double g[2][kStRows];
  float eg[2][kStRows], dt[2][kStRows], w[2][kStRows], all[2];
};
static_assert(sizeof(SsdTcDecay) % 16 == 0, "the second chunk's pairs of doubles");

__device__ __forceinline__ void st_split2(float x, float y, uint32_t& hi, uint32_t& lo) {
  hi = pack2_bf16(x, y);
  lo = pack2_bf16(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xffff0000u));
}

__global__ void __launch_bounds__(kStThreads, 1) ssd_tc_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                const __grid_constant__ CUtensorMap map_g, const SsdTcParams p) {
  extern __shared__ unsigned char dyn[];
  __shared__ SsdTcBars bars;
  __shared__ SsdTcDecay s_d[2];
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;
  const msa_lm_ssd_args& a = p.a;
  unsigned char* sm = reinterpret_cast<unsigned char*>(((uintptr_t)dyn + 1023) & ~(uintptr_t)1023);
  volatile int* abort_flag = &s_abort;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int h0 = blockIdx.x * 2, ps = blockIdx.y, sq = ps + a.n_decode, gr = h0 / (a.heads / a.groups);
  const int inner = a.heads * kStV, bc = a.groups * kStN, chan = inner + 2 * bc;
  const int len = a.cu[sq + 1] - a.cu[sq], n_chunks = (len + kStRows - 1) / kStRows;
  const long long n0 = a.cu[sq], row0 = n0 - a.n_decode;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&bars.full[i], 3); mbar_init(&bars.free[i], 9); mbar_init(&bars.g_full[i], 1); }
    mbar_init(&bars.z_done, 1); mbar_init(&bars.s_done, 1); mbar_init(&bars.o_done, 1); mbar_init(&bars.drain, 1);
    mbar_init(&bars.r_done, 1); mbar_init(&bars.h_done, 1); mbar_init(&bars.r_ready, 8); mbar_init(&bars.p_ready, 8); mbar_init(&bars.s_ready, 4); mbar_init(&bars.x_ready, 4); mbar_init(&bars.o_free, 8);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 23) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem_base, lanes = tmem + ((uint32_t)(warp % 4 * 32) << 16);
  const int col = threadIdx.x % 128, hd = col / kStV;                 // lane: of head hd (for the scores: row col % 64 for head hd)
  auto wait = [&](uint64_t* bar, uint32_t parity, int code) {         // a whole warp; false: some wait of the block ran out
    const bool ok = mbar_wait(bar, parity & 1u, abort_flag, p.status, code);
    return (bool)__all_sync(0xffffffffu, ok);
  };
  auto arrive = [&](uint64_t* bar) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
  };
  auto at = [](int r, int c) { return r * 128 + ((c ^ (r & 7)) << 4); };   // 16 bytes of a tile with 128-byte rows

  if (warp < 8) {
    // ---- scores -> P: the first four warps columns 0 .. 31, the others the rest, which rows below 32 have no use for
    const int t = col % kStRows, part = warp / 4;
    const bool on = part == 0 || t >= 32;                // of the whole warp
    for (int ch = 0; ch < n_chunks; ++ch) {
      const SsdTcDecay& d = s_d[ch & 1];
      if (!wait(&bars.full[ch & 1], ch >> 1, 50) || !wait(&bars.z_done, ch, 51)) break;      // the products before have left P, too
      tc_fence_after();
      const double gt = d.g[hd][t];
      unsigned char* row = sm + kStP + hd * 2 * kStPlane;
      if (on) {
#pragma unroll
        for (int k0 = 0; k0 < 32; k0 += 16) {
          const int c0 = part * 32 + k0;
          uint32_t z[16], hi[8], lo[8];
          tmem_ld16(lanes + kStZ + c0, z);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const double2 g = *reinterpret_cast<const double2*>(&d.g[hd][c0 + i]);
            const float2 dt = *reinterpret_cast<const float2*>(&d.dt[hd][c0 + i]);
            const float x = __uint_as_float(z[i]) * exp2f((float)(gt - g.x)) * dt.x;
            const float y = __uint_as_float(z[i + 1]) * exp2f((float)(gt - g.y)) * dt.y;
            // masked as bits: a branch around every element would expose its whole latency
            st_split2(__uint_as_float(__float_as_uint(x) & (c0 + i <= t ? 0xffffffffu : 0u)),
                      __uint_as_float(__float_as_uint(y) & (c0 + i + 1 <= t ? 0xffffffffu : 0u)), hi[i / 2], lo[i / 2]);
          }
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            unsigned char* dst = row + at(t, c0 / 8 + k);
            *reinterpret_cast<uint4*>(dst) = make_uint4(hi[4 * k], hi[4 * k + 1], hi[4 * k + 2], hi[4 * k + 3]);
            *reinterpret_cast<uint4*>(dst + kStPlane) = make_uint4(lo[4 * k], lo[4 * k + 1], lo[4 * k + 2], lo[4 * k + 3]);
          }
        }
      }
      tc_fence_before();
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      arrive(&bars.p_ready);
    }
  } else if (warp < 12) {
    // ---- states, and the chunk's values: weighted and transposed
    float* state = a.state + ((long long)a.slot[sq] * a.heads + h0 + hd) * kStN * kStV + col % kStV;
    const bool fresh = a.start[sq] == 0;
    auto put_state = [&](int n, const uint32_t (&x)[16]) {              // 16 of the state's rows and their planes
      uint32_t planes[16];
#pragma unroll
      for (int i = 0; i < 8; ++i) st_split2(__uint_as_float(x[2 * i]), __uint_as_float(x[2 * i + 1]), planes[i], planes[8 + i]);
      tmem_st16(lanes + kStS + n, x);
      tmem_st16(lanes + kStD + n, planes);
    };
    float all = 1.f;
    auto next_state = [&](int n, uint32_t (&x)[16]) {                   // the state behind a chunk: decayed, and what the chunk adds
      uint32_t add[16];
      tmem_ld16(lanes + kStS + n, x);
      tmem_ld16(lanes + kStD + n, add);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i] = __float_as_uint(fmaf(all, __uint_as_float(x[i]), __uint_as_float(add[i])));
    };
    if (n_chunks == 0 && fresh)
      for (int n = 0; n < kStN; ++n) state[n * kStV] = 0.f;
    bool ok = true;
    for (int ch = 0; ch < n_chunks && ok; ++ch) {
      const int b = ch & 1;
      if (!(ok = wait(&bars.full[b], ch >> 1, 52))) break;
      if (ch > 0 && !(ok = wait(&bars.s_done, ch + 1, 53))) break;
      tc_fence_after();
      for (int n = 0; n < kStN; n += 16) {
        uint32_t x[16];
        if (ch == 0) {
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] = fresh ? 0u : __float_as_uint(state[(n + i) * kStV]);
        } else {
          next_state(n, x);
        }
        put_state(n, x);
      }
      all = s_d[b].all[hd];
      tmem_st_wait();
      tc_fence_before();
      arrive(&bars.s_ready);
      const unsigned char* val = sm + b * kStBuf + kStX + hd * kStPlane + col % 8 * 2;
      unsigned char* row = sm + kStXt + b * 2 * kStPlane;
#pragma unroll
      for (int t = 0; t < kStRows; t += 32) {
        uint32_t x[16], hi[16], lo[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const uint32_t x0 = *reinterpret_cast<const uint16_t*>(val + at(t + 2 * i, col % kStV / 8));
          const uint32_t x1 = *reinterpret_cast<const uint16_t*>(val + at(t + 2 * i + 1, col % kStV / 8));
          const float2 w = *reinterpret_cast<const float2*>(&s_d[b].w[hd][t + 2 * i]);
          x[i] = x0 | x1 << 16;
          st_split2(w.x * __uint_as_float(x0 << 16), w.y * __uint_as_float(x1 << 16), hi[i], lo[i]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
          *reinterpret_cast<uint4*>(row + at(col, t / 8 + k)) = make_uint4(x[4 * k], x[4 * k + 1], x[4 * k + 2], x[4 * k + 3]);
        tmem_st16(lanes + kStWh + t / 2, hi);
        tmem_st16(lanes + kStWl + t / 2, lo);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tmem_st_wait();
      tc_fence_before();
      arrive(&bars.x_ready);
      if (warp > 8) continue;
      if (!(ok = wait(&bars.x_ready, ch, 64))) break;      // the four warps have read the values: the gates take their place
      if (lane == 0) {
        mbar_expect_tx(&bars.g_full[b], 2 * kStPlane);
#pragma unroll
        for (int blk = 0; blk < 2; ++blk)
          tma_load_2d(sm + b * kStBuf + kStX + blk * kStPlane, &map_g, h0 * kStV + blk * 64, (int)n0 + ch * kStRows, &bars.g_full[b]);
      }
    }
    if (ok && n_chunks > 0 && wait(&bars.s_done, n_chunks + 1, 54)) {
      tc_fence_after();
      for (int n = 0; n < kStN; n += 16) {
        uint32_t x[16];
        next_state(n, x);
#pragma unroll
        for (int i = 0; i < 16; ++i) state[(n + i) * kStV] = __uint_as_float(x[i]);
      }
    }
  } else if (warp < 20) {
    // ---- outputs: half of the tokens to four warps each.  The read-out of the state is decayed where it stands; the chunk's own tokens add to it.
    const int part = (warp - 12) / 4 * (kStRows / 2);
    const float skip = a.d_skip[h0 + hd];
    float* out = a.y + n0 * inner + h0 * kStV + col;
    const uint32_t own = lanes + (hd ? kStO2 : kStO1) + part;
    for (int ch = 0; ch < n_chunks; ++ch) {
      const int b = ch & 1, rows = min(kStRows, len - ch * kStRows);
      float o[kStRows / 2];
      if (!wait(&bars.full[b], ch >> 1, 62) || !wait(&bars.r_done, ch, 65)) break;
      tc_fence_after();
#pragma unroll
      for (int t = 0; t < kStRows / 2; t += 16) {
        uint32_t x[16];
        tmem_ld16(lanes + kStO1 + part + t, x);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = __float_as_uint(s_d[b].eg[hd][part + t + i] * __uint_as_float(x[i]));
        tmem_st16(own + t, x);
      }
      tmem_st_wait();
      tc_fence_before();
      arrive(&bars.r_ready);
      if (!wait(&bars.o_done, ch, 55)) break;
      tc_fence_after();
#pragma unroll
      for (int t = 0; t < kStRows / 2; t += 16) {
        uint32_t x[16];
        tmem_ld16(own + t, x);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) o[t + i] = __uint_as_float(x[i]);
      }
      tc_fence_before();
      arrive(&bars.o_free);
      if (!wait(&bars.g_full[b], ch >> 1, 63)) break;      // a barrier per buffer: the next chunk's gates may come before these are asked for
      const unsigned char *row = sm + kStXt + b * 2 * kStPlane, *gate = sm + b * kStBuf + kStX + hd * kStPlane + col % 8 * 2;
      float* dst = out + (long long)(ch * kStRows + part) * inner;
#pragma unroll
      for (int t = 0; t < kStRows / 2; t += 8) {
        if (part + t >= rows) break;
        const uint4 xv = *reinterpret_cast<const uint4*>(row + at(col, (part + t) / 8));
        const uint32_t x[4] = {xv.x, xv.y, xv.z, xv.w};
        float y[8];                                       // all eight before the first condition: their latencies overlap
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float z = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(gate + at(part + t + i, col % kStV / 8)));
          const float xx = __uint_as_float(i & 1 ? x[i / 2] & 0xffff0000u : x[i / 2] << 16);
          y[i] = fmaf(skip, xx, o[t + i]) * silu_act<__nv_bfloat16>(z);
        }
        if (part + t + 8 <= rows) {
#pragma unroll
          for (int i = 0; i < 8; ++i) dst[(long long)(t + i) * inner] = y[i];
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (part + t + i < rows) dst[(long long)(t + i) * inner] = y[i];
        }
      }
      arrive(&bars.free[b]);
    }
  } else if (warp < 23) {
    // ---- operands: whole chunks by TMA, the last rows of a portion by cp.async (what follows them is zero); decays
    const int k = warp - 20, t = threadIdx.x - 640;
    const double rate = -1.4426950408889634 * expf(a.a_log[h0 + min(k, 1)]);
    const int x_b = inner + gr * kStN, x_c = x_b + bc;
    for (int ch = 0; ch < n_chunks; ++ch) {
      const int b = ch & 1, rows = min(kStRows, len - ch * kStRows);
      if (!wait(&bars.free[b], (ch >> 1) ^ 1, 56)) break;
      unsigned char* buf = sm + b * kStBuf;
      if (rows == kStRows) {
        if (k == 2 && lane == 0) {
          const int y = (int)(row0 + ch * kStRows);
          mbar_expect_tx(&bars.full[b], 8 * kStPlane);
#pragma unroll
          for (int blk = 0; blk < 2; ++blk) {
            tma_load_2d(buf + kStB + blk * kStPlane, &map_x, x_b + blk * 64, y, &bars.full[b]);
            tma_load_2d(buf + kStC + blk * 2 * kStPlane, &map_x, x_c + blk * 64, y, &bars.full[b]);
            tma_load_2d(buf + kStC + (blk * 2 + 1) * kStPlane, &map_x, x_c + blk * 64, y, &bars.full[b]);
            tma_load_2d(buf + kStX + blk * kStPlane, &map_x, h0 * kStV + blk * 64, y, &bars.full[b]);
          }
        }
      } else {
        const uint32_t base = smem_u32(buf);
        const __nv_bfloat16* src = p.xbc + (row0 + ch * kStRows) * chan;
        for (int i = t; i < kStRows * 16; i += 96) {                      // 16 pieces a row: blocks of 64 columns
          const int r = i / 16, c = i % 16, blk = c / 8;
          const bool on = r < rows;
          const long long off = (on ? (long long)r * chan : 0) + c * 8;
          const uint32_t n = on ? 16u : 0u;
          cp_async16(base + kStC + blk * 2 * kStPlane + at(r, c % 8), src + x_c + off, n);
          cp_async16(base + kStC + blk * 2 * kStPlane + kStPlane + at(r, c % 8), src + x_c + off, n);
          cp_async16(base + kStB + blk * kStPlane + at(r, c % 8), src + x_b + off, n);
          cp_async16(base + kStX + blk * kStPlane + at(r, c % 8), src + h0 * kStV + off, n);
        }
        cp_async_commit();
      }
      if (k < 2) {                                                        // a warp per head, two rows a lane
        const int r = 2 * lane;
        const float* dt = p.dt + (row0 + ch * kStRows) * a.heads + h0 + k;
        const float d0 = r < rows ? dt[(long long)r * a.heads] : 0.f, d1 = r + 1 < rows ? dt[(long long)(r + 1) * a.heads] : 0.f;
        const SsdDecays g = ssd_decays(rate, d0, d1);
        const double row[2] = {g.first, g.second};
        const float step[2] = {d0, d1};
        SsdTcDecay& d = s_d[b];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          d.g[k][r + e] = row[e];
          d.eg[k][r + e] = exp2f((float)row[e]);
          d.dt[k][r + e] = step[e];
          d.w[k][r + e] = step[e] * exp2f((float)(g.total - row[e]));
        }
        if (lane == (rows - 1) / 2) d.all[k] = exp2f((float)((rows & 1) ? g.first : g.second));
      }
      if (rows < kStRows) {
        cp_async_wait<0>();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      if (rows < kStRows || k < 2) arrive(&bars.full[b]);                 // the third warp's arrival went with the whole chunk's copies
    }
    cp_async_wait<0>();
    if (s_abort) {                                                        // copies in flight land before the block's memory goes
      const unsigned long long w0 = global_ns();
      while (global_ns() - w0 < 1000000ull) {}
    }
  } else if (lane == 0) {
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (8u << 24);        // 128 lanes
    auto n_of = [](int n) { return (uint32_t)(n >> 3) << 17; };
    auto one = [&](uint64_t* bar, uint32_t parity, int code) { return mbar_wait(bar, parity & 1u, abort_flag, p.status, code); };
    bool ok = true;
    for (int ch = 0; ch < n_chunks && ok; ++ch) {
      const int b = ch & 1;
      const uint32_t base = smem_u32(sm + b * kStBuf), planes = smem_u32(sm + kStP);
      if (!(ok = one(&bars.full[b], ch >> 1, 57))) break;
      tc_fence_after();
#pragma unroll
      for (int k = 0; k < 8; ++k)
        tc_mma_bf16(tmem + kStZ, make_smem_desc(base + kStC + k / 4 * 2 * kStPlane) + 2 * (k % 4), make_smem_desc(base + kStB + k / 4 * kStPlane) + 2 * (k % 4),
                    idesc | n_of(kStRows), k > 0);
      tc_commit(&bars.z_done);
      if (!(ok = one(&bars.s_ready, ch, 59) && one(&bars.o_free, ch + 1, 58))) break;
      tc_fence_after();
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint64_t c = make_smem_desc(base + kStC + k / 4 * 2 * kStPlane) + 2 * (k % 4);
        const uint32_t s = tmem + kStD + 16 * k;
        tc_mma_bf16_ts(tmem + kStO1, s + 8, c, idesc | n_of(kStRows), k > 0);
        tc_mma_bf16_ts(tmem + kStO1, s, c, idesc | n_of(kStRows), 1u);
      }
      tc_commit(&bars.r_done);
      if (!(ok = one(&bars.x_ready, ch, 60) && one(&bars.r_done, ch, 66))) break;          // the planes have been read: their place is taken
      tc_fence_after();
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint64_t key = make_smem_desc_mn(base + kStB + k * 2048, kStPlane);
        tc_mma_bf16_ts(tmem + kStD, tmem + kStWl + 8 * k, key, idesc | (1u << 16) | n_of(kStN), k > 0);
        tc_mma_bf16_ts(tmem + kStD, tmem + kStWh + 8 * k, key, idesc | (1u << 16) | n_of(kStN), 1u);
      }
      tc_commit(&bars.s_done);
      if (!(ok = one(&bars.p_ready, ch, 61) && one(&bars.r_ready, ch, 67))) break;
      tc_fence_after();
      // 16 tokens reach the columns from theirs on.  First 32 columns at a time, then the 16 left; products into the same columns keep their
      // order only if they have the same shape, hence the wait between.
      auto add = [&](int k, int c0, int n) {
        const uint64_t x = make_smem_desc(smem_u32(sm + kStXt + b * 2 * kStPlane)) + 2 * k;
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int hh = 0; hh < 2; ++hh)
            tc_mma_bf16(tmem + (hh ? kStO2 : kStO1) + c0, x, make_smem_desc(planes + (hh * 2 + 1 - e) * kStPlane + c0 * 128) + 2 * k, idesc | n_of(n), 1u);
      };
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (k == 0) add(k, 0, 32);
        add(k, 32, 32);
      }
      tc_commit(&bars.h_done);
      if (!(ok = one(&bars.h_done, ch, 68))) break;
      tc_fence_after();
      add(1, 16, 16);
      add(3, 48, 16);
      tc_commit(&bars.o_done);
      tc_commit(&bars.free[b]);
    }
    tc_commit(&bars.drain);
    const unsigned long long w0 = global_ns();
    while (!mbar_try_wait(&bars.drain, 0) && global_ns() - w0 < kWaitLimitNs) {}
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 23) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

}  // namespace msa

using namespace msa;

extern "C" int msa_lm_ssd_walk_supported(int32_t heads, int32_t groups, int32_t n_state, int32_t vdim) {
  return n_state == kStN && vdim == kStV && groups > 0 && heads % (2 * groups) == 0;
}

extern "C" int msa_lm_ssd_walk(const msa_lm_ssd_args* a, const void* xbc, const float* dt, int32_t* status, void* stream) {
  MSA_OK_OR_RETURN(ssd_check(a, "ssd_walk"));
  MSA_REQUIRE(a->dtype == MSA_BF16 && msa_lm_ssd_walk_supported(a->heads, a->groups, a->n_state, a->vdim) && xbc && dt && status,
              "ssd_walk: unsupported sizes or null pointer");
  MSA_REQUIRE(aligned16(xbc) && a->n_seq - a->n_decode < 65536, "ssd_walk: alignment or too many portions");
  MSA_REQUIRE(aligned16(a->proj) && a->proj_stride % 8 == 0, "ssd_walk: rows of proj off the 16-byte boundary");
  if (a->n_seq == a->n_decode) return MSA_OK;
  const int inner = a->heads * kStV, chan = inner + 2 * a->groups * kStN;
  CUtensorMap mx, mg;
  MSA_OK_OR_RETURN(make_map(&mx, xbc, (uint64_t)(a->n_tok - a->n_decode), chan, chan, 64, kStRows));
  MSA_OK_OR_RETURN(make_map(&mg, a->proj, (uint64_t)a->n_tok, inner, a->proj_stride, 64, kStRows));
  static DeviceSmem configured{};
  MSA_OK_OR_RETURN(ensure_dynamic_smem(ssd_tc_kernel, kStSmem, configured));
  ssd_tc_kernel<<<dim3((unsigned)a->heads / 2, (unsigned)(a->n_seq - a->n_decode)), kStThreads, kStSmem, (cudaStream_t)stream>>>(
      mx, mg, SsdTcParams{*a, (const __nv_bfloat16*)xbc, dt, status});
  MSA_LAUNCH_OK("ssd_tc_kernel");
  return MSA_OK;
}
