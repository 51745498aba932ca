// x @ w.T for the few rows of a decode step (bf16 operands, fp32 accumulation), optionally with the feed-forward's gate.
//
// Bound by the weights, which come from HBM once: 2 bytes per weight, whatever the number of rows.  Every warp streams 16 or 32
// weight rows of a slice of K straight into registers, 64-byte pieces of a row by four neighbouring lanes, 8 KB in flight, and
// multiplies them with m16n8k16; the warps of a block share the rows and split K, and meet in shared memory in a fixed order.
// The order of K inside a block of 32 is free as long as both operands follow it: lane t of a quad holds k = 8t .. 8t+7, one
// 16-byte load, and feeds them to two products.  The kernel is launched early (programmatic dependent launch): the first pieces of the
// weights, which no kernel of a step writes, are fetched while the kernel before it still runs; all else waits for that kernel.
//
// Measured (bf16 out, 8 rows, a chain of products with fresh weights in a CUDA graph; torch.mm beside it): 2048 x 2048 3.5 us
// (6.7), 2048 x 6144 6.5 (14.9), 2048 x 10240 9.2 (23.1), 12288 x 2048 10.9 (9.9 and 1.8 for the gate, which is part of this one).
// Weights through a TMA ring into tcgen05.mma with 16 columns took 12.9 us for 12288 x 2048 and 12.4 for 2048 x 10240: four
// products per 16 KB cost about as much as fetching them, and start and end of a tile another 3 us.  With 16 rows this kernel's x takes as
// much from L2 as w from HBM, and a whole decode step was no faster than with the library's products (459 us both).
#include "lm_common.cuh"

namespace msa {

constexpr int kRgMaxRows = 8, kRgMaxWarps = 16, kRgBlock = 32, kRgTurn = 4;   // kRgBlock: K of a 16-byte load per lane

struct RowsGemmParams {
  const __nv_bfloat16* x; long long x_stride, x_batch;
  const __nv_bfloat16* w; long long w_stride, w_batch;
  void* out; long long out_stride, out_batch;
  int n, features, k, early, out_f32;                              // features: output columns (half the rows of w with the activation)
};

__device__ __forceinline__ uint4 ld_stream(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
// What the kernel before this one wrote: past L1, and not before the wait above it.
__device__ __forceinline__ uint4 ld_fresh(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
// The same, into shared memory.  Without `in`: zeros.
__device__ __forceinline__ void send_fresh(uint32_t dst, const __nv_bfloat16* p, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(p), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// MT: 16-row tiles of w per warp (with the activation 2: gate rows and the up rows that belong to them).  A block's rows of w:
// 16 * MT; blockDim / 32 slices of K.
// AHEAD: x comes through shared memory, two turns ahead.  Loaded when its turn is there, it costs each turn its way from L2: 2048 x 10240
// took 10.4 us so and 9.2 ahead, 2048 x 6144 6.9 and 6.5, 10304 x 2048 10.6 and 9.2, 32768 x 2048 26.1 and 23.7 (8 rows).  With two turns or
// fewer there is nothing to be ahead of (2048 x 2048 3.5 and 4.0), and with the activation it was slower (12288 x 2048 10.9 and 11.5, 6144 x
// 1024 3.6 and 5.2: fewer registers, more blocks on the SMs that are free first).
template <int MT, bool ACT, bool AHEAD>
__global__ void __launch_bounds__(kRgMaxWarps * 32) rows_gemm_kernel(const RowsGemmParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int kRows = 16 * MT, kPitch = kRows + 4, KB = kRgTurn / MT;   // KB: blocks of K fetched at once
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, warps = blockDim.x / 32, g = lane / 4, t = lane % 4;
  const int cols = ACT ? 16 : kRows, f0 = blockIdx.x * cols;       // output columns of this block
  grid_launch_dependents();
  // x of two turns: a lane's own pieces, which no other lane reads.  Then the sums, [warp][row of x][kPitch].
  uint4* s_x = reinterpret_cast<uint4*>(smem) + warp * 2 * KB * 32 + lane;
  float* s_part = reinterpret_cast<float*>(smem + (AHEAD ? (size_t)warps * 2 * KB * 512 : 0));
  const __nv_bfloat16* w = p.w + blockIdx.y * p.w_batch + 8 * t;
  const __nv_bfloat16* wr[MT][2];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {                                  // rows past the last one repeat it; nobody reads their sums
      int r = min(f0 + (ACT ? 0 : 16 * m) + g + 8 * h, p.features - 1);
      if (ACT && m == 1) r += p.features;
      wr[m][h] = w + r * p.w_stride;
    }
  const __nv_bfloat16* x = p.x + blockIdx.y * p.x_batch + 8 * t;
  x += min(g, p.n - 1) * p.x_stride;
  const int blocks = (p.k + kRgBlock - 1) / kRgBlock;
  const int b0 = (int)((long long)blocks * warp / warps), b1 = (int)((long long)blocks * (warp + 1) / warps);
  const int k_end = min(b1 * kRgBlock, p.k) - 8 * t;               // this lane's pieces start below it
  const uint4 zero = make_uint4(0, 0, 0, 0);
  float acc[MT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[m][i] = 0.f;
  uint4 a[2][KB][MT][2];                                           // one turn in use while the other is on its way
  auto fetch = [&](uint4 (&a)[KB][MT][2], int b) {
#pragma unroll
    for (int i = 0; i < KB; ++i) {
      const int k = (b + i) * kRgBlock;
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) a[i][m][h] = k < k_end ? ld_stream(wr[m][h] + k) : zero;
    }
  };
  auto send = [&](int turn, int b) {
#pragma unroll
    for (int i = 0; i < KB; ++i) {
      const bool in = g < p.n && (b + i) * kRgBlock < k_end;          // rows past the last one: zeros, nobody reads their sums
      send_fresh((uint32_t)__cvta_generic_to_shared(s_x + (turn * KB + i) * 32), in ? x + (b + i) * kRgBlock : x, in);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto multiply = [&](const uint4 (&a)[KB][MT][2], int turn, int b) {
    uint4 v[KB];
    if constexpr (AHEAD) asm volatile("cp.async.wait_group 1;" ::: "memory");   // the turn's pieces; the next turn's may be on their way
#pragma unroll
    for (int i = 0; i < KB; ++i) {
      if constexpr (!AHEAD) v[i] = (b + i) * kRgBlock < k_end ? ld_fresh(x + (b + i) * kRgBlock) : zero;
      else v[i] = s_x[(turn * KB + i) * 32];
    }
#pragma unroll
    for (int i = 0; i < KB; ++i)
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const uint4 lo = a[i][m][0], hi = a[i][m][1];
        mma16816(acc[m], lo.x, hi.x, lo.y, hi.y, v[i].x, v[i].y);
        mma16816(acc[m], lo.z, hi.z, lo.w, hi.w, v[i].z, v[i].w);
      }
    if constexpr (AHEAD) __syncwarp();                              // read before the next pieces land there
  };
  if (!p.early) grid_dependency_wait();
  fetch(a[0], b0);
  fetch(a[1], b0 + KB);
  if (p.early) grid_dependency_wait();
  if constexpr (AHEAD) {
    send(0, b0);
    send(1, b0 + KB);
  }
  for (int b = b0; b < b1; b += 2 * KB) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      multiply(a[i], i, b + i * KB);
      if constexpr (AHEAD) send(i, b + (2 + i) * KB);
      fetch(a[i], b + (2 + i) * KB);
    }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int i = 0; i < 4; ++i) s_part[(warp * kRgMaxRows + 2 * t + (i & 1)) * kPitch + 16 * m + g + 8 * (i >> 1)] = acc[m][i];
  __syncthreads();
  for (int i = threadIdx.x; i < p.n * cols; i += blockDim.x) {
    const int row = i / cols, c = i % cols, f = f0 + c;
    if (f >= p.features) continue;
    float v = 0.f, u = 0.f;
    for (int q = 0; q < warps; ++q) {
      v += s_part[(q * kRgMaxRows + row) * kPitch + c];
      if constexpr (ACT) u += s_part[(q * kRgMaxRows + row) * kPitch + 16 + c];
    }
    if constexpr (ACT) v = silu_f(v) * u;
    const long long o = blockIdx.y * p.out_batch + row * p.out_stride + f;
    if (p.out_f32) reinterpret_cast<float*>(p.out)[o] = v;
    else reinterpret_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(v);
  }
}

template <int MT, bool ACT, bool AHEAD>
int launch_rows_gemm(const RowsGemmParams& p, int batch, int cols, int warps, cudaStream_t stream) {
  static DeviceSmem state{};
  const size_t smem = (size_t)warps * ((AHEAD ? 2 * (kRgTurn / MT) * 512 : 0) + kRgMaxRows * (16 * MT + 4) * 4);
  auto kernel = rows_gemm_kernel<MT, ACT, AHEAD>;
  MSA_OK_OR_RETURN(ensure_dynamic_smem(kernel, smem, state));
  MSA_CUDA_OK(launch_kernel_pdl(kernel, dim3((unsigned)((p.features + cols - 1) / cols), (unsigned)batch), dim3(warps * 32), smem, stream,
                                p.early != 0, p));
  return MSA_OK;
}

template <int MT, bool ACT>
int launch_rows_gemm(const RowsGemmParams& p, int batch, cudaStream_t stream) {
  const int cols = ACT ? 16 : 16 * MT, blocks = (p.k + kRgBlock - 1) / kRgBlock;
  const long long ctas = (long long)((p.features + cols - 1) / cols) * batch;
  int n_sm = 0;
  MSA_OK_OR_RETURN(device_sm_count(&n_sm));
  int warps = ctas <= n_sm ? 16 : (ctas <= 2 * n_sm ? 8 : 4);      // 16 warps fit an SM: one block of them, two or four
  while (warps > 1 && blocks < 2 * warps) warps /= 2;              // at least 64 of K per warp
  if constexpr (!ACT)
    if (blocks > 2 * (kRgTurn / MT) * warps) return launch_rows_gemm<MT, ACT, true>(p, batch, cols, warps, stream);
  return launch_rows_gemm<MT, ACT, false>(p, batch, cols, warps, stream);
}

}  // namespace msa

using namespace msa;

extern "C" int msa_lm_rows_gemm(const msa_lm_rows_gemm_args* args, void* stream) {
  MSA_REQUIRE(args, "rows_gemm: null arguments");
  const msa_lm_rows_gemm_args a = *args;
  MSA_REQUIRE(a.x && a.w && a.out && dtype_ok(a.out_dtype), "rows_gemm: null pointer or bad dtype");
  MSA_REQUIRE(a.n > 0 && a.n <= kRgMaxRows && a.w_rows > 0 && a.k > 0 && a.batch > 0 && a.batch < 65536, "rows_gemm: sizes out of range");
  MSA_REQUIRE(!a.act || a.w_rows % 2 == 0, "rows_gemm: the activation needs as many up as gate rows");
  MSA_REQUIRE(a.k % 8 == 0 && a.x_stride % 8 == 0 && a.w_stride % 8 == 0 && aligned16(a.x) && aligned16(a.w) &&
                  (a.batch == 1 || (a.x_batch % 8 == 0 && a.w_batch % 8 == 0)),
              "rows_gemm: k and strides must be multiples of 8 elements, pointers 16-byte aligned");
  const RowsGemmParams p{(const __nv_bfloat16*)a.x, a.x_stride, a.x_batch, (const __nv_bfloat16*)a.w, a.w_stride, a.w_batch, a.out, a.out_stride,
                         a.out_batch, a.n, a.act ? a.w_rows / 2 : a.w_rows, a.k, a.early ? 1 : 0, a.out_dtype == MSA_F32 ? 1 : 0};
  cudaStream_t st = (cudaStream_t)stream;
  if (a.act) return launch_rows_gemm<2, true>(p, a.batch, st);
  int n_sm = 0;
  MSA_OK_OR_RETURN(device_sm_count(&n_sm));
  // Taller tiles halve what the rows of x take from L2.  Tiles of 16 and of 32 rows, 8 rows of x in a chain of products: 9472 x 2048 8.7 and 7.4 us,
  // 12288 x 2048 12.5 and 10.2, 16384 x 4096 26.6 and 25.1, a vocabulary of 32768 x 2048 27.2 and 24.1, of 151936 x 2048 102.5 and 94.9.
  // Below the line 32 rows are faster too (4736 x 2048 5.1 and 4.8, 8192 x 2048 7.7 and 6.6, 4096 x 4096 7.3 and 7.2) and are not taken:
  // they split K over other warps, which moves last bits.
  return (long long)a.w_rows * a.batch >= 64ll * n_sm ? launch_rows_gemm<2, false>(p, a.batch, st) : launch_rows_gemm<1, false>(p, a.batch, st);
}
