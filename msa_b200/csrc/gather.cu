// Fetch of the selected documents' pooled K/V from the pinned host bank.
//
// The host bank keeps a document's chunks contiguous ([chunk][K|V][Hkv][D]), so one
// selected document is one linear run of host memory.  The gather kernel reads it through
// the device-visible mapping with 16-byte loads (PCIe reads, no staging copy, no host
// thread involved) and scatters it into the head-major [Hkv, entries, D] layout the
// attention path consumes.  Bound by PCIe bandwidth: 2*chunks*Hkv*D*e bytes per document.
#include <cstdlib>

#include "common.cuh"

namespace msa {

constexpr int kPlanWarps = 32;         // samples in work at a time
constexpr int kPlanMaxK = 64;          // two winners per lane
constexpr int kPlanSamples = 1024;     // samples between two scans of the totals

// One warp per sample, lane l holds winners l and l + 32.  What bounds the plan is the chain of dependent reads (winner -> shard
// -> document -> length and offset), so a sample's winners take each step of it together, and their order by (owner rank, local
// id) comes from counting with shuffles.  6.7 us for one question, 11.5 us for 32 (one thread
// per sample with an insertion sort: 13 and 30 us).
//
// status[2] counts winners that were dropped because their owner rank or local id does not exist in the
// directory (a corrupt candidate, or a directory that no longer matches the bank): nothing is read for them.
__global__ void __launch_bounds__(kPlanWarps * 32)
gather_plan_kernel(const int64_t* __restrict__ sel_local, const int32_t* __restrict__ sel_rank, int n_seq, int k,
                   int world, const int64_t* __restrict__ shard_doc_base, long long n_dir_rows,
                   const int64_t* __restrict__ doc_chunk_offset, const int32_t* __restrict__ doc_chunk_len,
                   const uint64_t* __restrict__ shard_kv_base, long long chunk_bytes, long long sample_stride,
                   int64_t* __restrict__ plan, int64_t* __restrict__ n_sel, int64_t* __restrict__ total,
                   int64_t* total_host, int64_t* report, int32_t* status, int64_t* __restrict__ resident, int slot_len) {
  constexpr long long kNone = 0x7fffffffffffffffll;
  __shared__ long long s_base[kPlanSamples];      // totals of the samples, then what stands in front of each
  __shared__ long long s_warp[kPlanWarps], s_carry;
  __shared__ unsigned char s_free[kPlanWarps][kPlanMaxK];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const unsigned all = 0xffffffffu;
  if (threadIdx.x == 0) s_carry = 0;
  for (int first = 0; first < n_seq; first += kPlanSamples) {
    const int here = min(kPlanSamples, n_seq - first);
    for (int i = warp; i < here; i += kPlanWarps) {
      const int b = first + i;
      long long key[2], len[2], src[2];
      int dropped = 0, n = 0;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int j = lane + 32 * u;
        key[u] = kNone; len[u] = 0; src[u] = 0;
        if (j < k) {
          const long long lid = sel_local[(long long)b * k + j];
          const int r = sel_rank ? sel_rank[(long long)b * k + j] : 0;
          if (lid > 0) {                                     // else: dummy document or invalidated winner
            // shard r owns directory rows [base[r], base[r+1]); row base[r] is its dummy document
            const bool known = r >= 0 && r < world;
            const long long lo = known ? shard_doc_base[r] : 0, hi = !known ? 0 : r + 1 < world ? shard_doc_base[r + 1] : n_dir_rows;
            if (known && lid < hi - lo) {
              key[u] = ((long long)r << 40) | lid;
              len[u] = max(doc_chunk_len[lo + lid], 0);
              src[u] = (long long)(shard_kv_base[r] + (unsigned long long)(doc_chunk_offset[lo + lid] * chunk_bytes));
            } else {
              ++dropped;
            }
          }
        }
        n += __popc(__ballot_sync(all, key[u] != kNone));
      }
      if (dropped && status) atomicAdd(status + 2, dropped);
      // place[u] winners stand before this one in the order of the keys (equal keys: by index), with ahead[u] entries
      int place[2] = {0, 0};
      long long ahead[2] = {0, 0};
      bool again[2] = {false, false};                        // an equal key stands before
      for (int j = 0; j < k; ++j) {
        const long long other = __shfl_sync(all, j < 32 ? key[0] : key[1], j & 31), entries = __shfl_sync(all, j < 32 ? len[0] : len[1], j & 31);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const bool same = other == key[u] && j < lane + 32 * u;
          if (other < key[u] || same) { ++place[u]; ahead[u] += entries; }
          again[u] = again[u] || same;
        }
      }
      // Resident set (a decode loop that refreshes the same segment every step): the sample's room is k slots of
      // slot_len entries, resident[b][s] is the document whose entries slot s holds.  When the k winners are all
      // valid and every one holds exactly slot_len entries, the winners that are already in a slot stay where they
      // are and only the others are planned, into the slots of the documents that dropped out.  Any other sample
      // is planned in full (below) and its table is cleared.
      bool keep_slots = resident != nullptr && n == k && sample_stride == (long long)k * slot_len;
      keep_slots = __all_sync(all, keep_slots && (lane >= k || len[0] == slot_len) && (lane + 32 >= k || len[1] == slot_len));
      long long mine;
      if (keep_slots) {
        int64_t* res = resident + (long long)b * k;
        bool hit[2] = {false, false}, kept[2] = {false, false};
        long long have[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) have[u] = lane + 32 * u < k ? res[lane + 32 * u] : -1;
        for (int j = 0; j < k; ++j) {
          const long long slot_has = __shfl_sync(all, j < 32 ? have[0] : have[1], j & 31), winner = __shfl_sync(all, j < 32 ? key[0] : key[1], j & 31);
#pragma unroll
          for (int u = 0; u < 2; ++u) { hit[u] = hit[u] || slot_has == key[u]; kept[u] = kept[u] || winner == have[u]; }
        }
        unsigned fresh_lo = 0, fresh_hi = 0;                 // winners without a slot, by their place
        unsigned free_before = 0;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int j = lane + 32 * u;
          hit[u] = hit[u] && !again[u];
          const unsigned bit = j < k && !hit[u] ? 1u << (place[u] & 31) : 0u;
          fresh_lo |= __reduce_or_sync(all, place[u] < 32 ? bit : 0u);
          fresh_hi |= __reduce_or_sync(all, place[u] < 32 ? 0u : bit);
          const bool open = j < k && !kept[u];
          const unsigned ballot = __ballot_sync(all, open);
          if (open) s_free[warp][free_before + __popc(ballot & ((1u << lane) - 1u))] = (unsigned char)j;
          free_before += __popc(ballot);
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int j = lane + 32 * u;
          if (j >= k) continue;
          int64_t* row = plan + ((long long)b * k + place[u]) * 4;
          const unsigned below_lo = place[u] < 32 ? fresh_lo & ((1u << place[u]) - 1u) : fresh_lo;
          const unsigned below_hi = place[u] < 32 ? 0u : fresh_hi & ((1u << (place[u] - 32)) - 1u);
          const unsigned turn = __popc(below_lo) + __popc(below_hi);
          const bool load = !hit[u] && turn < free_before;   // (a document named twice may find no slot)
          const int slot = load ? s_free[warp][turn] : 0;
          if (load) res[slot] = key[u];
          row[0] = load ? src[u] : 0;
          row[1] = load ? slot_len : 0;
          row[2] = load ? (long long)slot * slot_len : 0;
          row[3] = b;
        }
        __syncwarp();
        mine = (long long)k * slot_len;
      } else {
        const long long room = sample_stride > 0 ? sample_stride : kNone;
        mine = 0;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int j = lane + 32 * u;
          const long long begin = min(ahead[u], room), end = min(ahead[u] + len[u], room);     // past the sample's room: cut
          mine = max(mine, end);
          if (j < k) {
            if (resident != nullptr) resident[(long long)b * k + j] = -1;
            int64_t* row = plan + ((long long)b * k + place[u]) * 4;
            row[0] = src[u];
            row[1] = end - begin;
            row[2] = end > begin ? begin : 0;   // offset inside the sample; packed mode adds the sample's base below
            row[3] = b;
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mine = max(mine, __shfl_xor_sync(all, mine, o));
      }
      if (lane == 0) { s_base[i] = mine; n_sel[b] = mine; }
    }
    __syncthreads();
    // exclusive scan of the totals, carried between rounds
    long long v = threadIdx.x < here ? s_base[threadIdx.x] : 0, sum = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const long long up = __shfl_up_sync(all, sum, o); if (lane >= o) sum += up; }
    if (lane == 31) s_warp[warp] = sum;
    __syncthreads();
    long long before = s_carry, round = 0;
    for (int w = 0; w < kPlanWarps; ++w) { if (w < warp) before += s_warp[w]; round += s_warp[w]; }
    if (threadIdx.x < here) s_base[threadIdx.x] = before + sum - v;
    __syncthreads();
    if (threadIdx.x == 0) s_carry += round;
    if (sample_stride == 0)
      for (int i = threadIdx.x; i < here * k; i += kPlanWarps * 32) {
        int64_t* row = plan + ((long long)first * k + i) * 4;
        if (row[1] > 0) row[2] += s_base[i / k];
      }
    __syncthreads();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    total[0] = s_carry;
    if (total_host) *reinterpret_cast<volatile int64_t*>(total_host) = s_carry;
    if (report) {                               // what the host reads back after a synchronise: the total and the status words
      volatile int64_t* out = report;
      out[0] = s_carry;
      for (int w = 0; w < 2; ++w) {
        const unsigned lo = status ? (unsigned)atomicAdd(status + 2 * w, 0) : 0u, hi = status ? (unsigned)atomicAdd(status + 2 * w + 1, 0) : 0u;
        out[1 + w] = (int64_t)(((unsigned long long)hi << 32) | lo);
      }
    }
  }
}

constexpr int kGatherThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kGatherThreads)
gather_kernel(const int64_t* __restrict__ plan, int n_items, int n_kv_heads, int head_dim, T* __restrict__ out_k,
              T* __restrict__ out_v, long long out_head_stride, long long out_entries, long long out_sample_stride,
              const int64_t* __restrict__ total) {
  if (total) {                                     // packed by what the plan found: [heads, total, head_dim], in room for out_entries
    out_entries = min(out_entries, (long long)*total);
    out_head_stride = out_entries * head_dim;
  }
  constexpr int V = Elem<T>::kVec;
  const int vec_half = n_kv_heads * head_dim / V;  // 16-byte vectors in one chunk's K (or V)
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
  const int64_t* row = plan + (long long)item * 4;
  const long long dst0 = row[2];
  // clamp once: nothing is read for entries that have no room (out_entries counts per sample when the
  // destination is strided by sample, over the whole output otherwise)
  const long long len = min((long long)row[1], out_entries - dst0);
  if (len <= 0) continue;
  const uint4* src = reinterpret_cast<const uint4*>((uintptr_t)row[0]);
  const long long sample_off = out_sample_stride * row[3];
  const long long n_vec = len * 2 * vec_half;
  // each thread keeps four independent 16-byte PCIe reads in flight
  for (long long v0 = threadIdx.x; v0 < n_vec; v0 += 4ll * kGatherThreads) {
    uint4 val[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long v = v0 + (long long)u * kGatherThreads;
      if (v < n_vec) val[u] = src[v];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long v = v0 + (long long)u * kGatherThreads;
      if (v >= n_vec) continue;
      const long long chunk = v / (2 * vec_half);
      const int w = (int)(v % (2 * vec_half));
      const int in_half = w % vec_half;
      const int h = (in_half * V) / head_dim, d = (in_half * V) % head_dim;
      const long long entry = dst0 + chunk;
      T* dst = (w < vec_half ? out_k : out_v) + sample_off + (long long)h * out_head_stride + entry * head_dim + d;
      *reinterpret_cast<uint4*>(dst) = val[u];
    }
  }
  }
}

}  // namespace msa

using namespace msa;

// The plan and gather kernels run on a side stream beside kernels that need almost all of an SM's shared memory
// (the persistent routing kernels).  A kernel with little shared memory of its own leaves the SM configured for a
// large L1, and a CTA that needs 200 KB cannot join it there until the SM has drained: measured on B200, a 3.2 GB
// routing launch took 758 us instead of 461 us next to a 24-CTA gather, because the routing CTAs of the occupied
// SMs started only when the first wave had ended.  Asking for the largest shared-memory carve-out keeps those SMs
// open (507 us).
static int prefer_shared_carveout() {
  static bool done[kMaxDevices] = {};
  int device = 0;
  MSA_OK_OR_RETURN(current_device(&device));
  if (done[device] || getenv("MSA_B200_GATHER_DEFAULT_CARVEOUT")) return MSA_OK;
  MSA_CUDA_OK(cudaFuncSetAttribute(gather_kernel<__nv_bfloat16>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   cudaSharedmemCarveoutMaxShared));
  MSA_CUDA_OK(cudaFuncSetAttribute(gather_kernel<float>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   cudaSharedmemCarveoutMaxShared));
  MSA_CUDA_OK(cudaFuncSetAttribute(gather_plan_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   cudaSharedmemCarveoutMaxShared));
  done[device] = true;
  return MSA_OK;
}

namespace {
int gather_plan_launch(const int64_t* sel_local, const int32_t* sel_rank, int32_t n_seq, int32_t k, int32_t world,
                       const int64_t* shard_doc_base, int64_t n_dir_rows, const int64_t* doc_chunk_offset,
                       const int32_t* doc_chunk_len, const uint64_t* shard_kv_base, int64_t chunk_bytes,
                       int64_t sample_stride, int64_t* plan, int64_t* n_sel, int64_t* total, int64_t* total_host_mapped,
                       int64_t* report, int32_t* status, int64_t* resident, int32_t slot_len, void* stream) {
  MSA_REQUIRE(sel_local && shard_doc_base && doc_chunk_offset && doc_chunk_len && shard_kv_base && plan && n_sel &&
                  total, "gather_plan: null pointer");
  MSA_REQUIRE(n_seq >= 0 && k >= 1 && k <= kPlanMaxK && world >= 1, "gather_plan: bad sizes (k must be <= %d)",
              kPlanMaxK);
  MSA_REQUIRE(n_dir_rows >= world, "gather_plan: n_dir_rows=%lld is smaller than the %d dummy rows of the shards",
              (long long)n_dir_rows, world);
  MSA_REQUIRE(chunk_bytes > 0 && chunk_bytes % 16 == 0, "gather_plan: chunk_bytes must be a multiple of 16");
  MSA_REQUIRE(sample_stride >= 0, "gather_plan: sample_stride must not be negative");
  MSA_REQUIRE(resident == nullptr || (slot_len > 0 && sample_stride == (int64_t)k * slot_len),
              "gather_plan: a resident table needs sample_stride == k * slot_len");
  MSA_OK_OR_RETURN(prefer_shared_carveout());
  gather_plan_kernel<<<1, kPlanWarps * 32, 0, (cudaStream_t)stream>>>(
      sel_local, sel_rank, n_seq, k, world, shard_doc_base, n_dir_rows, doc_chunk_offset, doc_chunk_len, shard_kv_base,
      chunk_bytes, sample_stride, plan, n_sel, total, total_host_mapped, report, status, resident, slot_len);
  MSA_LAUNCH_OK("gather_plan_kernel");
  return MSA_OK;
}
}  // namespace

extern "C" int msa_gather_plan(const int64_t* sel_local, const int32_t* sel_rank, int32_t n_seq, int32_t k,
                               int32_t world, const int64_t* shard_doc_base, int64_t n_dir_rows,
                               const int64_t* doc_chunk_offset, const int32_t* doc_chunk_len,
                               const uint64_t* shard_kv_base, int64_t chunk_bytes, int64_t sample_stride,
                               int64_t* plan, int64_t* n_sel, int64_t* total, int64_t* total_host_mapped,
                               int32_t* status, void* stream) {
  return gather_plan_launch(sel_local, sel_rank, n_seq, k, world, shard_doc_base, n_dir_rows, doc_chunk_offset, doc_chunk_len,
                            shard_kv_base, chunk_bytes, sample_stride, plan, n_sel, total, total_host_mapped, nullptr, status,
                            nullptr, 0, stream);
}

extern "C" int msa_gather_plan_report(const int64_t* sel_local, const int32_t* sel_rank, int32_t n_seq, int32_t k,
                                      int32_t world, const int64_t* shard_doc_base, int64_t n_dir_rows,
                                      const int64_t* doc_chunk_offset, const int32_t* doc_chunk_len,
                                      const uint64_t* shard_kv_base, int64_t chunk_bytes, int64_t sample_stride,
                                      int64_t* plan, int64_t* n_sel, int64_t* total, int64_t* report,
                                      int32_t* status, void* stream) {
  MSA_REQUIRE(report != nullptr, "gather_plan_report: null pointer");
  return gather_plan_launch(sel_local, sel_rank, n_seq, k, world, shard_doc_base, n_dir_rows, doc_chunk_offset, doc_chunk_len,
                            shard_kv_base, chunk_bytes, sample_stride, plan, n_sel, total, nullptr, report, status, nullptr, 0,
                            stream);
}

extern "C" int msa_gather_plan_resident(const int64_t* sel_local, const int32_t* sel_rank, int32_t n_seq, int32_t k,
                                        int32_t world, const int64_t* shard_doc_base, int64_t n_dir_rows,
                                        const int64_t* doc_chunk_offset, const int32_t* doc_chunk_len,
                                        const uint64_t* shard_kv_base, int64_t chunk_bytes, int32_t slot_len,
                                        int64_t* resident, int64_t* plan, int64_t* n_sel, int64_t* total,
                                        int32_t* status, void* stream) {
  MSA_REQUIRE(resident != nullptr, "gather_plan_resident: null pointer");
  return gather_plan_launch(sel_local, sel_rank, n_seq, k, world, shard_doc_base, n_dir_rows, doc_chunk_offset, doc_chunk_len,
                            shard_kv_base, chunk_bytes, (int64_t)k * slot_len, plan, n_sel, total, nullptr, nullptr, status,
                            resident, slot_len, stream);
}

static int gather_launch(const int64_t* plan, int32_t n_items, int32_t dtype, int32_t n_kv_heads,
                         int32_t head_dim, void* out_k, void* out_v, int64_t out_head_stride,
                         int64_t out_entries, int64_t out_sample_stride, const int64_t* total, int32_t max_ctas, void* stream) {
  MSA_REQUIRE(dtype_ok(dtype), "gather_run: unknown dtype %d", dtype);
  MSA_REQUIRE(plan && n_items >= 0 && n_kv_heads > 0 && head_dim > 0 && max_ctas >= 0 && out_sample_stride >= 0,
              "gather_run: bad arguments");
  // The link is saturated by a few hundred KB of reads in flight (16 KB per CTA).  Measured on B200 with
  // 32 KiB documents: 49.8 GB/s alone from 12 CTAs up; next to the HBM-bound decode-time scoring the
  // neighbour loses 0.18 ms per layer with 512 CTAs and 0.05 ms with 16-32; next to the tensor-bound prefill
  // scoring one CTA per document is best (35 GB/s against 20 GB/s at 24 CTAs).
  const int grid = (max_ctas > 0 && max_ctas < n_items) ? max_ctas : n_items;
  const int vec = 16 / (int)dtype_size(dtype);
  MSA_REQUIRE(head_dim % vec == 0 && out_head_stride % vec == 0 && out_sample_stride % vec == 0,
              "gather_run: rows must be 16-byte multiples");
  if (n_items == 0 || out_entries == 0) return MSA_OK;
  MSA_REQUIRE(out_k && out_v && aligned16(out_k) && aligned16(out_v), "gather_run: bad output pointers");
  MSA_OK_OR_RETURN(prefer_shared_carveout());
  if (dtype == MSA_BF16)
    gather_kernel<__nv_bfloat16><<<grid, kGatherThreads, 0, (cudaStream_t)stream>>>(
        plan, n_items, n_kv_heads, head_dim, (__nv_bfloat16*)out_k, (__nv_bfloat16*)out_v, out_head_stride, out_entries,
        out_sample_stride, total);
  else
    gather_kernel<float><<<grid, kGatherThreads, 0, (cudaStream_t)stream>>>(
        plan, n_items, n_kv_heads, head_dim, (float*)out_k, (float*)out_v, out_head_stride, out_entries,
        out_sample_stride, total);
  MSA_LAUNCH_OK("gather_kernel");
  return MSA_OK;
}

extern "C" int msa_gather_run(const int64_t* plan, int32_t n_items, int32_t dtype, int32_t n_kv_heads,
                              int32_t head_dim, void* out_k, void* out_v, int64_t out_head_stride,
                              int64_t out_entries, int64_t out_sample_stride, int32_t max_ctas, void* stream) {
  return gather_launch(plan, n_items, dtype, n_kv_heads, head_dim, out_k, out_v, out_head_stride, out_entries, out_sample_stride, nullptr, max_ctas,
                       stream);
}

extern "C" int msa_gather_run_total(const int64_t* plan, int32_t n_items, int32_t dtype, int32_t n_kv_heads, int32_t head_dim, void* out_k,
                                    void* out_v, int64_t capacity, const int64_t* total, int32_t max_ctas, void* stream) {
  MSA_REQUIRE(total && capacity >= 0, "gather_run_total: null total or negative capacity");
  return gather_launch(plan, n_items, dtype, n_kv_heads, head_dim, out_k, out_v, 0, capacity, 0, total, max_ctas, stream);
}
