// Argument checks shared by the two files of the recurrences.
#pragma once
#include "lm_common.cuh"

namespace msa {
int wkv_check(const msa_lm_wkv_args* a, const char* what);
int ssd_check(const msa_lm_ssd_args* a, const char* what);

// A head's log2 decays of a chunk of up to 64 tokens summed up by one warp, two tokens per lane (steps d0, d1; 0 behind the last one): the
// sums up to and with each of the two, and the last lane's.  One text for both ways over the chunks, which have to come to the same bits.
struct SsdDecays { double first, second, total; };
__device__ __forceinline__ SsdDecays ssd_decays(double rate, float d0, float d1) {
  const int lane = threadIdx.x & 31;
  double sum = rate * d0 + rate * d1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double x = __shfl_up_sync(0xffffffffu, sum, o);
    if (lane >= o) sum += x;
  }
  return {sum - rate * d1, sum, __shfl_sync(0xffffffffu, sum, 31)};
}
}  // namespace msa
