// What the chunk-of-columns recurrences (delta_rule.cu, dplr_delta.cu) share: a thread holds two neighbouring columns of the
// state and a sixteenth of their entries as pairs (d, d + 1), so that products run two entries an instruction, and the sixteen
// lanes of a column group join their partial sums.
#pragma once
#include "common.cuh"

namespace llmi {

constexpr int REC_BATCH = 4;          // tokens a barrier
constexpr int REC_STAGES = 3;         // batches of tokens in shared memory

__device__ __forceinline__ float2 pair_of(float v) { return make_float2(v, v); }
// (.x of the pairs: entries 0 and 2 of a chunk of four, .y: 1 and 3, as two chains of single products would have it)
__device__ __forceinline__ float pair_sum(float2 v) { return v.x + v.y; }

// Four sums over the sixteen lanes of a group at once: (a, b) come back to every lane; the return value is c's sum in the
// lanes with sub & 3 = 2 and d's in those with sub & 3 = 3.  Each sum has the tree of a butterfly over lanes 1, 2, 4, 8 apart
// (the same bits), but the values part ways round by round: seven shuffles instead of sixteen.
__device__ __forceinline__ float join_four(float& a, float& b, float c, float d, int sub) {
  const bool odd = sub & 1, high = sub & 2;
  float first = odd ? b : a, second = odd ? d : c;
  first += __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
  second += __shfl_xor_sync(0xffffffffu, odd ? c : d, 1);
  float m = high ? second : first;
  m += __shfl_xor_sync(0xffffffffu, high ? first : second, 2);
  m += __shfl_xor_sync(0xffffffffu, m, 4);
  m += __shfl_xor_sync(0xffffffffu, m, 8);
  a = __shfl_sync(0xffffffffu, m, 0, 16);
  b = __shfl_sync(0xffffffffu, m, 1, 16);
  return m;
}

__device__ __forceinline__ void rec_copy16(void* dst, const void* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void rec_copy4(void* dst, const void* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

// Four entries (64 i + 4 sub ..) of two neighbouring columns, [column][chunk][pair of entries], from or to rows of D entries a column.
template <int NI>
__device__ __forceinline__ void rec_load_state(float2 (&S)[2][NI][2], const float* S_g, int D, int sub, bool holds) {
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const float4 v = holds ? *reinterpret_cast<const float4*>(S_g + c * D + 64 * i + 4 * sub) : make_float4(0.f, 0.f, 0.f, 0.f);
      S[c][i][0] = make_float2(v.x, v.y);
      S[c][i][1] = make_float2(v.z, v.w);
    }
}
template <int NI>
__device__ __forceinline__ void rec_store_state(const float2 (&S)[2][NI][2], float* S_g, int D, int sub) {
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int i = 0; i < NI; ++i)
      *reinterpret_cast<float4*>(S_g + c * D + 64 * i + 4 * sub) = make_float4(S[c][i][0].x, S[c][i][0].y, S[c][i][1].x, S[c][i][1].y);
}

}  // namespace llmi
