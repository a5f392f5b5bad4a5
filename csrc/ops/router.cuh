// Top-k routing of one token by one warp without shared memory: what the all-to-all's dispatch uses
// when it routes a token in the team that is about to send it, and what the stand-alone kernel
// (router.cu) does where its own way has too many candidates or is the longer one.
//
// Each lane keeps PER_LANE logits in registers (expert = j * 32 + lane, so the loads of a warp
// are coalesced). The choice is made on logit + bias, mapped to an unsigned key of the same
// order, so that a round of the arg-max is two warp reductions in hardware (redux.sync): the
// maximum key, then the lowest expert index among the lanes that hold it (ties go to the lower
// expert index, as torch.topk does). The chosen logits stay in a register of lane r for round r,
// so the softmax over them is one more pair of warp reductions; the weight is made of the plain
// logit.
#pragma once

#include <cuda_bf16.h>

#include <cfloat>
#include <cstdint>

namespace pplx::ops {

// A float that is not -0 as an unsigned of the same order; at least 1, so that 0 can mean "no candidate".
__device__ __forceinline__ uint32_t route_key_of_sum(float choice) {
  const uint32_t bits = __float_as_uint(choice);
  return max(bits ^ (static_cast<uint32_t>(static_cast<int32_t>(bits) >> 31) | 0x80000000u), 1u);
}
__device__ __forceinline__ uint32_t route_key(float choice) { return route_key_of_sum(choice + 0.0f); }   // -0 -> +0

// Softmax over the k chosen logits; lane r < k holds the r-th, the others hold -FLT_MAX and get 0.
// `span`: a power of two >= k; lanes from there on need not be looked at.
__device__ __forceinline__ float softmax_of_chosen(float my_val, int k, int lane, int span) {
  float m = my_val;
  for (int off = span >> 1; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  const float ex = lane < k ? __expf(my_val - m) : 0.f;
  float sum = ex;
  for (int off = span >> 1; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  return lane < k ? ex / sum : 0.f;
}

// All 32 lanes call. On return lane r < k holds the r-th chosen expert in *idx and its softmax
// weight in *weight; the other lanes hold (0, 0).
template <int PER_LANE>
__device__ __forceinline__ void route_token_warp(const void* logits_row, bool logits_bf16, const float* bias,
                                                 int num_experts, int k, uint32_t* idx, float* weight) {
  const int lane = threadIdx.x & 31;
  uint32_t key[PER_LANE];   // logit + bias as an order-preserving unsigned; 0 = no candidate
  float val[PER_LANE];      // logit: what the weight is made of
  #pragma unroll
  for (int j = 0; j < PER_LANE; ++j) {
    const int e = j * 32 + lane;
    float v = -FLT_MAX;
    uint32_t u = 0;
    if (e < num_experts) {
      v = logits_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(logits_row)[e])
                      : static_cast<const float*>(logits_row)[e];
      u = route_key(bias != nullptr ? v + bias[e] : v);
    }
    val[j] = v;
    key[j] = u;
  }

  float my_val = -FLT_MAX;   // lane r keeps the logit chosen in round r
  uint32_t my_idx = 0;
  #pragma unroll 1
  for (int r = 0; r < k; ++r) {
    uint32_t best = 0;
    #pragma unroll
    for (int j = 0; j < PER_LANE; ++j) best = max(best, key[j]);
    const uint32_t top = __reduce_max_sync(0xffffffffu, best);
    // the lowest expert index that holds the maximum: in this lane the lowest j, then over the warp
    uint32_t cand = 0xffffffffu;
    #pragma unroll
    for (int j = PER_LANE - 1; j >= 0; --j) {
      if (key[j] == top) cand = static_cast<uint32_t>(j * 32 + lane);
    }
    const uint32_t w_e = __reduce_min_sync(0xffffffffu, cand);
    // the owner retires the winner and hands its plain logit to lane r
    float chosen = 0.f;
    if ((w_e & 31u) == static_cast<uint32_t>(lane)) {
      #pragma unroll
      for (int j = 0; j < PER_LANE; ++j) {
        if (j == static_cast<int>(w_e >> 5)) {
          chosen = val[j];
          key[j] = 0u;
        }
      }
    }
    chosen = __shfl_sync(0xffffffffu, chosen, w_e & 31u);
    if (lane == r) {
      my_val = chosen;
      my_idx = w_e;
    }
  }

  *weight = softmax_of_chosen(my_val, k, lane, 32);
  *idx = lane < k ? my_idx : 0u;
}

}  // namespace pplx::ops
