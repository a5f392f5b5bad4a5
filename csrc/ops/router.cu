// Stand-alone top-k routing, one warp per token.
//
// A round of arg-max per chosen expert (router.cuh) costs two warp reductions and a pass over every
// lane's registers, and the issue slots are what a large batch waits for: 32,768 tokens of 256 experts
// with k = 8 took 36 us for 17 MB of bf16 logits, and take 21 us (507 warp instructions a token) here,
// nearly whatever k is:
//   1. every lane takes the maximum of its own keys;
//   2. a bound t that at least k of these maxima reach, and only a few more, is found by bisection
//      (a comparison, a ballot and a count a step); the k-th largest key is no smaller;
//   3. the keys >= t, usually k and a few more, are compacted into shared memory, one per lane;
//   4. a candidate's rank among them is its place in the result.
// Ties break to the lower expert index, which is part of the comparison. With more than 32 candidates (many
// logits tied with the bound, or a large k) a token takes the rounds of router.cuh; where that is the
// rule, and where k is 1 or 2, a kernel that does nothing else runs instead (rounds_win() below).
// Ranking the maxima against one another instead of the bisection, and carrying the logits along
// instead of reading the k chosen ones again, took 26.6 us.
#include "router.h"

#include <cuda_bf16.h>

#include <algorithm>
#include <cfloat>
#include <cmath>

#include "../a2a/ptx.cuh"
#include "../core/error.h"
#include "../core/launch.h"
#include "router.cuh"

namespace pplx::ops {
namespace {

constexpr int kMaxWarps = 8;
// resident blocks of kMaxWarps warps: what the registers allow
template <int PER_LANE> constexpr int kBlocksPerSm = PER_LANE <= 4 ? 8 : PER_LANE <= 8 ? 5 : 2;

struct alignas(16) WarpScratch {
  uint64_t cand[32];   // key in the high word, ~expert in the low one: larger is better, 0 is none
  uint32_t chosen[32];
};

// Stores `value` where key >= bound. One predicated instruction: as an `if` around the store the
// unrolled loop that calls this became a loop over arrays in local memory.
__device__ __forceinline__ void store_candidate(uint32_t key, uint32_t bound, uint64_t* at, uint32_t not_expert) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ge.u32 p, %0, %1;\n"
      "@p st.shared.v2.u32 [%2], {%3, %0};\n"
      "}\n"
      :
      : "r"(key), "r"(bound), "r"(static_cast<uint32_t>(__cvta_generic_to_shared(at))), "r"(not_expert)
      : "memory");
}

// N (1, 2 or 4) consecutive words, by a coherent load that stays behind grid_wait().
template <int N>
__device__ __forceinline__ void load_words(const void* p, uint32_t* w) {
  if constexpr (N == 4) {
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "l"(p) : "memory");
  } else if constexpr (N == 2) {
    asm volatile("ld.global.v2.u32 {%0,%1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "l"(p) : "memory");
  } else {
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(w[0]) : "l"(p) : "memory");
  }
}

// PER_LANE consecutive elements of a row as floats.
template <int PER_LANE, typename T>
__device__ __forceinline__ void load_run(const T* p, float (&v)[PER_LANE]) {
  constexpr int kWords = PER_LANE * static_cast<int>(sizeof(T)) / 4;
  constexpr int kVec = kWords < 4 ? kWords : 4;
  uint32_t w[kWords];
  #pragma unroll
  for (int j = 0; j < kWords; j += kVec) load_words<kVec>(reinterpret_cast<const uint32_t*>(p) + j, w + j);
  #pragma unroll
  for (int j = 0; j < kWords; ++j) {
    if constexpr (sizeof(T) == 4) {
      v[j] = __uint_as_float(w[j]);
    } else {
      v[2 * j] = __uint_as_float(w[j] << 16);
      v[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
    }
  }
}

template <int PER_LANE>
__device__ __forceinline__ void rounds_of_token(const TopkRouteParams& p, int token, int lane) {
  const void* row = static_cast<const char*>(p.logits) + static_cast<int64_t>(token) * p.logits_stride * (p.logits_bf16 ? 2 : 4);
  uint32_t idx;
  float weight;
  route_token_warp<PER_LANE>(row, p.logits_bf16, p.bias, p.num_experts, p.k, &idx, &weight);
  if (lane < p.k) {
    p.indices[token * p.indices_stride + lane] = idx;
    p.weights[token * p.weights_stride + lane] = weight;
  }
}

// As a call: the ranking kernel needs its registers for other things.
template <int PER_LANE>
__device__ __noinline__ void route_by_rounds(const TopkRouteParams& p, int token, int lane) {
  rounds_of_token<PER_LANE>(p, token, lane);
}

__device__ __forceinline__ float to_float(float x) { return x; }
__device__ __forceinline__ float to_float(__nv_bfloat16 x) { return __bfloat162float(x); }

// kVec: rows are 16-byte aligned and num_experts is a multiple of PER_LANE; a lane's experts are
// consecutive and come in as vectors. Otherwise expert = j * 32 + lane, one element a load.
template <int PER_LANE, typename T, bool kVec>
__global__ void __launch_bounds__(kMaxWarps * 32, kBlocksPerSm<PER_LANE>) topk_route_kernel(const __grid_constant__ TopkRouteParams p) {
  __shared__ WarpScratch scratch[kMaxWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5;
  WarpScratch& ws = scratch[warp];
  const int E = p.num_experts, k = p.k;
  const uint32_t below = (1u << lane) - 1u;
  const bool mine = !kVec || lane * PER_LANE < E;   // a lane's run is all inside or all outside
  grid_wait();
  grid_allow_next();
  float bias[PER_LANE];
  #pragma unroll
  for (int j = 0; j < PER_LANE; ++j) {
    const int e = kVec ? lane * PER_LANE + j : j * 32 + lane;
    // never -0: the sum below is then never -0 either, which would not compare equal to +0 as a key
    bias[j] = p.bias != nullptr && e < E ? p.bias[e] + 0.f : 0.f;
  }
  const int tokens = p.bound != nullptr ? min(p.tokens, *p.bound) : p.tokens;
  int span = 1;   // lanes of the softmax
  while (span < k) span <<= 1;
  for (int token = blockIdx.x * warps + warp; token < tokens; token += gridDim.x * warps) {
    const T* row = static_cast<const T*>(p.logits) + static_cast<int64_t>(token) * p.logits_stride;
    uint32_t key[PER_LANE];
    #pragma unroll
    for (int j = 0; j < PER_LANE; ++j) key[j] = 0;
    if constexpr (kVec) {
      if (mine) {
        float val[PER_LANE];
        load_run<PER_LANE>(row + lane * PER_LANE, val);
        #pragma unroll
        for (int j = 0; j < PER_LANE; ++j) key[j] = route_key_of_sum(val[j] + bias[j]);
      }
    } else {
      #pragma unroll
      for (int j = 0; j < PER_LANE; ++j) {
        if (j * 32 + lane < E) key[j] = route_key_of_sum(to_float(row[j * 32 + lane]) + bias[j]);
      }
    }
    uint32_t best = 0;
    #pragma unroll
    for (int j = 0; j < PER_LANE; ++j) best = max(best, key[j]);
    // At least k lanes have best >= lo, fewer than k have best >= hi. Lanes whose run of experts lies past
    // the last one hold no key and are left out: with them in, the minimum is 0 and everything is a
    // candidate (160 experts fill 20 lanes of 8: 32,768 tokens took 37 us, and 29 by rounds alone).
    uint32_t lo = __reduce_min_sync(0xffffffffu, best - 1u) + 1u;   // no key, 0, is the largest here
    uint32_t hi = __reduce_max_sync(0xffffffffu, best);
    if (E > 32) {
      int have = kVec ? E / PER_LANE : 32;   // lanes with a key: k at least, see launch()
      for (int step = 0; step < 12 && have > k + 2 && hi - lo > 1; ++step) {
        const uint32_t mid = lo + (hi - lo) / 2;
        const int n = __popc(__ballot_sync(0xffffffffu, best >= mid));
        if (n >= k) {
          lo = mid;
          have = n;
        } else {
          hi = mid;
        }
      }
    } else {
      lo = 0;   // all of them are candidates
    }
    const uint32_t bound = max(lo, 1u);
    // the candidates' places in the scratch: any order will do
    uint32_t lanes[PER_LANE];
    int total = 0;
    #pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
      lanes[j] = __ballot_sync(0xffffffffu, key[j] >= bound);
      total += __popc(lanes[j]);
    }
    if (total <= 32) {
      // Empty places compare as none. No other lane stores to these: nothing between here and the
      // barrier orders one lane's stores after another's.
      if (lane >= total) ws.cand[lane] = 0;
      int before = 0;
      #pragma unroll
      for (int j = 0; j < PER_LANE; ++j) {
        store_candidate(key[j], bound, &ws.cand[before + __popc(lanes[j] & below)],
                        ~static_cast<uint32_t>(kVec ? lane * PER_LANE + j : j * 32 + lane));
        before += __popc(lanes[j]);
      }
      __syncwarp();
      const uint64_t me = ws.cand[lane];
      int place = 0;
      #pragma unroll 1
      for (int i = 0; i < total; i += 4) {   // what is past the last candidate is 0
        const ulonglong2 c01 = *reinterpret_cast<const ulonglong2*>(&ws.cand[i]);
        const ulonglong2 c23 = *reinterpret_cast<const ulonglong2*>(&ws.cand[i + 2]);
        place += c01.x > me ? 1 : 0;
        place += c01.y > me ? 1 : 0;
        place += c23.x > me ? 1 : 0;
        place += c23.y > me ? 1 : 0;
      }
      if (lane < total && place < k) ws.chosen[place] = ~static_cast<uint32_t>(me);
      __syncwarp();
      uint32_t out_idx = 0;
      float out_val = -FLT_MAX;
      if (lane < k) {
        out_idx = ws.chosen[lane];
        out_val = to_float(row[out_idx]);
      }
      const float weight = softmax_of_chosen(out_val, k, lane, span);
      if (lane < k) {
        p.indices[token * p.indices_stride + lane] = out_idx;
        p.weights[token * p.weights_stride + lane] = weight;
      }
    } else {
      route_by_rounds<PER_LANE>(p, token, lane);
    }
    __syncwarp();   // the scratch is rewritten by the next token
  }
}

template <int PER_LANE>
__global__ void __launch_bounds__(kMaxWarps * 32) topk_rounds_kernel(const __grid_constant__ TopkRouteParams p) {
  grid_wait();
  grid_allow_next();
  const int tokens = p.bound != nullptr ? min(p.tokens, *p.bound) : p.tokens;
  const int token = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (token < tokens) rounds_of_token<PER_LANE>(p, token, threadIdx.x & 31);
}

// Whether the rounds alone beat the ranking. Its candidates have to fit 32 places: with L lanes that hold
// E / L keys each, a bound that k + 1 of their maxima reach lets through about
// E (1 - (1 - (k + 1) / L)^(L / E)) keys. From about 33 on a token does both more often than not; with more
// than 16 keys a lane, whose rounds are long, ranking pays up to 36. 32,768 tokens, rounds and ranking in us:
// 256 experts k = 20 73 and 66, k = 24 85 and 102; 320 experts k = 14 102 and 76, k = 16 114 and 130; 512
// experts k = 18 135 and 87, k = 20 146 and 157; 1000 experts k = 20 335 and 304, k = 24 379 and 428. With four
// keys a lane or fewer the ranking keeps up at any k (128 experts k = 32 84 and 75). One or two rounds are
// shorter than the ranking's set-up where a lane holds four or eight keys (256 experts k = 1 13.1 and 17.5).
template <int PER_LANE>
bool rounds_win(int experts, int k, bool vec) {
  if (k <= 2) return PER_LANE == 4 || PER_LANE == 8;
  if (PER_LANE < 8 || k < 8) return false;
  const double lanes = vec ? experts / PER_LANE : 32;
  const double left = std::max(0.0, 1.0 - (k + 1) / lanes);
  return experts * (1.0 - std::pow(left, lanes / experts)) > (PER_LANE > 16 ? 36.0 : 33.0);
}

template <int PER_LANE, typename T>
void launch(const TopkRouteParams& p, int sms, cudaStream_t stream) {
  constexpr uintptr_t kAlign = std::min<size_t>(16, PER_LANE * sizeof(T));
  // The bound needs k lanes with a key: a vector layout that fills fewer gives way to the one element a
  // load, which fills all 32 (with 32 experts or fewer every key is a candidate and no bound is needed).
  const bool vec = p.num_experts % PER_LANE == 0 && reinterpret_cast<uintptr_t>(p.logits) % kAlign == 0 &&
                   p.logits_stride * sizeof(T) % kAlign == 0 &&
                   (p.num_experts / PER_LANE >= p.k || p.num_experts <= 32);
  // Few tokens: one warp a block, so that they spread over the SMs. Many: one wave of resident blocks
  // whose warps loop, with the bias in registers.
  const int warps = p.tokens <= sms * 4 ? 1 : kMaxWarps;
  const int groups = (p.tokens + warps - 1) / warps;
  const bool rounds = rounds_win<PER_LANE>(p.num_experts, p.k, vec);
  const int blocks = rounds ? groups : std::min(groups, sms * (warps == 1 ? 4 : kBlocksPerSm<PER_LANE>));
  const void* kernel = rounds ? reinterpret_cast<const void*>(topk_rounds_kernel<PER_LANE>)
                       : vec  ? reinterpret_cast<const void*>(topk_route_kernel<PER_LANE, T, true>)
                              : reinterpret_cast<const void*>(topk_route_kernel<PER_LANE, T, false>);
  void* args[] = {const_cast<TopkRouteParams*>(&p)};
  PPLX_CUDA_CHECK(launch_overlapped(kernel, dim3(blocks), dim3(warps * 32), args, 0, stream));
}

template <typename T>
void launch_typed(const TopkRouteParams& p, int sms, cudaStream_t stream) {
  const int per_lane = (p.num_experts + 31) / 32;
  static_assert(sizeof(T) == 2 || sizeof(T) == 4, "bf16 or fp32 logits");
  if (per_lane <= 2) launch<2, T>(p, sms, stream);
  else if (per_lane <= 4) launch<4, T>(p, sms, stream);
  else if (per_lane <= 8) launch<8, T>(p, sms, stream);
  else if (per_lane <= 16) launch<16, T>(p, sms, stream);
  else launch<32, T>(p, sms, stream);
}

}  // namespace

void topk_route(const TopkRouteParams& p, cudaStream_t stream) {
  PPLX_REQUIRE(p.num_experts >= 1 && p.num_experts <= 1024, "between 1 and 1024 experts");
  PPLX_REQUIRE(p.k >= 1 && p.k <= 32 && p.k <= p.num_experts, "k must be in [1, min(32, num_experts)]");
  if (p.tokens == 0) return;
  int device = 0, sms = 0;
  PPLX_CUDA_CHECK(cudaGetDevice(&device));
  PPLX_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  if (p.logits_bf16) launch_typed<__nv_bfloat16>(p, sms, stream);
  else launch_typed<float>(p, sms, stream);
}

}  // namespace pplx::ops
