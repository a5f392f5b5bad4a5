// Dispatch and combine of a group of one rank, and the reduction of rows that another kernel wrote.
//
// With one rank nothing has to be announced, received or waited for: the general kernels
// (a2a_kernels.cu) would write every token as a record into this rank's own receive region and read
// it back, and copy every expert row into the combine region before reducing it. Here dispatch goes
// from the caller's tokens straight to the expert rows and combine from the expert rows straight to
// the tokens, which is what both cannot do without.
//
//   dispatch  every block counts the routes of all tokens in shared memory (so no block waits for
//             another), scans the padded totals, gives the routes of its own tokens their rows and
//             copies or quantises the tokens into them;
//   combine   every warp reduces a piece of a token, up to eight rows in flight per lane.
//
// Both are bound by HBM at prefill sizes and by the chain index -> row -> bytes at decode sizes.
// 4096 tokens, hidden 7168 bf16, top-8 of 256 experts: dispatch 136 -> 90 us, combine 292 -> 89 us
// (529 MB each, 81 us at the measured copy rate).
//
// The tables that the general combine and the expert GEMM's scatter mode read (row_src, row_tk,
// expert_meta, rec_*) are filled too, so that any combine may follow. The epoch words are left alone:
// the general kernels' tags and parities count only their own launches.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "a2a_device.cuh"
#include "a2a_ll.cuh"
#include "a2a_kernels.h"

namespace pplx {
namespace {

constexpr int kSingleThreads = 1024;
constexpr int kSingleWarps = kSingleThreads / 32;
constexpr int kCombineThreads = 768;   // 80 registers: eight 16-byte loads in flight and their addresses
constexpr int kCombineWarps = kCombineThreads / 32;
constexpr int kBatchTokens = 64;   // tokens whose rows a block keeps in shared memory at a time

struct SingleDispatch {
  A2AConfig cfg;
  A2ALocal ws;
  DispatchSendArgs send;
  DispatchRecvArgs recv;
  int32_t parts;   // blocks that share a token (> 1 only when there are fewer tokens than blocks)
};

__device__ __forceinline__ int bounded_tokens(const A2AConfig& cfg, int num_tokens, const int32_t* bound_m) {
  int T = num_tokens;
  if (bound_m != nullptr) T = min(T, *bound_m);
  return max(0, min(T, cfg.max_num_tokens));
}

// One piece of a token on its way to its rows: V 16-byte vectors of the row per lane.
template <int V, bool kQuant>
struct Piece {
  Vec16 v[V];
  float scale[kQuant ? V : 1];
};

template <int V, bool kQuant>
__device__ __forceinline__ void load_piece(Piece<V, kQuant>& p, const uint8_t* src, uint32_t first, uint32_t nvec, bool pow2) {
  const uint32_t lane = threadIdx.x & 31u;
  if constexpr (kQuant) {
    Vec16 lo[V], hi[V];
    #pragma unroll
    for (int u = 0; u < V; ++u) {
      const uint32_t i = first + 32 * u + lane;
      lo[u] = hi[u] = Vec16{0, 0, 0, 0};
      if (i < nvec) {
        lo[u] = ld_input_v4(src + 32ull * i);
        hi[u] = ld_input_v4(src + 32ull * i + 16);
      }
    }
    #pragma unroll
    for (int u = 0; u < V; ++u) p.v[u] = quantize16(lo[u], hi[u], &p.scale[u], pow2);
  } else {
    #pragma unroll
    for (int u = 0; u < V; ++u) {
      const uint32_t i = first + 32 * u + lane;
      if (i < nvec) p.v[u] = ld_input_v4(src + 16ull * i);
    }
  }
}

template <int V, bool kQuant>
__global__ void __launch_bounds__(kSingleThreads, 1) dispatch_single_kernel(const __grid_constant__ SingleDispatch d) {
  extern __shared__ uint32_t dyn_smem[];
  __shared__ uint32_t s_rows[kBatchTokens * kMaxTopK];
  __shared__ uint32_t s_warp_sum[kSingleWarps];
  __shared__ uint32_t s_padded;
  const A2AConfig& cfg = d.cfg;
  const A2ALocal& ws = d.ws;
  const DispatchSendArgs& a = d.send;
  const DispatchRecvArgs& r = d.recv;
  const uint32_t E = cfg.num_experts;
  const uint32_t K = cfg.topk;
  uint32_t* total = dyn_smem;      // [E] routes of tokens from t0 on, then of all tokens
  uint32_t* next = dyn_smem + E;   // [E] routes of tokens before t0, then the next free row
  const int warp = threadIdx.x >> 5;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t nvec = cfg.d_payload_bytes / 16;
  const uint32_t chunks = (nvec + 32 * V - 1) / (32 * V);
  const int T = bounded_tokens(cfg, a.num_tokens, a.bound_m);

  // this block's tokens [t0, t1) and, of each, the pieces [c0, c1)
  const uint32_t parts = d.parts;
  uint32_t t0, t1, part = 0;
  if (parts > 1) {
    t0 = min(blockIdx.x / parts, static_cast<uint32_t>(T));
    t1 = min(t0 + 1, static_cast<uint32_t>(T));
    part = blockIdx.x % parts;
  } else {
    t0 = static_cast<uint32_t>(static_cast<uint64_t>(T) * blockIdx.x / gridDim.x);
    t1 = static_cast<uint32_t>(static_cast<uint64_t>(T) * (blockIdx.x + 1) / gridDim.x);
  }
  const uint32_t c0 = chunks * part / parts, c1 = chunks * (part + 1) / parts;
  const uint32_t nc = c1 - c0;
  const bool pow2 = a.quantize == 2;

  // The bytes of the first piece do not depend on where it goes.
  Piece<V, kQuant> piece;
  auto load = [&](uint32_t token, uint32_t chunk) {
    load_piece<V, kQuant>(piece, a.x + static_cast<uint64_t>(token) * a.x_stride, chunk * 32 * V, nvec, pow2);
  };
  uint32_t unit = warp;
  if (unit < (t1 - t0) * nc) load(t0 + unit / nc, c0 + unit % nc);

  if (ws.status[0] != 0) {   // an earlier failure, for all blocks alike: the word is never cleared
    if (blockIdx.x == 0 && threadIdx.x == 0) ws.single_done[0] += 1;
    return;
  }
  for (uint32_t i = threadIdx.x; i < 2 * E; i += kSingleThreads) dyn_smem[i] = 0;
  __syncthreads();
  // ---- routes per expert, those of earlier blocks' tokens apart ----
  auto count = [&](uint32_t e, bool earlier, uint32_t t) {
    if (e < E) atomicAdd(earlier ? &next[e] : &total[e], 1u);
    else if (blockIdx.x == 0) report(ws, kStatusBadExpertIndex, kPhaseDispatchSend, t, e);
  };
  const uint32_t routes = static_cast<uint32_t>(T) * K;
  if (a.indices_stride == K && (reinterpret_cast<uintptr_t>(a.indices) & 15u) == 0) {
    const uint32_t quads = routes / 4, limit = t0 * K;
    #pragma unroll 4
    for (uint32_t q = threadIdx.x; q < quads; q += kSingleThreads) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(a.indices) + q);
      const uint32_t e[4] = {v.x, v.y, v.z, v.w};
      #pragma unroll
      for (int c = 0; c < 4; ++c) count(e[c], 4 * q + c < limit, (4 * q + c) / K);
    }
    const uint32_t i = quads * 4 + threadIdx.x;
    if (i < routes) count(a.indices[i], i < limit, i / K);
  } else {
    for (uint32_t i = threadIdx.x; i < routes; i += kSingleThreads) {
      const uint32_t t = i / K;
      count(a.indices[t * a.indices_stride + i % K], t < t0, t);
    }
  }
  __syncthreads();
  // ---- expert-major layout: exclusive scan of the padded totals, kSingleThreads experts at a time ----
  const uint32_t pad = cfg.expert_padding;
  const uint32_t row_cap = r.out_rows ? min(r.out_rows, cfg.max_recv_rows) : cfg.max_recv_rows;
  uint32_t carry = 0;
  for (uint32_t e0 = 0; e0 < E; e0 += kSingleThreads) {
    const uint32_t e = e0 + threadIdx.x;
    const uint32_t n = e < E ? total[e] + next[e] : 0u;
    const uint32_t padded = pad == 1 ? n : (n + pad - 1) / pad * pad;
    uint32_t incl = padded;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= static_cast<uint32_t>(o)) incl += up;
    }
    if (lane == 31) s_warp_sum[warp] = incl;
    __syncthreads();
    uint32_t before = static_cast<int>(lane) < warp ? s_warp_sum[lane] : 0u, all = s_warp_sum[lane];
    before = __reduce_add_sync(0xffffffffu, before);
    all = __reduce_add_sync(0xffffffffu, all);
    const uint32_t off = carry + before + incl - padded;
    carry += all;
    if (e < E) {
      next[e] += off;
      if (blockIdx.x == 0) {
        r.out_num_tokens[e] = static_cast<int32_t>(n);
        ws.expert_meta[2 + e] = n;
        ws.expert_meta[2 + E + e] = off;
        // rows that only exist as padding carry no source
        for (uint32_t row = off + n; row < off + padded && row < cfg.max_recv_rows; ++row) ws.row_src[row] = kNoSlot;
      }
    }
    __syncthreads();   // s_warp_sum is written again
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ws.expert_meta[0] = min(carry, row_cap);
    ws.expert_meta[1] = T;
    if (carry > row_cap) report(ws, kStatusRowOverflow, kPhaseDispatchRecv, carry, row_cap);
    ws.single_done[0] += 1;
    ws.stats[0] += T;
  }
  // ---- rows of this block's routes, then the bytes ----
  const bool pre = cfg.combine_mode == kCombinePreReduce;
  const int hs = cfg.hidden_dim_scale;
  const float* xs = reinterpret_cast<const float*>(a.x_scale);
  float* os = reinterpret_cast<float*>(r.out_x_scale);
  for (uint32_t b0 = t0; b0 < t1; b0 += kBatchTokens) {
    const uint32_t b1 = min(b0 + kBatchTokens, t1);
    for (uint32_t i = threadIdx.x; i < (b1 - b0) * K; i += kSingleThreads) {
      const uint32_t t = b0 + i / K, k = i % K;
      const uint32_t e = a.indices[t * a.indices_stride + k];
      uint32_t row = kNoSlot;
      if (e < E) {
        if (parts > 1) {   // the blocks of a token must come to the same answer: no atomics
          row = next[e];
          for (uint32_t q = 0; q < k; ++q) row += a.indices[t * a.indices_stride + q] == e ? 1u : 0u;
        } else {
          row = atomicAdd(&next[e], 1u);
        }
        if (row >= row_cap) row = kNoSlot;
      }
      s_rows[i] = row;
      if (part == 0) {
        const uint64_t tk = static_cast<uint64_t>(t) * K + k;
        ws.route_row[tk] = row;
        if (row != kNoSlot) {
          ws.row_src[row] = 0;
          ws.row_tk[row] = static_cast<uint32_t>(tk);
        }
        if (pre) {
          ws.rec_rows[tk] = row;
          ws.rec_weights[tk] = a.weights[t * a.weights_stride + k];
          if (k == 0) {
            ws.rec_token[2 * t] = t;
            ws.rec_token[2 * t + 1] = 0;
          }
        }
      }
    }
    __syncthreads();
    for (; unit < (b1 - t0) * nc; unit += kSingleWarps) {
      const uint32_t t = t0 + unit / nc, chunk = c0 + unit % nc;
      if (unit != static_cast<uint32_t>(warp)) load(t, chunk);
      const uint32_t* rows = s_rows + (t - b0) * K;
      for (uint32_t k = 0; k < K; ++k) {
        const uint32_t row = rows[k];
        if (row == kNoSlot) continue;   // uniform across the warp
        uint8_t* dst = r.out_x + static_cast<uint64_t>(row) * r.out_x_stride;
        #pragma unroll
        for (int u = 0; u < V; ++u) {
          const uint32_t i = chunk * 32 * V + 32 * u + lane;
          if (i < nvec) {
            st_stream_v4(dst + 16ull * i, piece.v[u]);
            if constexpr (kQuant) {
              if ((i & 7u) == 0) {
                os[static_cast<int64_t>(row) * r.out_x_scale_stride_token +
                   static_cast<int64_t>(i >> 3) * r.out_x_scale_stride_elem] = piece.scale[u];
              }
            }
          }
        }
      }
      if constexpr (!kQuant) {
        if (hs > 0 && os != nullptr && chunk == c0 && part == 0) {
          for (int j = lane; j < hs; j += 32) {
            const float s = xs[t * a.x_scale_stride_token + j * a.x_scale_stride_elem];
            for (uint32_t k = 0; k < K; ++k) {
              if (rows[k] == kNoSlot) continue;
              os[static_cast<int64_t>(rows[k]) * r.out_x_scale_stride_token +
                 static_cast<int64_t>(j) * r.out_x_scale_stride_elem] = s;
            }
          }
        }
      }
    }
    if (b1 < t1) __syncthreads();   // the next batch rewrites the rows
  }
}

// ---------------------------------------------------------------------------
// combine
// ---------------------------------------------------------------------------

struct SingleCombine {
  A2AConfig cfg;
  A2ALocal ws;
  CombineRecvArgs recv;
  const uint8_t* rows;        // expert_y, or the combine receive region (external)
  uint64_t row_stride;
  const uint32_t* arrived;    // external: the counter the sending kernel raises
  int32_t granules_per_unit;  // 8-element granules of a token that a warp reduces at a time, / 32
};

template <typename Y, typename O>
__global__ void __launch_bounds__(kCombineThreads, 1) combine_single_kernel(const __grid_constant__ SingleCombine c) {
  const A2AConfig& cfg = c.cfg;
  const A2ALocal& ws = c.ws;
  const CombineRecvArgs& a = c.recv;
  const bool external = a.external != 0;
  const uint32_t K = cfg.topk;
  const uint32_t lane = threadIdx.x & 31u;
  const int T = bounded_tokens(cfg, a.num_tokens, a.bound_m);
  const uint32_t epoch = external ? read_epoch(ws, 1) : 0u;
  bool go = ws.status[0] == 0;
  if (external) {
    __shared__ uint32_t s_arrived;
    if (threadIdx.x == 0) {
      const uint32_t expected = read_epoch(ws, 2) + 1;
      uint64_t waited;
      s_arrived = wait_flag(c.arrived, expected, cfg.wait_limit_ns, &waited) ? 1u : 0u;
      if (!s_arrived) report(ws, kStatusWaitTimeout, kPhaseCombineRecv, 0, expected);
      if (blockIdx.x == 0) atomicMax(&ws.stats[3], static_cast<unsigned long long>(waited));
    }
    __syncthreads();
    go = go && s_arrived != 0;
  } else if (static_cast<uint32_t>(T) > ws.expert_meta[1]) {
    // rows of tokens that were not dispatched never come
    if (threadIdx.x == 0 && go) report(ws, kStatusWaitTimeout, kPhaseCombineRecv, ws.expert_meta[1], T);
    go = false;
  }
  if (go) {
    const uint32_t ngran = cfg.hidden_dim / 8;
    const uint32_t per_unit = 32 * c.granules_per_unit;
    const uint32_t pieces = (ngran + per_unit - 1) / per_unit;
    const bool given_weights = external || cfg.combine_mode == kCombinePerRoute;
    constexpr int kVecs = Elem8<Y>::kBytes / 16;
    constexpr int U = 8 / kVecs;   // rows in flight per lane
    const uint32_t warps = gridDim.x * kCombineWarps;
    for (uint32_t unit = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; unit < T * pieces; unit += warps) {
      const uint32_t t = unit / pieces, g0 = unit % pieces * per_unit;
      // lane k: where the token's k-th row is, and its weight
      uint32_t my_row = kNoSlot;
      float my_w = 0.f;
      if (lane < K) {
        if (external) {
          if (a.indices[t * a.indices_stride + lane] < static_cast<uint32_t>(cfg.num_experts)) my_row = t * K + lane;
        } else {
          my_row = ws.route_row[static_cast<uint64_t>(t) * K + lane];
        }
        my_w = given_weights ? a.weights[t * a.weights_stride + lane] : ws.rec_weights[static_cast<uint64_t>(t) * K + lane];
      }
      uint8_t* out_row = a.out_tokens + static_cast<uint64_t>(t) * a.out_tokens_stride * sizeof(O);
      for (uint32_t g = g0 + lane; g < min(g0 + per_unit, (ngran + 31) & ~31u); g += 32) {
        const bool inside = g < ngran;
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (a.accumulate && inside) Elem8<O>::load(out_row + static_cast<uint64_t>(g) * Elem8<O>::kBytes, acc, true);
        for (uint32_t k0 = 0; k0 < K; k0 += U) {
          // raw bytes in flight, converted as they are added: as floats they would not fit the registers
          Vec16 v[U][kVecs];
          float w[U];
          #pragma unroll
          for (int u = 0; u < U; ++u) {
            const uint32_t row = __shfl_sync(0xffffffffu, my_row, k0 + u);
            w[u] = __shfl_sync(0xffffffffu, my_w, k0 + u);
            const bool have = inside && k0 + u < K && row != kNoSlot;
            w[u] = have ? w[u] : 0.f;
            const uint8_t* p = c.rows + static_cast<uint64_t>(row) * c.row_stride + static_cast<uint64_t>(g) * Elem8<Y>::kBytes;
            #pragma unroll
            for (int i = 0; i < kVecs; ++i) v[u][i] = have ? ld_stream_v4(p + 16 * i) : Vec16{0, 0, 0, 0};
          }
          #pragma unroll
          for (int u = 0; u < U; ++u) {
            #pragma unroll
            for (int i = 0; i < kVecs; ++i) {
              float f[8];
              VecElems<Y>::unpack(v[u][i], f);
              #pragma unroll
              for (int q = 0; q < 8 / kVecs; ++q) acc[i * (8 / kVecs) + q] = fmaf(w[u], f[q], acc[i * (8 / kVecs) + q]);
            }
          }
        }
        if (inside) Elem8<O>::store(out_row + static_cast<uint64_t>(g) * Elem8<O>::kBytes, acc);
      }
    }
  }
  if (external) {
    finish_recv(cfg, ws, 1, epoch, kTraceCRecvAllDone, true);
  } else if (blockIdx.x == 0 && threadIdx.x == 0) {
    ws.single_done[1] += 1;
  }
}

template <typename F>
cudaError_t with_types(int y, int o, F&& f) {
  auto inner = [&](auto* yp) {
    switch (o) {
      case kDtypeBF16: return f(yp, static_cast<__nv_bfloat16*>(nullptr));
      case kDtypeF16: return f(yp, static_cast<__half*>(nullptr));
      case kDtypeF32: return f(yp, static_cast<float*>(nullptr));
      default: return cudaErrorInvalidValue;
    }
  };
  switch (y) {
    case kDtypeBF16: return inner(static_cast<__nv_bfloat16*>(nullptr));
    case kDtypeF16: return inner(static_cast<__half*>(nullptr));
    case kDtypeF32: return inner(static_cast<float*>(nullptr));
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t a2a_launch_dispatch_single(const A2AConfig& cfg, const A2ALocal& ws, const DispatchSendArgs& send,
                                       const DispatchRecvArgs& recv, cudaStream_t stream) {
  SingleDispatch d{cfg, ws, send, recv, 1};
  const int blocks = cfg.num_blocks;
  const int64_t nvec = cfg.d_payload_bytes / 16;
  // Four vectors a lane where every warp gets two such pieces at least, else one, and where there
  // are fewer tokens than half the blocks several blocks share a token.
  const bool wide = static_cast<int64_t>(send.num_tokens) * ((nvec + 127) / 128) >= 2ll * blocks * kSingleWarps;
  if (!wide && send.num_tokens > 0) {
    d.parts = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(blocks / send.num_tokens, (nvec + 31) / 32)));
  }
  const size_t smem = 2 * sizeof(uint32_t) * cfg.num_experts;
  void* args[] = {&d};
  const void* kernel = send.quantize != 0
                           ? (wide ? reinterpret_cast<const void*>(dispatch_single_kernel<4, true>)
                                   : reinterpret_cast<const void*>(dispatch_single_kernel<1, true>))
                           : (wide ? reinterpret_cast<const void*>(dispatch_single_kernel<4, false>)
                                   : reinterpret_cast<const void*>(dispatch_single_kernel<1, false>));
  return cudaLaunchKernel(kernel, dim3(blocks), dim3(kSingleThreads), args, smem, stream);
}

cudaError_t a2a_launch_combine_single(const A2AConfig& cfg, const A2ALocal& ws, const CombineRecvArgs& recv,
                                      const uint8_t* rows, uint64_t row_stride, const uint32_t* arrived, int y_dtype,
                                      int out_dtype, cudaStream_t stream) {
  SingleCombine c{cfg, ws, recv, rows, row_stride, arrived, 1};
  // two granules a lane and unit where there are eight such units per warp, so that the last round
  // of units is a small part of the whole
  const int64_t granules = cfg.hidden_dim / 8;
  if (recv.num_tokens * ((granules + 63) / 64) >= 8ll * cfg.num_blocks * kCombineWarps) c.granules_per_unit = 2;
  return with_types(y_dtype, out_dtype, [&](auto* yp, auto* op) {
    using Y = std::remove_pointer_t<decltype(yp)>;
    using O = std::remove_pointer_t<decltype(op)>;
    void* args[] = {&c};
    return cudaLaunchKernel(reinterpret_cast<const void*>(combine_single_kernel<Y, O>), dim3(cfg.num_blocks),
                            dim3(kCombineThreads), args, 0, stream);
  });
}

cudaError_t a2a_preload_single() {
  cudaFuncAttributes attr;
  cudaError_t e = cudaFuncGetAttributes(&attr, dispatch_single_kernel<4, true>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, dispatch_single_kernel<1, true>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, dispatch_single_kernel<4, false>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, dispatch_single_kernel<1, false>);
  for (int y : {kDtypeBF16, kDtypeF16, kDtypeF32}) {
    for (int o : {kDtypeBF16, kDtypeF16, kDtypeF32}) {
      if (e != cudaSuccess) return e;
      e = with_types(y, o, [&](auto* yp, auto* op) {
        return cudaFuncGetAttributes(&attr, combine_single_kernel<std::remove_pointer_t<decltype(yp)>,
                                                                  std::remove_pointer_t<decltype(op)>>);
      });
    }
  }
  return e;
}

}  // namespace pplx
