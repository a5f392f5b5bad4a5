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
// Both are bound by HBM at prefill sizes and by the chain index -> row -> bytes at decode sizes. Hidden 7168
// bf16, top-8 of 256 experts, a pass of both: 4096 tokens 429 us with the general kernels, 191 us here
// (529 MB each way, 81 us at the measured copy rate; one after another and with cold caches the dispatch
// takes 100 us, the combine 89); 128 tokens 31 and 13.2 us.
//
// The tables that the general combine and the expert GEMM's scatter mode read (row_src, row_tk,
// expert_meta, rec_*) are filled too, so that any combine may follow. The epoch words are left alone:
// the general kernels' tags and parities count only their own launches.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "../core/launch.h"
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
  int32_t bulk_scales;   // rows of scales are contiguous and 16-byte aligned: the bulk-copy engine writes them
  int32_t parts;   // blocks that share a token (> 1 only when there are fewer tokens than blocks)
};

__device__ __forceinline__ int bounded_tokens(const A2AConfig& cfg, int num_tokens, const int32_t* bound_m) {
  int T = num_tokens;
  if (bound_m != nullptr) T = min(T, *bound_m);
  return max(0, min(T, cfg.max_num_tokens));
}

// Two ways for a piece of a token to reach its rows.
//   kBulk false: one 16-byte vector a lane, stored to every row: the shortest way for few tokens.
//   kBulk true: pieces of 2 KiB in a warp's own pair of buffers in shared memory; the bulk-copy engine
//     brings the bytes in (or the warp quantises them into the buffer) and writes them to every row.
//     With vectors in registers, four a lane, the stores of 4096 quantised tokens of 7168 reached
//     3.6 TB/s and those of bf16 tokens 5.2 TB/s.
constexpr uint32_t kPieceBytes = 2048;
constexpr uint32_t kPieceScales = kPieceBytes / 128;                            // of a quantised piece
constexpr uint32_t kPieceBuffer = kPieceBytes + kPieceScales * sizeof(float);   // a multiple of 16

// 32 vectors of a row, one a lane, quantised from twice as many of bf16.
__device__ __forceinline__ Vec16 load_quantised(const uint8_t* src, uint32_t i, uint32_t nvec, bool pow2, float* scale) {
  Vec16 lo = {0, 0, 0, 0}, hi = {0, 0, 0, 0};
  if (i < nvec) {
    lo = ld_after_wait_v4(src + 32ull * i);
    hi = ld_after_wait_v4(src + 32ull * i + 16);
  }
  return quantize16(lo, hi, scale, pow2);
}

template <bool kBulk, bool kQuant>
__global__ void __launch_bounds__(kSingleThreads, 1) dispatch_single_kernel(const __grid_constant__ SingleDispatch d) {
  extern __shared__ __align__(128) uint8_t dyn_smem[];   // [pieces of every warp (kBulk) | counters]
  __shared__ uint32_t s_rows[kBatchTokens * kMaxTopK];
  __shared__ uint32_t s_warp_sum[kSingleWarps];
  __shared__ uint64_t s_bars[kSingleWarps][2];
  __shared__ uint32_t s_failed;
  const A2AConfig& cfg = d.cfg;
  const A2ALocal& ws = d.ws;
  const DispatchSendArgs& a = d.send;
  const DispatchRecvArgs& r = d.recv;
  const uint32_t E = cfg.num_experts;
  const uint32_t K = cfg.topk;
  uint32_t* total = reinterpret_cast<uint32_t*>(dyn_smem + (kBulk ? kSingleWarps * 2 * kPieceBuffer : 0));
  uint32_t* next = total + E;
  // total: [E] routes of tokens from t0 on; next: [E] routes of tokens before t0, then the next free row
  const int warp = threadIdx.x >> 5;
  const uint32_t lane = threadIdx.x & 31u;
  // shared memory only: this may run under the end of the kernel before
  for (uint32_t i = threadIdx.x; i < 2 * E; i += kSingleThreads) total[i] = 0;
  if constexpr (kBulk && !kQuant) {
    if (lane == 0) {
      mbar_init(&s_bars[warp][0], 1);
      mbar_init(&s_bars[warp][1], 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }
  __syncthreads();
  grid_wait();
  grid_allow_next();
  // One thread reads the status word for its block: block 0 of this very launch may write it (an expert
  // that does not exist, rows that do not fit), and a block that starts late must not be of two minds. The
  // block decides after the count, when the word has come in anyway (128 tokens of 14 KiB: waiting for it
  // before costs 0.2 us).
  uint32_t status = 0;
  if (threadIdx.x == 0) status = *reinterpret_cast<volatile const uint32_t*>(&ws.status[0]);
  const uint32_t nvec = cfg.d_payload_bytes / 16;
  constexpr uint32_t kPieceVecs = kBulk ? kPieceBytes / 16 : 32;
  const uint32_t chunks = (nvec + kPieceVecs - 1) / kPieceVecs;
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

  // The bytes of the first pieces do not depend on where they go.
  uint32_t unit = warp;
  const uint32_t units = (t1 - t0) * nc;
  Vec16 piece;
  float piece_scale = 0.f;
  uint8_t* const buffers = dyn_smem + warp * 2 * kPieceBuffer;
  auto source = [&](uint32_t u) { return a.x + static_cast<uint64_t>(t0 + u / nc) * a.x_stride; };
  auto fetch = [&](uint32_t u, uint32_t slot) {   // kBulk, not quantised: the engine fills a buffer
    if (u < units && lane == 0) {
      const uint32_t off = (c0 + u % nc) * kPieceBytes;
      const uint32_t bytes = min(kPieceBytes, cfg.d_payload_bytes - off);
      mbar_expect_tx(&s_bars[warp][slot], bytes);
      bulk_g2s(buffers + slot * kPieceBuffer, source(u) + off, bytes, &s_bars[warp][slot]);
    }
  };
  auto load = [&](uint32_t u) {   // not kBulk
    const uint32_t i = (c0 + u % nc) * 32 + lane;
    if constexpr (kQuant) piece = load_quantised(source(u), i, nvec, pow2, &piece_scale);
    else if (i < nvec) piece = ld_after_wait_v4(source(u) + 16ull * i);
  };
  const uint32_t routes = static_cast<uint32_t>(T) * K;
  const bool vector_indices = a.indices_stride == K && (reinterpret_cast<uintptr_t>(a.indices) & 15u) == 0;
  const uint32_t quads = vector_indices ? routes / 4 : 0u;
  constexpr uint32_t kQuads = 4;
  Vec16 quad[kQuads];
  auto load_quads = [&](uint32_t q0) {
    #pragma unroll
    for (uint32_t u = 0; u < kQuads; ++u) {
      const uint32_t q = q0 + u * kSingleThreads;
      if (q < quads) quad[u] = ld_after_wait_v4(a.indices + 4ull * q);
    }
  };
  load_quads(threadIdx.x);
  if constexpr (kBulk && !kQuant) {
    fetch(unit, 0);
  } else if constexpr (!kBulk) {
    if (unit < units) load(unit);
  }
  // ---- routes per expert, those of earlier blocks' tokens apart ----
  auto count = [&](uint32_t e, bool earlier, uint32_t t) {
    if (e < E) atomicAdd(earlier ? &next[e] : &total[e], 1u);
    else if (blockIdx.x == 0) report(ws, kStatusBadExpertIndex, kPhaseDispatchSend, t, e);
  };
  if (vector_indices) {
    const uint32_t limit = t0 * K;
    for (uint32_t q0 = threadIdx.x; q0 < quads; q0 += kQuads * kSingleThreads) {
      if (q0 != threadIdx.x) load_quads(q0);
      #pragma unroll
      for (uint32_t u = 0; u < kQuads; ++u) {
        const uint32_t q = q0 + u * kSingleThreads;
        if (q >= quads) break;
        const uint32_t e[4] = {quad[u].x, quad[u].y, quad[u].z, quad[u].w};
        #pragma unroll
        for (uint32_t c = 0; c < 4; ++c) count(e[c], 4 * q + c < limit, (4 * q + c) / K);
      }
    }
    const uint32_t i = quads * 4 + threadIdx.x;
    if (i < routes) count(a.indices[i], i < limit, i / K);
  } else {
    for (uint32_t i = threadIdx.x; i < routes; i += kSingleThreads) {
      const uint32_t t = i / K;
      count(a.indices[t * a.indices_stride + i % K], t < t0, t);
    }
  }
  if (threadIdx.x == 0) s_failed = status;
  __syncthreads();
  if (s_failed != 0) {
    if constexpr (kBulk && !kQuant) {   // no copy may still be on its way into a block that has left
      if (lane == 0 && unit < units) mbar_wait_timed(&s_bars[warp][0], 0, cfg.wait_limit_ns);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) ws.single_done[0] += 1;
    return;
  }
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
  uint32_t slot = 0, parities = 0;
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
    for (; unit < (b1 - t0) * nc; unit += kSingleWarps, slot ^= 1u) {
      const uint32_t t = t0 + unit / nc, chunk = c0 + unit % nc;
      const uint32_t* rows = s_rows + (t - b0) * K;
      if constexpr (kBulk) {
        const uint32_t off = chunk * kPieceBytes;
        const uint32_t bytes = min(kPieceBytes, cfg.d_payload_bytes - off);
        uint8_t* const buffer = buffers + slot * kPieceBuffer;
        float* const buffer_scales = reinterpret_cast<float*>(buffer + kPieceBytes);
        // the stores of this buffer's last piece, two pieces ago, have read it
        asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        __syncwarp();
        if constexpr (kQuant) {
          #pragma unroll
          for (int u = 0; u < 4; ++u) {
            float scale;
            const uint32_t j = 32 * u + lane;
            const Vec16 q = load_quantised(source(unit), off / 16 + j, nvec, pow2, &scale);
            *reinterpret_cast<Vec16*>(buffer + 16 * j) = q;
            if ((lane & 7u) == 0) buffer_scales[j >> 3] = scale;
          }
          fence_proxy_async_smem();
          __syncwarp();
        } else {
          // the other buffer is free once the stores of the piece before have read it
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          __syncwarp();
          fetch(unit + kSingleWarps, slot ^ 1u);
          if (!__all_sync(0xffffffffu, mbar_wait_timed(&s_bars[warp][slot], (parities >> slot) & 1u, cfg.wait_limit_ns))) {
            if (lane == 0) report(ws, kStatusWaitTimeout, kPhaseDispatchSend, t, bytes);
          }
          parities ^= 1u << slot;
        }
        if (lane < K && rows[lane] != kNoSlot) {
          bulk_s2g(r.out_x + static_cast<uint64_t>(rows[lane]) * r.out_x_stride + off, buffer, bytes);
          if (kQuant && d.bulk_scales) {
            bulk_s2g(os + static_cast<int64_t>(rows[lane]) * r.out_x_scale_stride_token + off / 128, buffer_scales,
                     bytes / 128 * sizeof(float));
          }
        }
        bulk_commit();
        if (kQuant && !d.bulk_scales && os != nullptr) {
          for (uint32_t i = lane; i < bytes / 128 * K; i += 32) {
            const uint32_t row = rows[i % K], j = i / K;
            if (row != kNoSlot) {
              os[static_cast<int64_t>(row) * r.out_x_scale_stride_token +
                 static_cast<int64_t>(off / 128 + j) * r.out_x_scale_stride_elem] = buffer_scales[j];
            }
          }
        }
      } else {
        if (unit != static_cast<uint32_t>(warp)) load(unit);
        const uint32_t i = chunk * 32 + lane;
        for (uint32_t k = 0; k < K; ++k) {
          const uint32_t row = rows[k];
          if (row == kNoSlot || i >= nvec) continue;
          st_stream_v4(r.out_x + static_cast<uint64_t>(row) * r.out_x_stride + 16ull * i, piece);
          if (kQuant && os != nullptr && (i & 7u) == 0) {
            os[static_cast<int64_t>(row) * r.out_x_scale_stride_token +
               static_cast<int64_t>(i >> 3) * r.out_x_scale_stride_elem] = piece_scale;
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
  if constexpr (kBulk) bulk_wait0();   // this lane's stores have been performed
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
  uint32_t segment;           // combine_bulk_kernel: bytes of each row that a warp reduces at a time
};

// Called by all threads of every block, before any row is read: the status word, or something else than 0
// where the rows of another kernel do not come. It may change while a warp's lanes look at it: they vote.
__device__ __forceinline__ uint32_t combine_status(const SingleCombine& c) {
  const A2ALocal& ws = c.ws;
  const uint32_t status = *reinterpret_cast<volatile const uint32_t*>(&ws.status[0]);
  if (!c.recv.external) return status;
  __shared__ uint32_t s_arrived;
  if (threadIdx.x == 0) {
    const uint32_t expected = read_epoch(ws, 2) + 1;
    uint64_t waited;
    s_arrived = wait_flag(c.arrived, expected, c.cfg.wait_limit_ns, &waited) ? 1u : 0u;
    if (!s_arrived) report(ws, kStatusWaitTimeout, kPhaseCombineRecv, 0, expected);
    if (blockIdx.x == 0) atomicMax(&ws.stats[3], static_cast<unsigned long long>(waited));
  }
  __syncthreads();
  return s_arrived != 0 ? status : ~0u;
}

__device__ __forceinline__ void combine_finish(const SingleCombine& c, uint32_t epoch) {
  if (c.recv.external) {
    finish_recv(c.cfg, c.ws, 1, epoch, kTraceCRecvAllDone, true);
  } else if (blockIdx.x == 0 && threadIdx.x == 0) {
    c.ws.single_done[1] += 1;
  }
}

// Lane k: where token t's k-th row is and its weight. The routes of the combine decide what is reduced, as
// in the general kernels: one with an expert that does not exist is left out (in the pre-reduced mode
// only a token that has no other), so that a caller may dispatch by bound_m and combine the padding too, or
// mask single routes. Loaded by one call and judged by another, so that nothing waits for the loads
// in between (judged at once, 4096 tokens of 8 rows of 14 KiB took 25 us more); all of them at once: as
// plain loads the compiler moves them behind the first comparison.
struct Route {
  uint32_t row = kNoSlot, expert = ~0u;
  float w = 0.f;
};
__device__ __forceinline__ Route load_route(const SingleCombine& c, uint32_t t, uint32_t lane) {
  const A2AConfig& cfg = c.cfg;
  const CombineRecvArgs& a = c.recv;
  const uint32_t K = cfg.topk;
  Route r;
  if (lane < K) {
    const uint64_t tk = static_cast<uint64_t>(t) * K + lane;
    const float* weight = a.external || cfg.combine_mode == kCombinePerRoute ? a.weights + t * a.weights_stride + lane
                                                                             : c.ws.rec_weights + tk;
    r.expert = ld_after_wait_u32(a.indices + t * a.indices_stride + lane);
    r.row = a.external ? static_cast<uint32_t>(tk) : ld_after_wait_u32(c.ws.route_row + tk);
    r.w = __uint_as_float(ld_after_wait_u32(weight));
  }
  return r;
}
// Tokens that were dispatched: the rows of a later one never come.
__device__ __forceinline__ uint32_t tokens_dispatched(const SingleCombine& c) {
  return c.recv.external ? ~0u : ld_after_wait_u32(&c.ws.expert_meta[1]);
}
__device__ __noinline__ uint32_t route_of_a_later_token(const A2ALocal& ws, bool valid, uint32_t t, uint32_t dispatched) {
  if (__any_sync(0xffffffffu, valid) && (threadIdx.x & 31u) == 0) report(ws, kStatusWaitTimeout, kPhaseCombineRecv, t, dispatched);
  return kNoSlot;   // the table holds an earlier dispatch's
}
// The row, or kNoSlot. All 32 lanes call.
__device__ __forceinline__ uint32_t route_place(const SingleCombine& c, const Route& r, uint32_t t, uint32_t dispatched) {
  bool valid = r.expert < static_cast<uint32_t>(c.cfg.num_experts);
  if (c.cfg.combine_mode != kCombinePerRoute) valid = __any_sync(0xffffffffu, valid);
  if (t >= dispatched) return route_of_a_later_token(c.ws, valid, t, dispatched);
  return valid ? r.row : kNoSlot;
}

// acc += w_k * row_k over the rows of `have` (bit k: row k is there), 16 bytes of each, at `p` and every
// `stride` bytes from there. All 32 lanes call; lane k holds w_k.
template <typename Y>
__device__ __forceinline__ void reduce_rows(float (&acc)[8], const uint8_t* p, uint32_t stride, uint32_t K, uint32_t have,
                                            float w) {
  constexpr int N = VecElems<Y>::N;
  auto add = [&](uint32_t k) {
    const float wk = __shfl_sync(0xffffffffu, w, k);
    float f[8];
    VecElems<Y>::unpack(*reinterpret_cast<const Vec16*>(p + k * stride), f);
    #pragma unroll
    for (int q = 0; q < N; ++q) acc[q] = fmaf(wk, f[q], acc[q]);
  };
  if (have == (1u << K) - 1u) {   // the rule: no branch between the loads
    uint32_t k = 0;
    for (; k + 8 <= K; k += 8) {
      #pragma unroll
      for (uint32_t u = 0; u < 8; ++u) add(k + u);
    }
    for (; k + 2 <= K; k += 2) {
      add(k);
      add(k + 1);
    }
    if (k < K) add(k);
  } else {
    for (uint32_t k = 0; k < K; ++k) {
      if ((have >> k) & 1u) add(k);
    }
  }
}

// Many tokens: every warp has the rows of a piece of a token brought into one of its two buffers in
// shared memory by the bulk-copy engine and reduces them from there while the next piece's are on
// their way. With register loads a warp has 4 KiB in flight at most and waits for its routes in
// between (118 us for 4096 tokens of 8 rows of 14 KiB, 4.3 TB/s).
constexpr int kBulkWarps = 12;
constexpr uint32_t kBulkBuffer = 8 * 1024;   // the rows of one piece; two a warp

template <typename Y, typename O>
__global__ void __launch_bounds__(kBulkWarps * 32, 1) combine_bulk_kernel(const __grid_constant__ SingleCombine c) {
  extern __shared__ __align__(128) uint8_t dyn_smem[];
  __shared__ uint64_t s_bars[kBulkWarps][2];
  const A2AConfig& cfg = c.cfg;
  const CombineRecvArgs& a = c.recv;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t K = cfg.topk;
  uint64_t* const bars = s_bars[warp];
  if (lane == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  grid_wait();
  grid_allow_next();
  const uint32_t T = bounded_tokens(cfg, a.num_tokens, a.bound_m);
  const uint32_t epoch = a.external ? read_epoch(c.ws, 1) : 0u;
  const uint32_t dispatched = tokens_dispatched(c);
  const uint32_t status = combine_status(c);
  constexpr int N = VecElems<Y>::N;   // elements of a 16-byte vector
  const uint32_t row_bytes = static_cast<uint32_t>(cfg.hidden_dim) * sizeof(Y);
  const uint32_t seg = c.segment;     // bytes of every row in a piece, a multiple of 512
  const uint32_t pieces = (row_bytes + seg - 1) / seg;
  const uint32_t jobs = T * pieces;
  const uint32_t step = gridDim.x * kBulkWarps;
  // Routes are fetched one job before the rows, rows one job before they are reduced.
  uint32_t job = blockIdx.x * kBulkWarps + warp;   // the warps of a block work on neighbouring pieces
  auto route = [&](uint32_t j) { return j < jobs ? load_route(c, j / pieces, lane) : Route(); };
  const Route first = route(job);
  if (__all_sync(0xffffffffu, status == 0)) {
    // rows of a kernel that is still running on another stream: written by plain stores that the
    // arrival counter covers, read by the bulk-copy engine below
    if (a.external) asm volatile("fence.proxy.async;" ::: "memory");
    uint8_t* const buffers = dyn_smem + warp * 2 * kBulkBuffer;
    auto fetch = [&](uint32_t j, const Route& route, uint32_t slot) -> uint32_t {   // returns which rows come
      if (j >= jobs) return 0;
      const uint32_t r = route_place(c, route, j / pieces, dispatched);
      const uint32_t have = __ballot_sync(0xffffffffu, r != kNoSlot);
      if (have != 0) {
        const uint32_t off = j % pieces * seg;
        const uint32_t bytes = min(seg, row_bytes - off);
        if (lane == 0) mbar_expect_tx(&bars[slot], __popc(have) * bytes);
        __syncwarp();
        if (r != kNoSlot) {
          bulk_g2s(buffers + slot * kBulkBuffer + lane * seg, c.rows + static_cast<uint64_t>(r) * c.row_stride + off, bytes,
                   &bars[slot]);
        }
      }
      return have;
    };
    uint32_t have = fetch(job, first, 0);
    float w = first.w;
    Route next = route(job + step);
    uint32_t slot = 0, parities = 0;
    for (; job < jobs; job += step) {
      const uint32_t next_have = fetch(job + step, next, slot ^ 1u);   // no rows past the last job
      const Route after = route(job + 2 * step);
      const uint32_t t = job / pieces, off = job % pieces * seg;
      const uint32_t bytes = min(seg, row_bytes - off);
      if (have != 0) {
        if (!__all_sync(0xffffffffu, mbar_wait_timed(&bars[slot], (parities >> slot) & 1u, cfg.wait_limit_ns))) {
          if (lane == 0) report(c.ws, kStatusWaitTimeout, kPhaseCombineRecv, t, bytes);
        }
        parities ^= 1u << slot;
      }
      uint8_t* out_row = a.out_tokens + static_cast<uint64_t>(t) * a.out_tokens_stride * sizeof(O);
      for (uint32_t i0 = 0; i0 < bytes; i0 += 512) {
        const uint32_t i = i0 + 16 * lane;
        const bool inside = i < bytes;   // past the end a lane reads stale bytes of its buffer and drops them
        const uint64_t elem = (off + i) / sizeof(Y);
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (a.accumulate && inside) load_elems<O, N>(out_row, elem, acc);
        reduce_rows<Y>(acc, buffers + slot * kBulkBuffer + i, seg, K, have, w);
        if (inside) store_elems<O, N>(out_row, elem, acc);
      }
      __syncwarp();   // the buffer is filled again
      have = next_have;
      w = next.w;
      next = after;
      slot ^= 1u;
    }
  }
  combine_finish(c, epoch);
}

template <typename Y, typename O>
__global__ void __launch_bounds__(kCombineThreads, 1) combine_single_kernel(const __grid_constant__ SingleCombine c) {
  const A2AConfig& cfg = c.cfg;
  const A2ALocal& ws = c.ws;
  const CombineRecvArgs& a = c.recv;
  const uint32_t K = cfg.topk;
  const uint32_t lane = threadIdx.x & 31u;
  grid_wait();
  grid_allow_next();
  const int T = bounded_tokens(cfg, a.num_tokens, a.bound_m);
  const uint32_t epoch = a.external ? read_epoch(ws, 1) : 0u;
  const uint32_t dispatched = tokens_dispatched(c);
  const uint32_t status = combine_status(c);
  const uint32_t ngran = cfg.hidden_dim / 8;
  const uint32_t pieces = (ngran + 31) / 32;
  constexpr int kVecs = Elem8<Y>::kBytes / 16;
  constexpr int U = 8 / kVecs;   // rows in flight per lane
  const uint32_t warps = gridDim.x * kCombineWarps;
  for (uint32_t unit = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; unit < T * pieces; unit += warps) {
    const uint32_t t = unit / pieces;
    const Route route = load_route(c, t, lane);
    if (__any_sync(0xffffffffu, status != 0)) break;   // comes in with the first routes
    const uint32_t my_row = route_place(c, route, t, dispatched);
    const float my_w = route.w;
    uint8_t* out_row = a.out_tokens + static_cast<uint64_t>(t) * a.out_tokens_stride * sizeof(O);
    const uint32_t g = unit % pieces * 32 + lane;
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
  combine_finish(c, epoch);
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
  SingleDispatch d{cfg, ws, send, recv, 0, 1};
  const int blocks = cfg.num_blocks;
  const int64_t nvec = cfg.d_payload_bytes / 16;
  const int64_t pieces = (cfg.d_payload_bytes + kPieceBytes - 1) / kPieceBytes;
  // The bulk way where every warp gets two pieces at least; below, one vector a lane, and where there
  // are fewer tokens than half the blocks several blocks share a token.
  const bool bulk = send.num_tokens * pieces >= 2ll * blocks * kSingleWarps;
  if (!bulk && send.num_tokens > 0) {
    d.parts = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(blocks / send.num_tokens, (nvec + 31) / 32)));
  }
  // (scales nobody asks for are not written, quantised or not)
  d.bulk_scales = recv.out_x_scale != nullptr && recv.out_x_scale_stride_elem == 1 && recv.out_x_scale_stride_token % 4 == 0 &&
                  cfg.hidden_dim_scale % 4 == 0 && reinterpret_cast<uintptr_t>(recv.out_x_scale) % 16 == 0;
  const size_t smem = 2 * sizeof(uint32_t) * cfg.num_experts + (bulk ? kSingleWarps * 2 * kPieceBuffer : 0);
  void* args[] = {&d};
  const void* kernel = send.quantize != 0
                           ? (bulk ? reinterpret_cast<const void*>(dispatch_single_kernel<true, true>)
                                   : reinterpret_cast<const void*>(dispatch_single_kernel<false, true>))
                           : (bulk ? reinterpret_cast<const void*>(dispatch_single_kernel<true, false>)
                                   : reinterpret_cast<const void*>(dispatch_single_kernel<false, false>));
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
  }
  return launch_overlapped(kernel, dim3(blocks), dim3(kSingleThreads), args, smem, stream);
}

cudaError_t a2a_launch_combine_single(const A2AConfig& cfg, const A2ALocal& ws, const CombineRecvArgs& recv,
                                      const uint8_t* rows, uint64_t row_stride, const uint32_t* arrived, int y_dtype,
                                      int out_dtype, cudaStream_t stream) {
  SingleCombine c{cfg, ws, recv, rows, row_stride, arrived, 1};
  // As much of every row as a buffer holds for all of a token's rows. Where that leaves every warp four
  // pieces or more their loads overlap; below, the shorter way through registers wins.
  const uint32_t row_bytes = static_cast<uint32_t>(cfg.hidden_dim) * cfg.out_elemsize;
  c.segment = std::min<uint32_t>(kBulkBuffer / cfg.topk / 512 * 512, (row_bytes + 511) / 512 * 512);
  const int64_t pieces = (row_bytes + c.segment - 1) / c.segment;
  // a bulk copy starts and ends on 16-byte boundaries
  const bool bulk = recv.num_tokens * pieces >= 4ll * cfg.num_blocks * kBulkWarps && row_bytes % 16 == 0 &&
                    reinterpret_cast<uintptr_t>(rows) % 16 == 0 && row_stride % 16 == 0;
  return with_types(y_dtype, out_dtype, [&](auto* yp, auto* op) {
    using Y = std::remove_pointer_t<decltype(yp)>;
    using O = std::remove_pointer_t<decltype(op)>;
    void* args[] = {&c};
    if (bulk) {
      constexpr int kSmem = kBulkWarps * 2 * kBulkBuffer;
      const cudaError_t e = cudaFuncSetAttribute(combine_bulk_kernel<Y, O>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
      if (e != cudaSuccess) return e;
      return launch_overlapped(reinterpret_cast<const void*>(combine_bulk_kernel<Y, O>), dim3(cfg.num_blocks),
                               dim3(kBulkWarps * 32), args, kSmem, stream);
    }
    return launch_overlapped(reinterpret_cast<const void*>(combine_single_kernel<Y, O>), dim3(cfg.num_blocks),
                             dim3(kCombineThreads), args, 0, stream);
  });
}

cudaError_t a2a_preload_single() {
  cudaFuncAttributes attr;
  cudaError_t e = cudaFuncGetAttributes(&attr, dispatch_single_kernel<true, true>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, dispatch_single_kernel<false, true>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, dispatch_single_kernel<true, false>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, dispatch_single_kernel<false, false>);
  for (int y : {kDtypeBF16, kDtypeF16, kDtypeF32}) {
    for (int o : {kDtypeBF16, kDtypeF16, kDtypeF32}) {
      if (e != cudaSuccess) return e;
      e = with_types(y, o, [&](auto* yp, auto* op) {
        using Y = std::remove_pointer_t<decltype(yp)>;
        using O = std::remove_pointer_t<decltype(op)>;
        const cudaError_t q = cudaFuncGetAttributes(&attr, combine_bulk_kernel<Y, O>);
        return q != cudaSuccess ? q : cudaFuncGetAttributes(&attr, combine_single_kernel<Y, O>);
      });
    }
  }
  return e;
}

}  // namespace pplx
