#include "peer_copy.h"

#include <algorithm>

#include "../a2a/ptx.cuh"

namespace pplx::fabric {
namespace {

constexpr uint32_t kRingBytes = 128 * 1024;  // shared memory of a bulk-copy CTA: chunks in flight
constexpr uint32_t kMaxStages = 8;
constexpr int kBulkThreads = 32;
// One bulk copy. Over NVLink large chunks are best; inside one GPU smaller ones spread a transfer
// over all SMs more evenly (1188 chunks of 32 KiB are 8.03 a CTA: nine rounds for eight).
constexpr uint32_t kPeerChunkBytes = 32 * 1024;
constexpr uint32_t kLocalChunkBytes = 16 * 1024;
constexpr int kPeerCtas = 64;                    // enough to saturate NVLink
constexpr uint64_t kSmallPageBytes = 16 * 1024;  // at or below: one warp per page (paged_copy_rows_kernel)
constexpr uint32_t kSimtChunkBytes = 32 * 1024;

// Page tables travel inside the kernel's parameters where they fit: no copy to the device in front
// of the kernel, no device buffer. Otherwise they are in device memory, or absent (page i is at
// index i).
struct DeviceTables {
  PagedCopyArgs c;
  __device__ __forceinline__ uint64_t src(uint32_t i) const {
    return (c.src_pages != nullptr ? c.src_pages[i] : i) * c.src_stride + c.src_offset;
  }
  __device__ __forceinline__ uint64_t dst(uint32_t i) const {
    return (c.dst_pages != nullptr ? c.dst_pages[i] : i) * c.dst_stride + c.dst_offset;
  }
};
struct InlineTables {
  PagedCopyArgs c;
  uint32_t pages[2 * kPagedCopyInlinePages];   // source, then destination
  __device__ __forceinline__ uint64_t src(uint32_t i) const { return pages[i] * c.src_stride + c.src_offset; }
  __device__ __forceinline__ uint64_t dst(uint32_t i) const {
    return pages[kPagedCopyInlinePages + i] * c.dst_stride + c.dst_offset;
  }
};
static_assert(sizeof(InlineTables) <= 4096, "kernel parameters");

// One elected thread per CTA drives a ring of shared-memory stages:
//   global --cp.async.bulk--> smem stage --cp.async.bulk--> (peer) global
// Loads complete on an mbarrier per stage, stores in bulk groups; a stage is reused once
// the store that read it has finished reading. SMs only issue descriptors.
template <typename Tables>
__global__ void __launch_bounds__(kBulkThreads)
paged_copy_bulk_kernel(const __grid_constant__ Tables t, const uint32_t chunk, const uint32_t stages) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t bars[kMaxStages];
  if (threadIdx.x != 0) return;
  const PagedCopyArgs& a = t.c;

  for (uint32_t s = 0; s < stages; ++s) mbar_init(&bars[s], 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");

  const uint32_t chunks_per_page = static_cast<uint32_t>((a.length + chunk - 1) / chunk);
  const uint64_t total = static_cast<uint64_t>(a.num_pages) * chunks_per_page;
  uint32_t phases = 0;   // bit s: the parity stage s waits for next
  uint64_t issued = 0;
  uint32_t load_stage = 0, store_stage = 0;
  bool failed = false;

  // Software pipeline: keep up to `stages` loads in flight, store each as it lands.
  auto item_of = [&](uint64_t n) { return blockIdx.x + n * gridDim.x; };
  auto load = [&](uint64_t n) {
    const uint64_t item = item_of(n);
    const uint32_t page = static_cast<uint32_t>(item / chunks_per_page);
    const uint64_t within = (item % chunks_per_page) * chunk;
    const uint32_t bytes = static_cast<uint32_t>(min(static_cast<uint64_t>(chunk), a.length - within));
    mbar_expect_tx(&bars[load_stage], bytes);
    bulk_g2s(smem + load_stage * chunk, a.src_base + t.src(page) + within, bytes, &bars[load_stage]);
    load_stage = load_stage + 1 == stages ? 0 : load_stage + 1;
  };
  uint64_t mine = 0;
  if (total > blockIdx.x) mine = (total - blockIdx.x + gridDim.x - 1) / gridDim.x;

  for (; issued < mine && issued < stages; ++issued) load(issued);
  for (uint64_t n = 0; n < mine; ++n) {
    const uint32_t s = store_stage;
    if (!mbar_wait_timed(&bars[s], (phases >> s) & 1u, 2000000000ull)) {
      failed = true;
      break;
    }
    phases ^= 1u << s;
    store_stage = s + 1 == stages ? 0 : s + 1;
    const uint64_t item = item_of(n);
    const uint32_t page = static_cast<uint32_t>(item / chunks_per_page);
    const uint64_t within = (item % chunks_per_page) * chunk;
    const uint32_t bytes = static_cast<uint32_t>(min(static_cast<uint64_t>(chunk), a.length - within));
    fence_proxy_async_smem();
    bulk_s2g(a.dst_base + t.dst(page) + within, smem + s * chunk, bytes);
    bulk_commit();
    // All but the newest store have finished reading their stage: the stage of store
    // n - 1 is free for the next load, while store n still overlaps with it.
    asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
    if (n >= 1 && issued < mine) {
      load(issued);  // issued == n - 1 + stages: lands in the stage of store n - 1
      ++issued;
    }
  }
  // Stores must be complete (not merely read) before the kernel, and with it the stream
  // event the host polls, finishes.
  bulk_wait0();
  if (failed) {
    atomicExch(a.error_flag, 1u);
    // loads that are still in flight land in this CTA's shared memory: wait for them
    // (bounded) before the CTA may exit
    for (uint64_t n = 0; n < issued && n < stages; ++n) {
      (void)mbar_wait_timed(&bars[n], (phases >> n) & 1u, 100000000ull);
    }
  }
}

// Fallback for arbitrary alignment: 16-byte vectors where both sides allow it, bytes else.
template <typename Tables>
__global__ void __launch_bounds__(256) paged_copy_simt_kernel(const __grid_constant__ Tables t) {
  const PagedCopyArgs& a = t.c;
  const uint32_t chunks_per_page = static_cast<uint32_t>((a.length + kSimtChunkBytes - 1) / kSimtChunkBytes);
  const uint64_t total = static_cast<uint64_t>(a.num_pages) * chunks_per_page;
  for (uint64_t item = blockIdx.x; item < total; item += gridDim.x) {
    const uint32_t page = static_cast<uint32_t>(item / chunks_per_page);
    const uint64_t within = (item % chunks_per_page) * kSimtChunkBytes;
    const uint64_t bytes = min(static_cast<uint64_t>(kSimtChunkBytes), a.length - within);
    const uint8_t* src = a.src_base + t.src(page) + within;
    uint8_t* dst = a.dst_base + t.dst(page) + within;
    const bool aligned = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0;
    if (aligned) {
      const uint64_t nvec = bytes / 16;
      for (uint64_t i = threadIdx.x; i < nvec; i += blockDim.x) {
        st_stream_v4(dst + 16 * i, ld_input_v4(src + 16 * i));
      }
      for (uint64_t i = nvec * 16 + threadIdx.x; i < bytes; i += blockDim.x) dst[i] = src[i];
    } else {
      for (uint64_t i = threadIdx.x; i < bytes; i += blockDim.x) dst[i] = src[i];
    }
  }
}

// Many small pages (rows of a weight shard, short KV pages): one warp per page, 16-byte vectors,
// four loads in flight per lane, as many CTAs as it takes to have every SM storing. A page this
// small is not worth a bulk-copy descriptor and a shared-memory round trip per page; what counts
// is how many independent pages are in flight.
constexpr int kRowsWarps = 8;

template <typename Tables>
__global__ void __launch_bounds__(kRowsWarps * 32) paged_copy_rows_kernel(const __grid_constant__ Tables t) {
  const PagedCopyArgs& a = t.c;
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t warp = static_cast<uint64_t>(blockIdx.x) * kRowsWarps + (threadIdx.x >> 5);
  const uint64_t warps = static_cast<uint64_t>(gridDim.x) * kRowsWarps;
  const uint32_t nvec = static_cast<uint32_t>(a.length / 16);
  for (uint64_t page = warp; page < a.num_pages; page += warps) {
    const uint8_t* src = a.src_base + t.src(static_cast<uint32_t>(page));
    uint8_t* dst = a.dst_base + t.dst(static_cast<uint32_t>(page));
    for (uint32_t i0 = lane; i0 < nvec; i0 += 128) {
      Vec16 v[4];
      #pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (i0 + 32 * u < nvec) v[u] = ld_input_v4(src + 16ull * (i0 + 32 * u));
      }
      #pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (i0 + 32 * u < nvec) st_stream_v4(dst + 16ull * (i0 + 32 * u), v[u]);
      }
    }
  }
}

int sm_count() {
  int sms = 0, device = 0;
  cudaGetDevice(&device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return std::max(sms, 1);
}

template <typename Tables>
cudaError_t launch(const Tables& t, bool local, int max_ctas, cudaStream_t stream) {
  const PagedCopyArgs& args = t.c;
  const uint64_t all = reinterpret_cast<uintptr_t>(args.src_base) | reinterpret_cast<uintptr_t>(args.dst_base) |
                       args.src_stride | args.dst_stride | args.src_offset | args.dst_offset | args.length;
  const bool aligned = (all & 15u) == 0;
  // A copy inside one GPU is bound by HBM, which takes every SM: 297 pages of 128 KiB in 11.7 us, and in
  // 19.6 us with 64 CTAs. Beside compute the whole grid is no worse: an expert GEMM that fills the GPU
  // took 133 us a launch with such copies back to back on another stream, and 139 us with 64 CTAs
  // (114 to 131 us alone, by what the power limit allows); a pass of four copies 1065 and 1107 us.
  if (max_ctas <= 0) max_ctas = local ? sm_count() : kPeerCtas;
  if (aligned && args.length <= kSmallPageBytes && args.num_pages >= 64) {
    const uint64_t wanted = (args.num_pages + kRowsWarps - 1) / kRowsWarps;
    const int grid = static_cast<int>(std::min<uint64_t>(wanted, static_cast<uint64_t>(sm_count()) * 4));
    paged_copy_rows_kernel<<<grid, kRowsWarps * 32, 0, stream>>>(t);
  } else if (aligned) {
    // per device and cheap: set it on every launch rather than tracking devices
    cudaError_t e = cudaFuncSetAttribute(paged_copy_bulk_kernel<Tables>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(kRingBytes));
    if (e != cudaSuccess) return e;
    const uint32_t chunk = local ? kLocalChunkBytes : kPeerChunkBytes;
    const uint64_t total = args.num_pages * ((args.length + chunk - 1) / chunk);
    const int grid = static_cast<int>(std::min<uint64_t>(total, static_cast<uint64_t>(max_ctas)));
    paged_copy_bulk_kernel<<<grid, kBulkThreads, kRingBytes, stream>>>(t, chunk, kRingBytes / chunk);
  } else {
    const uint64_t total = args.num_pages * ((args.length + kSimtChunkBytes - 1) / kSimtChunkBytes);
    const int grid = static_cast<int>(std::min<uint64_t>(total, static_cast<uint64_t>(max_ctas)));
    paged_copy_simt_kernel<<<grid, 256, 0, stream>>>(t);
  }
  return cudaGetLastError();
}

template <typename Tables>
cudaError_t warm_up(const Tables& t, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(paged_copy_bulk_kernel<Tables>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(kRingBytes));
  if (e != cudaSuccess) return e;
  paged_copy_bulk_kernel<<<1, kBulkThreads, kRingBytes, stream>>>(t, kLocalChunkBytes, kRingBytes / kLocalChunkBytes);
  paged_copy_simt_kernel<<<1, 256, 0, stream>>>(t);
  paged_copy_rows_kernel<<<1, kRowsWarps * 32, 0, stream>>>(t);
  return cudaGetLastError();
}

static_assert(kRingBytes / kLocalChunkBytes <= kMaxStages && kRingBytes / kPeerChunkBytes <= kMaxStages, "barriers");

}  // namespace

cudaError_t launch_paged_copy(const PagedCopyArgs& args, const uint32_t* host_src_pages, const uint32_t* host_dst_pages,
                              bool local, int max_ctas, cudaStream_t stream) {
  if (args.num_pages == 0 || args.length == 0) return cudaSuccess;
  if (host_src_pages == nullptr) return launch(DeviceTables{args}, local, max_ctas, stream);
  if (args.num_pages > kPagedCopyInlinePages) return cudaErrorInvalidValue;
  InlineTables t;
  t.c = args;
  std::copy_n(host_src_pages, args.num_pages, t.pages);
  std::copy_n(host_dst_pages, args.num_pages, t.pages + kPagedCopyInlinePages);
  return launch(t, local, max_ctas, stream);
}

cudaError_t warm_up_paged_copy(cudaStream_t stream) {
  // Empty launches: the kernels return at once, but their code is loaded and their attributes
  // are set. With lazy module loading the first launch of a kernel may otherwise have to wait
  // for kernels that are running, and one of those may be waiting for this copy.
  cudaError_t e = warm_up(DeviceTables{}, stream);
  if (e == cudaSuccess) e = warm_up(InlineTables{}, stream);
  if (e != cudaSuccess) return e;
  return cudaStreamSynchronize(stream);
}

}  // namespace pplx::fabric
