// Block upload into the device cache.
//
// The reference rewrites each block's links on the CPU and issues one
// clEnqueueWriteBuffer per channel plus one 4-byte write per parent pointer and
// far pointer (rayt/GPU data/gpu-octree-cache.cpp:102-234,
// gpu-octree-data.cpp:60-93).  Here one kernel scatters a batch of blocks into
// the channel buffers, rewriting stored links into the cache format on the way
// (gpu-octree-cache.cpp:120-141: a loaded, non-fault link becomes a near
// pointer relative to the node itself), and a second kernel applies the
// parent/far-pointer writes, which the host has reduced to the last write per
// address in the reference's order.  The blocks come either from a staging
// area filled by one host-to-device copy of the batch (upload_kernel) or
// straight from the block file mapped into host memory and registered with the
// device (upload_mapped_kernel: no host copy at all).
#include <algorithm>
#include <cstring>

#include "internal.h"

namespace rayt {
namespace {

constexpr int kThreads = 256;

// One CTA per staged block: a grid-stride copy of each channel section.
__global__ void __launch_bounds__(kThreads) upload_kernel(const __grid_constant__ UploadParams p) {
  const int b = blockIdx.x;
  const size_t nib = (size_t)p.nodes_in_block;
  const uint8_t* src = p.stage + (size_t)b * p.stride;
  if (p.slots[b] < 0) return;  // staged but not placed (read ahead, then not needed)
  const size_t slot = (size_t)p.slots[b];

  // channel 0: node links, stored format -> cache format
  const uint32_t* sl = reinterpret_cast<const uint32_t*>(src);
  uint32_t* dl = reinterpret_cast<uint32_t*>(p.chan[0]) + slot * nib;
  for (size_t n = threadIdx.x; n < nib; n += kThreads) {
    uint32_t l = sl[n];
    const uint32_t mask = l & 255u, fault = (l >> 8) & 1u;
    if (mask && !fault) {
      const uint32_t ptr = l >> 11;
      const uint32_t near_ptr = (1u << 20) + ptr - (uint32_t)n;  // NearPointerValue(n, ptr)
      l = (near_ptr << 11) | (l & (1u << 9)) | mask;             // fault 0, far 0, dup kept
    }
    dl[n] = l;
  }
  // other channels: raw copy, 16 bytes at a time when aligned
  size_t off = nib * 4;
  for (int c = 1; c < p.channels; ++c) {
    const size_t bytes = nib * (size_t)p.chan_bytes[c];
    const uint8_t* s = src + off;
    uint8_t* d = p.chan[c] + slot * bytes;
    if (((reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(d) | bytes) & 15u) == 0) {
      const uint4* s4 = reinterpret_cast<const uint4*>(s);
      uint4* d4 = reinterpret_cast<uint4*>(d);
      for (size_t i = threadIdx.x; i < bytes / 16; i += kThreads) d4[i] = s4[i];
    } else {
      for (size_t i = threadIdx.x; i < bytes; i += kThreads) d[i] = s[i];
    }
    off += bytes;
  }
}

// NearPointerValue rewrite of one stored link (see upload_kernel).
__device__ __forceinline__ uint32_t cache_link(uint32_t l, uint32_t n) {
  const uint32_t mask = l & 255u, fault = (l >> 8) & 1u;
  if (mask && !fault) l = (((1u << 20) + (l >> 11) - n) << 11) | (l & (1u << 9)) | mask;
  return l;
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// What a mapped batch of few blocks carries in its parameters: read from host
// memory, the slots and numbers cost a trip over the host link before the
// contents could be asked for.
struct InlineIds {
  int slots[kInlineBlocks], blocks[kInlineBlocks];
};

// Words [w0, w1) of a block's content (`words` in all, at `a` rounded down to
// whole words, `mis` bytes into the first), stored by `store(i, word)`.  A
// block record starts at any byte offset, so each warp reads rows of 32
// consecutive aligned words, every lane its own, and forms the content words
// with a funnel shift from its word and the next lane's (the row's last lane
// takes the next row's first word; after the last row it reads that word
// itself).  A warp issues kRows rows' loads before it uses them, so that enough
// reads are in flight over the host link.  The aligned words read hold at least
// one byte of the content (or of its block header), so they lie inside the
// file.
constexpr int kRows = 8;
template <typename Store>
__device__ __forceinline__ void copy_words(const uint32_t* a, uint32_t mis, uint32_t words, uint32_t w0, uint32_t w1,
                                           Store store) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t limit = words + (mis ? 1u : 0u);
  // warp-uniform trip count: each warp takes 32 * kRows words at a time
  for (uint32_t i0 = w0 + (uint32_t)warp * 32 * kRows; i0 < w1; i0 += (uint32_t)kThreads * kRows) {
    uint32_t lo[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const uint32_t i = i0 + 32 * r + lane;
      lo[r] = i < limit && i <= w1 ? a[i] : 0u;  // words past w1 are not used, but the one after it
    }
    uint32_t after = 0u;  // the word after the last row, for its last lane
    if (mis && lane == 31 && i0 + 32 * kRows < limit) after = a[i0 + 32 * kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      uint32_t w = lo[r];
      if (mis) {
        uint32_t hi = __shfl_down_sync(0xffffffffu, lo[r], 1);
        const uint32_t next_row = r + 1 < kRows ? __shfl_sync(0xffffffffu, lo[r + 1 < kRows ? r + 1 : r], 0) : after;
        if (lane == 31) hi = next_row;
        w = __funnelshift_r(lo[r], hi, 8u * mis);
      }
      const uint32_t i = i0 + 32 * r + lane;
      if (i < w1) store(i, w);
    }
  }
}

// `parts` CTAs per block, each a contiguous share of the block's content,
// reading it where it lies in the mapped block file (host memory the device
// reads directly).  A read over the host link takes microseconds, so what
// bounds a small batch (a later pass's transaction streams a few dozen blocks)
// is how many trips follow one another: the content is one run of words over
// all channel sections, and a share of it is one round of loads.  Sections of
// odd size are copied one by one, by bytes.
template <bool kInline>
__global__ void __launch_bounds__(kThreads) upload_mapped_kernel(const __grid_constant__ UploadParams p,
                                                                 const __grid_constant__ InlineIds ids) {
  if (blockIdx.x == 0 && threadIdx.x == 0) p.clock->start_ns = global_ns();
  const int b = blockIdx.x / p.parts, part = blockIdx.x - b * p.parts;
  const int slot_or_none = kInline ? ids.slots[b] : p.slots[b];
  if (slot_or_none < 0) return;  // staged but not placed, or superseded
  const size_t slot = (size_t)slot_or_none;
  const int block = kInline ? ids.blocks[b] : p.block_ids[b];
  const size_t nib = (size_t)p.nodes_in_block;
  const uint8_t* src = p.file + p.file_first + p.file_stride * (uint64_t)(uint32_t)block;
  const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 3u);
  if (const uint32_t words = p.section[p.channels]) {
    const uint32_t per = (words + p.parts - 1) / p.parts;
    const uint32_t w0 = min(words, per * part), w1 = min(words, w0 + per);
    copy_words(reinterpret_cast<const uint32_t*>(src - mis), mis, words, w0, w1, [&](uint32_t i, uint32_t w) {
      int c = 0;
#pragma unroll
      for (int k = 1; k < kMaxChannels; ++k) c += k < p.channels && i >= p.section[k];
      const uint32_t first = p.section[c];
      uint32_t* d = reinterpret_cast<uint32_t*>(p.chan[c]) + slot * (p.section[c + 1] - first);
      d[i - first] = c == 0 ? cache_link(w, i) : w;
    });
    return;
  }
  size_t off = 0;  // byte offset of the channel's section in the content
  for (int c = 0; c < p.channels; ++c) {
    const size_t bytes = nib * (size_t)p.chan_bytes[c];
    uint8_t* d = p.chan[c] + slot * bytes;
    if (((off | bytes) & 3u) == 0) {
      const uint32_t words = (uint32_t)(bytes / 4);
      const uint32_t per = (words + p.parts - 1) / p.parts;
      const uint32_t w0 = min(words, per * part), w1 = min(words, w0 + per);
      uint32_t* d4 = reinterpret_cast<uint32_t*>(d);
      copy_words(reinterpret_cast<const uint32_t*>(src + off - mis), mis, words, w0, w1,
                 [&](uint32_t i, uint32_t w) { d4[i] = c == 0 ? cache_link(w, i) : w; });
    } else {  // a section of odd size: bytes (links are always whole words)
      const size_t per = (bytes + p.parts - 1) / p.parts;
      const size_t b0 = min(bytes, per * part), b1 = min(bytes, b0 + per);
      for (size_t i = b0 + threadIdx.x; i < b1; i += kThreads) d[i] = src[off + i];
    }
    off += bytes;
  }
}

struct InlinePatches {
  Patch at[kInlinePatches];
};
// The batch's patches, after its contents: started while those are still on
// their way (a programmatic launch) and held at the dependency.
template <bool kInline>
__global__ void __launch_bounds__(kThreads) patch_kernel(const Patch* patches, int n, uint32_t* links,
                                                         uint32_t* far_ptrs, UploadClock* clock,
                                                         const __grid_constant__ InlinePatches at) {
  const int i = blockIdx.x * kThreads + threadIdx.x;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (i < n) {
    const Patch q = kInline ? at.at[i] : patches[i];
    if (q.far) far_ptrs[q.index] = q.value;
    else links[q.index] = q.value;
  }
  if (clock && i == 0) {
    const unsigned long long total = clock->total_ns + (global_ns() - clock->start_ns);
    clock->total_ns = total;
    *clock->host = total;
  }
}

template <typename... Params, typename... Args>
cudaError_t launch_after(void (*kernel)(Params...), int grid, cudaStream_t s, Args... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace

cudaError_t launch_upload(const UploadParams& p, const int* host_slots, const int* host_blocks, cudaStream_t s) {
  if (p.blocks <= 0) return cudaSuccess;
  if (!p.file) {
    upload_kernel<<<p.blocks, kThreads, 0, s>>>(p);
    return cudaGetLastError();
  }
  // about two CTAs per SM over the batch, at most 8 per block
  static const int sms = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
  }();
  UploadParams q = p;
  q.parts = std::max(1, std::min(8, (2 * sms + p.blocks - 1) / p.blocks));
  uint64_t bytes = 0;
  bool whole = true;  // every section is whole words
  for (int c = 0; c < p.channels; ++c) {
    const uint64_t section = (uint64_t)p.nodes_in_block * (uint64_t)p.chan_bytes[c];
    whole = whole && section % 4 == 0;
    q.section[c] = (uint32_t)(bytes / 4);
    bytes += section;
  }
  q.section[p.channels] = whole ? (uint32_t)(bytes / 4) : 0u;
  const int grid = p.blocks * q.parts;
  InlineIds ids;
  if (p.blocks <= kInlineBlocks) {
    std::memcpy(ids.slots, host_slots, sizeof(int) * (size_t)p.blocks);
    std::memcpy(ids.blocks, host_blocks, sizeof(int) * (size_t)p.blocks);
    upload_mapped_kernel<true><<<grid, kThreads, 0, s>>>(q, ids);
  } else {
    upload_mapped_kernel<false><<<grid, kThreads, 0, s>>>(q, ids);
  }
  return cudaGetLastError();
}

cudaError_t launch_patches(const Patch* patches, int n, uint32_t* links, uint32_t* far_ptrs, UploadClock* clock,
                           cudaStream_t s) {
  if (n <= 0 && !clock) return cudaSuccess;
  const int grid = std::max(1, (n + kThreads - 1) / kThreads);
  InlinePatches at;
  if (n <= kInlinePatches) {
    std::memcpy(at.at, patches, sizeof(Patch) * (size_t)n);
    return launch_after(patch_kernel<true>, grid, s, (const Patch*)nullptr, n, links, far_ptrs, clock, at);
  }
  return launch_after(patch_kernel<false>, grid, s, patches, n, links, far_ptrs, clock, at);
}

}  // namespace rayt
