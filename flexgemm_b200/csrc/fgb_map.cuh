// What the kernels that make a neighbour map share (fgb_neighbor_map.cu, fgb_strided.cu): the codes derived from a map
// row, the sort's digit histograms, the scan of the per-block counts.
#pragma once

#include "fgb_common.cuh"
#include "fgb_device.cuh"
#include "fgb_sort.cuh"

namespace fgb {

// What the map kernels hand on: the map and everything that later passes need from it.
struct MapOut {
  uint32_t* nbr;           // [n, V]
  int32_t* gray;           // [n]
  int32_t* binary;         // [n]
  uint32_t* block_counts;  // [V, nblk]
  uint32_t* digit_hist;    // the sort's digit histograms (fgb_sort.cuh), or null
  uint32_t nblk;
};

__device__ __forceinline__ uint32_t gray_to_binary(uint32_t x) {  // prefix xor from the top bit down
  x ^= x >> 1;
  x ^= x >> 2;
  x ^= x >> 4;
  x ^= x >> 8;
  x ^= x >> 16;
  return x;
}

// Writes the codes of the CTA's voxels and, where the sort follows, adds them to its digit histograms (which saves the
// sort's own pass over the codes): runs of equal codes in a warp -- neighbouring voxels mostly share theirs -- count once
// in shared memory, and the CTA's non-zero bins go to the global histograms.
__device__ __forceinline__ void emit_codes(const MapOut& o, uint32_t n0, uint32_t nv, int V, uint32_t gray, uint32_t* s_hist) {
  const int t = threadIdx.x, lane = t & 31;
  const uint32_t binary = gray_to_binary(gray);
  if (t < nv) {
    o.gray[n0 + t] = static_cast<int32_t>(gray);
    o.binary[n0 + t] = static_cast<int32_t>(binary);
  }
  if (o.digit_hist == nullptr) return;  // uniform
  const int passes = sort_passes_of(V);
  __syncthreads();  // s_hist lies over what the lookup has used
  for (int i = t; i < passes * kSortDigits; i += kMapBlock) s_hist[i] = 0;
  __syncthreads();
  const uint32_t key = sort_key_of(binary, V);
  const uint32_t prev = __shfl_up_sync(0xffffffffu, key, 1);
  const bool ok = t < nv;
  const unsigned valid = __ballot_sync(0xffffffffu, ok);
  const unsigned heads = __ballot_sync(0xffffffffu, ok && (lane == 0 || key != prev));
  if (heads >> lane & 1u) {
    const unsigned later = heads & ~((2u << lane) - 1u);
    const uint32_t len = static_cast<uint32_t>((later != 0u ? __ffs(later) - 1 : __popc(valid)) - lane);
    for (int p = 0; p < passes; ++p) atomicAdd(&s_hist[p * kSortDigits + sort_digit_of(key, p)], len);
  }
  __syncthreads();
  for (int i = t; i < passes * kSortDigits; i += kMapBlock) {
    const uint32_t c = s_hist[i];
    if (c != 0u) atomicAdd(&o.digit_hist[i], c);
  }
}

// Mask of the valid offsets of the thread's row of a map tile [rows][V] in shared memory; the CTA's valid counts per
// offset are added to s_count (for the pair-list offsets): lane v of each warp keeps the warp's count of offset v.
__device__ __forceinline__ uint32_t tile_codes(const uint32_t* s_nbr, uint32_t* s_count, uint32_t nv, int V) {
  const int t = threadIdx.x, lane = t & 31;
  uint32_t gray = 0;
  if (t < nv) {
    for (int k = 0; k < V; ++k) {
      if (s_nbr[t * V + k] != kInvalid) gray |= 1u << k;
    }
  }
  uint32_t mine = 0;
  for (int v = 0; v < V; ++v) {
    const uint32_t b = __ballot_sync(0xffffffffu, (gray >> v) & 1u);
    if (lane == v) mine = static_cast<uint32_t>(__popc(b));
  }
  if (lane < V && mine != 0u) atomicAdd(&s_count[lane], mine);
  return gray;
}

// What a build leaves for the host (besides the tensors): see block_scan_kernel.
struct ScanFinish {
  uint32_t* done;               // zeroed word: count of finished CTAs; null = leave the totals as they are
  const uint32_t* unsorted;     // copied to seg[V + 1] when not null
  const int32_t* build_status;  // copied to seg[V + 2] when not null
  uint32_t* host_words;         // mapped pinned memory [V + 3], then the sequence word; null = not wanted
  uint32_t host_seq;
};

cudaError_t launch_block_scan(uint32_t* block_counts, uint32_t nblk, int V, uint32_t* seg, const ScanFinish& fin, cudaStream_t s);

}  // namespace fgb
