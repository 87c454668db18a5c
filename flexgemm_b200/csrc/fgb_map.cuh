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
  uint32_t* host_words;         // host slot (flexgemm_b200.h), or null
  uint32_t host_seq;
};

// The block schedule: row blocks (pairs of 128-row tiles) by descending cost, a block's cost being the number of (tile,
// offset) products it runs.
// Costs of a block of two tiles lie in 0 .. 64.  Blocks of equal cost mostly stand together (the rows are sorted by
// mask), so a warp takes its places by one atomic per distinct cost, not per block.
struct ScheduleSmem {
  uint32_t count[65], start[65];
};
__device__ __forceinline__ void block_schedule(ScheduleSmem& sm, const uint32_t* masks, uint32_t num_tiles, uint32_t nb,
                                               uint32_t* __restrict__ order) {
  const int t = threadIdx.x, lane = t & 31;
  if (t < 65) sm.count[t] = 0;
  __syncthreads();
  auto cost_of = [&](uint32_t b) {  // the masks may have been written by other CTAs of this launch: loads that bypass L1
    const uint32_t t0 = 2 * b;
    return __popc(__ldcg(&masks[t0])) + (t0 + 1 < num_tiles ? __popc(__ldcg(&masks[t0 + 1])) : 0);
  };
  auto take = [&](uint32_t* counters, uint32_t b) -> uint32_t {  // whole warps call it; a place for every lane with b < nb
    const bool ok = b < nb;
    const int c = ok ? cost_of(b) : 65;
    const unsigned peers = __match_any_sync(0xffffffffu, c);
    const int leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if (ok && lane == leader) base = atomicAdd(&counters[c], static_cast<uint32_t>(__popc(peers)));
    base = __shfl_sync(0xffffffffu, base, leader);
    return base + static_cast<uint32_t>(__popc(peers & ((1u << lane) - 1u)));
  };
  for (uint32_t b0 = t - lane; b0 < nb; b0 += blockDim.x) take(sm.count, b0 + lane);
  __syncthreads();
  if (t == 0) {
    uint32_t acc = 0;
    for (int c = 64; c >= 0; --c) {
      sm.start[c] = acc;
      acc += sm.count[c];
    }
  }
  __syncthreads();
  for (uint32_t b0 = t - lane; b0 < nb; b0 += blockDim.x) {
    const uint32_t pos = take(sm.start, b0 + lane);
    if (b0 + lane < nb) order[pos] = b0 + lane;
  }
}
// The sort's digit histograms of rows in no order, made beside the scan.  The map kernel's own (emit_codes) are cheap while
// neighbouring rows share their codes; of shuffled rows every CTA would bring some 256 bins a pass to the global ones
// (164 k shuffled voxels: 17 us of a build, 5.3 M: 34).
struct HistJob {
  const int32_t* codes;
  uint32_t n;
  uint32_t* hist;            // null: no histograms
  const uint32_t* unsorted;  // they are made where this word is not 0
};
cudaError_t launch_block_scan(uint32_t* block_counts, uint32_t nblk, int V, uint32_t* seg, const ScanFinish& fin, const HistJob& job,
                              cudaStream_t s);

// ------------------------------------------------------------------ small inputs (fgb_small.cu)
constexpr int64_t kSmallRows = 8192;  // up to here one CTA sorts and plans, and a map CTA keeps the whole hash table in shared memory

// what one CTA derives from a map's codes
struct PlanJob {
  const int32_t* codes;   // [n] binary codes
  const int32_t* gray;    // [n]
  uint32_t n;
  int V;
  int64_t* sorted_idx;    // [n]
  uint32_t* tile_masks;   // [ceil(n / 128)]
  uint32_t* block_order;  // [ceil(n / 256)]
  uint32_t* counts;       // [V, nblk] per-block counts to turn into offsets, or null
  uint32_t* seg;          // with counts: the segment table [V + 1] (+ the words of `fin`)
  ScanFinish fin;
};
// one or two jobs (a null second one is left out), a CTA each
cudaError_t launch_small_plan(const PlanJob& a, const PlanJob* b, cudaStream_t s);
// the submanifold map of n <= kSmallRows rows
cudaError_t launch_small_map(const int32_t* coords, uint32_t n, int W, int H, int D, const int32_t* k, const int32_t* dil, int key_bits,
                             const MapOut& o, cudaStream_t s);

}  // namespace fgb
