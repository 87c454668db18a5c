// What the map kernels and the sort share: the digits of a sort key, and the sort's launch on prepared memory.
#pragma once

#include "fgb_common.cuh"

namespace fgb {

constexpr int kSortDigitBits = 9;
constexpr int kSortDigits = 1 << kSortDigitBits;  // 512
constexpr int kSortMaxPasses = 4;                 // 32 bits / 9

__host__ __device__ constexpr int sort_passes_of(int key_bits) { return (key_bits + kSortDigitBits - 1) / kSortDigitBits; }
// Codes with fewer than 32 significant bits are non-negative; with 32 bits they are signed, and flipping the top bit
// makes the unsigned digit order the signed order.
__host__ __device__ constexpr uint32_t sort_flip_of(int key_bits) { return key_bits == 32 ? 0x80000000u : 0u; }
__host__ __device__ constexpr uint32_t sort_key_of(uint32_t code, int key_bits) { return code ^ sort_flip_of(key_bits); }
__host__ __device__ constexpr uint32_t sort_digit_of(uint32_t key, int pass) { return (key >> (pass * kSortDigitBits)) & (kSortDigits - 1); }

// hist[p * 512 + d] += number of codes whose digit p is d, for every pass p, over share `block` of `blocks` of the codes.
// The whole CTA calls it; s_h [passes * 512] is zeroed.
__device__ __forceinline__ void digit_histograms(uint32_t* s_h, const int32_t* __restrict__ codes, uint32_t n, int key_bits, uint32_t block,
                                                 uint32_t blocks, uint32_t* __restrict__ hist) {
  const int lane = threadIdx.x & 31, passes = sort_passes_of(key_bits);
  const uint32_t per = (n + blocks - 1) / blocks;
  const uint32_t begin = min(n, block * per), end = min(n, begin + per);
  // whole warps walk the range so that every lane takes part in the votes
  for (uint32_t i0 = begin + (threadIdx.x & ~31u); i0 < end; i0 += blockDim.x) {
    const uint32_t i = i0 + lane;
    const bool ok = i < end;
    const uint32_t key = ok ? sort_key_of(static_cast<uint32_t>(__ldg(&codes[i])), key_bits) : 0u;
    const unsigned valid = __ballot_sync(0xffffffffu, ok);  // a prefix of the lanes
    // neighbouring voxels mostly share their code: the warp's keys are cut into runs of equal keys, and the first
    // lane of a run adds the run's length to the key's bin of every pass (equal keys share all their digits)
    const uint32_t prev = __shfl_up_sync(0xffffffffu, key, 1);
    const bool head = ok && (lane == 0 || key != prev);
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    if (head) {
      const unsigned later = heads & ~((2u << lane) - 1u);  // run heads above this lane
      const int next = later != 0u ? __ffs(later) - 1 : __popc(valid);
      const uint32_t len = static_cast<uint32_t>(next - lane);
      for (int p = 0; p < passes; ++p) atomicAdd(&s_h[p * kSortDigits + sort_digit_of(key, p)], len);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * kSortDigits; i += blockDim.x) {
    const uint32_t c = s_h[i];
    if (c != 0u) atomicAdd(&hist[i], c);
  }
}

struct SortLayout {
  size_t keys_a, vals_a, keys_b, vals_b;  // offsets in the key / value buffers
  size_t buffer_bytes;                    // all four
  uint32_t tiles;
  int items;                              // keys per thread
};
SortLayout sort_layout(int64_t n);

// The passes of the argsort (fgb_sort.cu) of `codes` on prepared memory: hist = digit histograms [kSortMaxPasses][512]
// filled in, followed by kSortMaxPasses zeroed tickets; lookback = zeroed words [passes][tiles][512].
cudaError_t launch_sort_passes(const int32_t* codes, int64_t n, int key_bits, int64_t* sorted_idx, char* buffers, const SortLayout& L,
                               uint32_t* hist, uint32_t* lookback, int32_t* err, cudaStream_t s);

// tile masks of 128 sorted rows and the block schedule of the conv kernels in one launch; `counter`: a zeroed word
cudaError_t launch_tile_plan(const int32_t* gray, const int64_t* sorted_idx, int64_t n, uint32_t* tile_masks, uint32_t* block_order,
                             uint32_t* counter, cudaStream_t s);


}  // namespace fgb
