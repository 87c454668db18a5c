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
