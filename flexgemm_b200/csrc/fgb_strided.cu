// Output coordinates and both neighbour maps of a strided convolution whose output voxels are those that some input
// voxel reaches (the usual case), rows in flat-index order.
//
// The output voxels are marked as bits of the output grid, one bit per cell.  Counting and prefixing the bits' words then
// gives the sorted, distinct coordinates without a hash set or a sort, and the rank of any marked cell -- the prefix of
// its word plus the set bits below it -- is its row: every (input voxel, offset) pair finds its output row with two
// loads, so both maps are written from the input side (the backward map in row order, the forward map as a scatter)
// without a hash table.  At 128^3 output cells the bits are 262 KB, at 8 x 512^3 128 MB.
// Before, on the RES=256 shell, k = 2, s = 2: hash set 25 us, library sort 36 us, table 16 us, lookup 22 us, and two more
// passes for the backward map's codes; the caller falls back to that path for grids too large for the bits.
#include <algorithm>

#include "fgb_map.cuh"

namespace fgb {

struct StridedGeom {
  int K[3], S[3], P[3], D[3];
  int in[3], out[3];  // grid extents
  int B, V;
};

// calls f(v, flat output cell) for every offset through which the input voxel feeds an output voxel
template <typename F>
__device__ __forceinline__ void for_targets(const int4 c, const StridedGeom& g, F f) {
  if (static_cast<unsigned>(c.x) >= static_cast<unsigned>(g.B)) return;
  auto target = [&](int axis, int pos, int k, int& o) -> bool {
    const int t = pos + g.P[axis] - k * g.D[axis];
    if (t < 0) return false;
    o = t / g.S[axis];
    return o * g.S[axis] == t && o < g.out[axis];
  };
  int v = 0;
  for (int kx = 0; kx < g.K[0]; ++kx) {
    int x;
    if (!target(0, c.y, kx, x)) {
      v += g.K[1] * g.K[2];
      continue;
    }
    for (int ky = 0; ky < g.K[1]; ++ky) {
      int y;
      if (!target(1, c.z, ky, y)) {
        v += g.K[2];
        continue;
      }
      const uint32_t line = ((static_cast<uint32_t>(c.x) * g.out[0] + x) * g.out[1] + y) * static_cast<uint32_t>(g.out[2]);
      for (int kz = 0; kz < g.K[2]; ++kz, ++v) {
        int z;
        if (target(2, c.w, kz, z)) f(v, line + z);
      }
    }
  }
}

// *outside = 1 when a row's batch index has no place in the grid (the hash path takes such rows as they are)
__global__ void __launch_bounds__(256) mark_cells_kernel(const int4* __restrict__ coords, uint32_t n, StridedGeom g, uint32_t* __restrict__ bits,
                                                         uint32_t* outside) {
  chain_release();
  chain_wait();
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;
  if (i >= n) return;
  // consecutive targets often lie in one word: they are collected and set together
  uint32_t word = kInvalid, mask = 0;
  const int4 c = __ldg(&coords[i]);
  if (static_cast<unsigned>(c.x) >= static_cast<unsigned>(g.B)) *outside = 1u;
  for_targets(c, g, [&](int, uint32_t cell) {
    const uint32_t w = cell >> 5, b = 1u << (cell & 31);
    if (w != word) {
      if (mask) atomicOr(&bits[word], mask);
      word = w, mask = 0;
    }
    mask |= b;
  });
  if (mask) atomicOr(&bits[word], mask);
}

constexpr int kRankThreads = 256;
constexpr int kRankWords = kRankThreads * 8;  // words of a CTA

__device__ __forceinline__ uint32_t cta_exclusive(uint32_t x, uint32_t* s_warp, uint32_t* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
  uint32_t inc = x;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += y;
  }
  if (lane == 31) s_warp[w] = inc;
  __syncthreads();
  uint32_t before = 0, all = 0;
  for (int k = 0; k < warps; ++k) {
    const uint32_t t = s_warp[k];
    if (k < w) before += t;
    all += t;
  }
  __syncthreads();
  *total = all;
  return before + inc - x;
}

// words of thread t of a CTA: 8 consecutive ones
__device__ __forceinline__ uint32_t load_words(const uint32_t* bits, uint32_t first, uint32_t (&w)[8]) {
  uint32_t count = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    // the bit array is padded to whole CTAs and zeroed
    const uint4 q = *reinterpret_cast<const uint4*>(bits + first + 4 * h);
    w[4 * h] = q.x, w[4 * h + 1] = q.y, w[4 * h + 2] = q.z, w[4 * h + 3] = q.w;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) count += __popc(w[i]);
  return count;
}

// cta_base[b] = set bits of CTA b's words; the CTA that ends last turns them into exclusive sums and tells the host the
// total
__global__ void __launch_bounds__(kRankThreads) count_cells_kernel(const uint32_t* __restrict__ bits, uint32_t* cta_base,
                                                                   uint32_t* done, const uint32_t* outside, uint32_t* host_words,
                                                                   uint32_t host_seq) {
  __shared__ uint32_t s_warp[32];
  __shared__ bool s_last;
  chain_release();
  chain_wait();
  uint32_t w[8], total;
  cta_exclusive(load_words(bits, blockIdx.x * kRankWords + threadIdx.x * 8, w), s_warp, &total);
  if (threadIdx.x == 0) {
    __stcg(&cta_base[blockIdx.x], total);
    __threadfence();
    s_last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  uint32_t carry = 0;
  for (uint32_t b0 = 0; b0 < gridDim.x; b0 += kRankThreads * 8) {
    uint32_t x[8], sum = 0;
    const uint32_t first = b0 + threadIdx.x * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      x[i] = first + i < gridDim.x ? __ldcg(&cta_base[first + i]) : 0u;
      sum += x[i];
    }
    uint32_t at = carry + cta_exclusive(sum, s_warp, &total);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (first + i < gridDim.x) __stcg(&cta_base[first + i], at);
      at += x[i];
    }
    carry += total;
  }
  if (threadIdx.x == 0) tell_host(host_words, host_seq, carry, 0u, __ldcg(outside));
}

// rows of the marked cells, and the row of the first cell of every word that has one
__global__ void __launch_bounds__(kRankThreads) emit_cells_kernel(const uint32_t* __restrict__ bits, const uint32_t* __restrict__ cta_base,
                                                                  StridedGeom g, uint32_t n_out, uint32_t* __restrict__ rank, int4* __restrict__ out) {
  __shared__ uint32_t s_warp[32];
  chain_release();
  chain_wait();
  uint32_t w[8], total;
  const uint32_t first = blockIdx.x * kRankWords + threadIdx.x * 8;
  uint32_t at = __ldg(&cta_base[blockIdx.x]) + cta_exclusive(load_words(bits, first, w), s_warp, &total);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (w[i] == 0u) continue;
    rank[first + i] = at;
    for (uint32_t m = w[i]; m != 0u; m &= m - 1u, ++at) {
      uint32_t cell = (first + i) * 32u + static_cast<uint32_t>(__ffs(m) - 1);
      const uint32_t z = cell % g.out[2];
      cell /= g.out[2];
      const uint32_t y = cell % g.out[1];
      cell /= g.out[1];
      const uint32_t b = cell / g.out[0], x = cell - b * g.out[0];
      if (at < n_out) out[at] = make_int4(static_cast<int>(b), static_cast<int>(x), static_cast<int>(y), static_cast<int>(z));
    }
  }
}

// Both maps from the input side; one thread per input voxel.  nbr must be filled with ones.  With a backward map the
// CTA's rows of it leave through shared memory, with their codes.
__global__ void __launch_bounds__(kMapBlock) strided_maps_kernel(const int4* __restrict__ coords, uint32_t n, StridedGeom g,
                                                                 const uint32_t* __restrict__ bits, const uint32_t* __restrict__ rank, uint32_t n_out,
                                                                 uint32_t* __restrict__ nbr, uint32_t* __restrict__ nbr_bwd, MapOut bwd) {
  extern __shared__ __align__(16) uint32_t s_nbr[];  // [kMapBlock * V], then the digit histograms over it
  chain_release();
  chain_wait();
  const uint32_t n0 = blockIdx.x * kMapBlock, nv = min(static_cast<uint32_t>(kMapBlock), n - n0);
  const int t = threadIdx.x;
  uint32_t gray = 0;
  if (nbr_bwd != nullptr) {
    for (int i = t; i < kMapBlock * g.V; i += kMapBlock) s_nbr[i] = kInvalid;
    __syncthreads();
  }
  if (t < nv) {
    const int4 c = __ldg(&coords[n0 + t]);
    if (c.y >= 0 && c.y < g.in[0] && c.z >= 0 && c.z < g.in[1] && c.w >= 0 && c.w < g.in[2])
      for_targets(c, g, [&](int v, uint32_t cell) {
        const uint32_t row = __ldg(&rank[cell >> 5]) + __popc(__ldg(&bits[cell >> 5]) & ((1u << (cell & 31)) - 1u));
        if (row >= n_out) return;
        nbr[size_t(row) * g.V + v] = n0 + t;
        if (nbr_bwd != nullptr) s_nbr[t * g.V + v] = row;
        gray |= 1u << v;
      });
  }
  if (nbr_bwd == nullptr) return;  // uniform
  __syncthreads();
  uint32_t* out = nbr_bwd + size_t(n0) * g.V;
  const uint32_t words = nv * g.V;
  for (uint32_t i = t; i < words; i += kMapBlock) out[i] = s_nbr[i];
  emit_codes(bwd, n0, nv, g.V, gray, s_nbr);
}

// codes, per-block counts and digit histograms of a finished map
__global__ void __launch_bounds__(kMapBlock) map_codes_kernel(const uint32_t* __restrict__ nbr, uint32_t n, int V, MapOut o) {
  extern __shared__ __align__(16) uint32_t s_nbr[];
  __shared__ uint32_t s_count[32];
  chain_release();
  const uint32_t n0 = blockIdx.x * kMapBlock, nv = min(static_cast<uint32_t>(kMapBlock), n - n0);
  const int t = threadIdx.x;
  if (t < 32) s_count[t] = 0;
  chain_wait();
  for (uint32_t i = t; i < nv * V; i += kMapBlock) s_nbr[i] = __ldg(&nbr[size_t(n0) * V + i]);
  __syncthreads();
  const uint32_t gray = tile_codes(s_nbr, s_count, nv, V);
  __syncthreads();
  if (t < V) o.block_counts[size_t(t) * o.nblk + blockIdx.x] = s_count[t];
  emit_codes(o, n0, nv, V, gray, s_nbr);
}

static size_t codes_smem(int V) { return std::max(size_t(kMapBlock) * V, size_t(sort_passes_of(V)) * kSortDigits) * sizeof(uint32_t); }

// ------------------------------------------------------------------ host side
static int strided_geom(const fgb_strided_call* c, StridedGeom* g) {
  if (!c) return FGB_E_NULL;
  if (c->n < 0 || c->n >= (int64_t(1) << 30) || c->b < 0) return FGB_E_SIZE;
  const int in[3] = {c->w, c->h, c->d};
  int64_t V = 1;
  for (int i = 0; i < 3; ++i) {
    if (in[i] <= 0 || c->k[i] <= 0 || c->s[i] <= 0 || c->p[i] < 0 || c->dil[i] <= 0) return FGB_E_SIZE;
    V *= c->k[i];
    if (V > 32) return FGB_E_SIZE;
    const int64_t span = int64_t(in[i]) + 2 * int64_t(c->p[i]) - int64_t(c->dil[i]) * (c->k[i] - 1) - 1;
    g->K[i] = c->k[i], g->S[i] = c->s[i], g->P[i] = c->p[i], g->D[i] = c->dil[i], g->in[i] = in[i];
    g->out[i] = static_cast<int>(std::max<int64_t>(span / c->s[i] + 1, 0));  // as fgb_sparse_out_grid
  }
  g->B = c->b, g->V = static_cast<int>(V);
  return FGB_OK;
}

struct GridMem {
  uint32_t words, ctas;
  size_t base_off, done_off, zero_bytes, rank_off, bytes;
};
// 0 cells, or more than the bits may take (2^31 cells = 256 MB), or a grid so empty that clearing and reading its bits
// would cost more than hashing the few voxels: no bits
static bool grid_mem(const StridedGeom& g, int64_t n, GridMem* m) {
  const double cells = double(g.B) * g.out[0] * g.out[1] * g.out[2];
  if (cells < 1.0 || cells > 2147483648.0 || cells / 32.0 > double(n) * 64.0 + (1 << 20)) return false;
  const uint64_t words = (static_cast<uint64_t>(cells) + 31) / 32;
  m->ctas = static_cast<uint32_t>((words + kRankWords - 1) / kRankWords);
  m->words = m->ctas * kRankWords;
  m->done_off = size_t(m->words) * 4;
  m->zero_bytes = m->done_off + 256;
  m->base_off = m->zero_bytes;
  m->rank_off = m->base_off + align256(int64_t(m->ctas) * 4);
  m->bytes = m->rank_off + size_t(m->words) * 4;
  return true;
}

struct StridedScratch {
  SortLayout sort, sort_bwd;
  size_t words_off, hist_off, hist_bwd_off, look_off, look_bwd_off, zero_bytes, codes_off, codes_bwd_off, buf_off, total;
};
static StridedScratch strided_scratch(int64_t n, int64_t n_out, int V, bool bwd) {
  StridedScratch c{};
  c.sort = sort_layout(n_out);
  c.sort_bwd = sort_layout(n);
  const size_t hist = align256((kSortMaxPasses * kSortDigits + kSortMaxPasses) * 4);
  const int passes = sort_passes_of(V);
  c.words_off = 0;  // [0] scan counter [1] plan counter [2] backward plan counter
  c.hist_off = 256;
  c.hist_bwd_off = c.hist_off + hist;
  c.look_off = c.hist_bwd_off + (bwd ? hist : 0);
  c.look_bwd_off = c.look_off + align256(int64_t(passes) * c.sort.tiles * kSortDigits * 4);
  c.zero_bytes = c.look_bwd_off + (bwd ? align256(int64_t(passes) * c.sort_bwd.tiles * kSortDigits * 4) : 0);
  c.codes_off = c.zero_bytes;
  c.codes_bwd_off = c.codes_off + align256(n_out * 4);
  c.buf_off = c.codes_bwd_off + (bwd ? align256(n * 4) : 0);
  c.total = c.buf_off + std::max(c.sort.buffer_bytes, bwd ? c.sort_bwd.buffer_bytes : size_t(0));
  return c;
}

}  // namespace fgb

extern "C" int64_t fgb_strided_grid_bytes(const fgb_strided_call* c) {
  using namespace fgb;
  StridedGeom g;
  const int rc = strided_geom(c, &g);
  if (rc != FGB_OK) return rc;
  GridMem m;
  return c->n > 0 && grid_mem(g, c->n, &m) ? static_cast<int64_t>(m.bytes) : 0;
}

extern "C" int fgb_strided_mark(const fgb_strided_call* c, void* stream) {
  using namespace fgb;
  StridedGeom g;
  GridMem m;
  const int rc = strided_geom(c, &g);
  if (rc != FGB_OK) return rc;
  if (c->n == 0 || !grid_mem(g, c->n, &m)) return FGB_E_SIZE;
  if (!c->coords || !c->grid_mem) return FGB_E_NULL;
  if ((reinterpret_cast<uintptr_t>(c->coords) & 15) || (reinterpret_cast<uintptr_t>(c->grid_mem) & 255)) return FGB_E_ALIGN;
  if (c->grid_bytes < static_cast<int64_t>(m.bytes)) return FGB_E_WORKSPACE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  char* mem = static_cast<char*>(c->grid_mem);
  uint32_t* bits = reinterpret_cast<uint32_t*>(mem);
  uint32_t* done = reinterpret_cast<uint32_t*>(mem + m.done_off);  // [0] count of finished CTAs [1] rows outside the grid's batches
  LaunchErrors chain;
  chain.add(cudaMemsetAsync(mem, 0, m.zero_bytes, s));
  chain.add(launch_chained(mark_cells_kernel, dim3(static_cast<unsigned>(ceil_div(c->n, 256))), dim3(256), 0, s,
                           reinterpret_cast<const int4*>(c->coords), static_cast<uint32_t>(c->n), g, bits, done + 1));
  chain.add(launch_chained(count_cells_kernel, dim3(m.ctas), dim3(kRankThreads), 0, s, static_cast<const uint32_t*>(bits),
                           reinterpret_cast<uint32_t*>(mem + m.base_off), done, static_cast<const uint32_t*>(done + 1), c->host_words, c->host_seq));
  return chain.first != cudaSuccess ? cuda_status(chain.first) : launch_status();
}

extern "C" int64_t fgb_strided_build_bytes(const fgb_strided_call* c) {
  using namespace fgb;
  StridedGeom g;
  const int rc = strided_geom(c, &g);
  if (rc != FGB_OK) return rc;
  if (c->n_out < 0 || c->n_out >= (int64_t(1) << 30)) return FGB_E_SIZE;
  return static_cast<int64_t>(strided_scratch(c->n, c->n_out, g.V, c->neighbor_map_bwd != nullptr).total);
}

extern "C" int fgb_strided_build(const fgb_strided_call* c, void* stream) {
  using namespace fgb;
  StridedGeom g;
  GridMem m;
  int rc = strided_geom(c, &g);
  if (rc != FGB_OK) return rc;
  if (c->n == 0 || !grid_mem(g, c->n, &m) || c->n_out <= 0 || c->n_out >= (int64_t(1) << 30)) return FGB_E_SIZE;
  if (!c->coords || !c->grid_mem || !c->out_coords) return FGB_E_NULL;
  if ((reinterpret_cast<uintptr_t>(c->coords) | reinterpret_cast<uintptr_t>(c->out_coords)) & 15) return FGB_E_ALIGN;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  char* gm = static_cast<char*>(c->grid_mem);
  const uint32_t* bits = reinterpret_cast<const uint32_t*>(gm);
  uint32_t* rank = reinterpret_cast<uint32_t*>(gm + m.rank_off);
  const uint32_t n = static_cast<uint32_t>(c->n), n_out = static_cast<uint32_t>(c->n_out);
  const int V = g.V;
  LaunchErrors chain;
  if (c->neighbor_map == nullptr) {  // coordinates only
    chain.add(launch_chained(emit_cells_kernel, dim3(m.ctas), dim3(kRankThreads), 0, s, bits,
                             reinterpret_cast<const uint32_t*>(gm + m.base_off), g, n_out, rank, reinterpret_cast<int4*>(c->out_coords)));
    return chain.first != cudaSuccess ? cuda_status(chain.first) : launch_status();
  }
  const bool with_bwd = c->neighbor_map_bwd != nullptr;
  if (!c->scratch || !c->gray_code || !c->sorted_idx || !c->tile_masks || !c->block_order || !c->block_offsets || !c->meta) return FGB_E_NULL;
  if (with_bwd && (!c->gray_code_bwd || !c->sorted_idx_bwd || !c->tile_masks_bwd || !c->block_order_bwd)) return FGB_E_NULL;
  if (reinterpret_cast<uintptr_t>(c->scratch) & 255) return FGB_E_ALIGN;
  const StridedScratch L = strided_scratch(c->n, c->n_out, V, with_bwd);
  if (c->scratch_bytes < static_cast<int64_t>(L.total)) return FGB_E_WORKSPACE;
  char* mem = static_cast<char*>(c->scratch);
  uint32_t* words = reinterpret_cast<uint32_t*>(mem + L.words_off);
  uint32_t* hist = reinterpret_cast<uint32_t*>(mem + L.hist_off);
  uint32_t* hist_bwd = reinterpret_cast<uint32_t*>(mem + L.hist_bwd_off);
  int32_t* codes = reinterpret_cast<int32_t*>(mem + L.codes_off);
  int32_t* codes_bwd = reinterpret_cast<int32_t*>(mem + L.codes_bwd_off);
  // few rows on both sides: no histograms or look-back words to clear, one launch for all that follows from the codes
  const bool small = c->n <= kSmallRows && c->n_out <= kSmallRows;
  if (!small) chain.add(cudaMemsetAsync(mem, 0, L.zero_bytes, s));
  chain.add(cudaMemsetAsync(c->neighbor_map, 0xFF, size_t(n_out) * V * 4, s));
  chain.add(launch_chained(emit_cells_kernel, dim3(m.ctas), dim3(kRankThreads), 0, s, bits,
                           reinterpret_cast<const uint32_t*>(gm + m.base_off), g, n_out, rank, reinterpret_cast<int4*>(c->out_coords)));
  const MapOut ob{c->neighbor_map_bwd, c->gray_code_bwd, codes_bwd, nullptr, small ? nullptr : hist_bwd, 0};
  chain.add(launch_chained(strided_maps_kernel, dim3(static_cast<unsigned>(ceil_div(c->n, kMapBlock))), dim3(kMapBlock), with_bwd ? codes_smem(V) : 0, s,
                           reinterpret_cast<const int4*>(c->coords), n, g, bits, static_cast<const uint32_t*>(rank), n_out, c->neighbor_map,
                           c->neighbor_map_bwd, ob));
  const uint32_t nblk = static_cast<uint32_t>(ceil_div(c->n_out, kMapBlock));
  const MapOut of{c->neighbor_map, c->gray_code, codes, c->block_offsets, small ? nullptr : hist, nblk};
  chain.add(launch_chained(map_codes_kernel, dim3(nblk), dim3(kMapBlock), codes_smem(V), s, static_cast<const uint32_t*>(c->neighbor_map), n_out, V, of));
  if (small) {
    PlanJob jf{codes, c->gray_code, n_out, V, c->sorted_idx, c->tile_masks, c->block_order, c->block_offsets, c->meta, {}};
    jf.fin.host_words = c->host_words, jf.fin.host_seq = c->host_seq;
    const PlanJob jb{codes_bwd, c->gray_code_bwd, n, V, c->sorted_idx_bwd, c->tile_masks_bwd, c->block_order_bwd, nullptr, nullptr, {}};
    if (chain.first == cudaSuccess) chain.add(launch_small_plan(jf, with_bwd ? &jb : nullptr, s));
    return chain.first != cudaSuccess ? cuda_status(chain.first) : launch_status();
  }
  ScanFinish fin{words, nullptr, nullptr, c->host_words, c->host_seq};
  chain.add(launch_block_scan(c->block_offsets, nblk, V, c->meta, fin, HistJob{}, s));
  if (chain.first == cudaSuccess)
    chain.add(launch_sort_passes(codes, c->n_out, V, c->sorted_idx, mem + L.buf_off, L.sort, hist, reinterpret_cast<uint32_t*>(mem + L.look_off), c->status, s));
  if (chain.first == cudaSuccess) chain.add(launch_tile_plan(c->gray_code, c->sorted_idx, c->n_out, c->tile_masks, c->block_order, words + 1, s));
  if (chain.first == cudaSuccess && with_bwd) {
    chain.add(launch_sort_passes(codes_bwd, c->n, V, c->sorted_idx_bwd, mem + L.buf_off, L.sort_bwd, hist_bwd,
                                 reinterpret_cast<uint32_t*>(mem + L.look_bwd_off), c->status, s));
    chain.add(launch_tile_plan(c->gray_code_bwd, c->sorted_idx_bwd, c->n, c->tile_masks_bwd, c->block_order_bwd, words + 2, s));
  }
  return chain.first != cudaSuccess ? cuda_status(chain.first) : launch_status();
}
