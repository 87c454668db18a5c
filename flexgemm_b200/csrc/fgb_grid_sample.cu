// Generic use of the coordinate hash table and the sparse grid sample built on it:
// insert / lookup of (b, x, y, z) rows, the nearest and trilinear neighbour maps of
// arbitrary query points, and the gather (forward) / scatter-add (backward) of
// features through such a map.  All of it is HBM-bound byte and index work.
#include <algorithm>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "fgb_common.cuh"
#include "fgb_hash.cuh"

namespace fgb {

__global__ void __launch_bounds__(256) fill_words_kernel(uint32_t* __restrict__ words, size_t count, uint32_t value) {
  for (size_t i = blockIdx.x * size_t(256) + threadIdx.x; i < count; i += size_t(gridDim.x) * 256) words[i] = value;
}

template <int kKeyBits>
__global__ void __launch_bounds__(256) hash_lookup_3d_kernel(const int4* __restrict__ query, uint32_t m, Grid3 g, void* table_mem,
                                                            uint32_t slots, uint32_t* __restrict__ out) {
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;
  if (i >= m) return;
  const int4 c = __ldg(&query[i]);
  uint32_t val = kInvalid;
  if (c.x >= 0 && c.y >= 0 && c.y < g.W && c.z >= 0 && c.z < g.H && c.w >= 0 && c.w < g.D)
    val = make_table<kKeyBits>(table_mem, slots).find(g.template key<kKeyBits>(c.x, c.y, c.z, c.w));
  out[i] = val;
}

// neighbor[q] = row of the voxel that contains query point q (coordinates truncated towards zero), or 0xffffffff
template <int kKeyBits>
__global__ void __launch_bounds__(256) nearest_map_kernel(const float* __restrict__ query, uint32_t B, uint32_t L, Grid3 g,
                                                         void* table_mem, uint32_t slots, uint32_t* __restrict__ neighbor) {
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;
  if (i >= B * L) return;
  const int b = static_cast<int>(i / L);
  const int x = static_cast<int>(__ldg(&query[3 * size_t(i)])), y = static_cast<int>(__ldg(&query[3 * size_t(i) + 1])),
            z = static_cast<int>(__ldg(&query[3 * size_t(i) + 2]));
  uint32_t val = kInvalid;
  if (x >= 0 && x < g.W && y >= 0 && y < g.H && z >= 0 && z < g.D)
    val = make_table<kKeyBits>(table_mem, slots).find(g.template key<kKeyBits>(b, x, y, z));
  neighbor[i] = val;
}

// The eight voxels around query point q (corner i: x + (i & 1), y + ((i >> 1) & 1), z + ((i >> 2) & 1) from the
// base floor(q - 0.5)) and their trilinear weights, normalised over the voxels that exist.
template <int kKeyBits>
__global__ void __launch_bounds__(256) trilinear_map_kernel(const float* __restrict__ query, uint32_t B, uint32_t L, Grid3 g,
                                                           void* table_mem, uint32_t slots, uint32_t* __restrict__ neighbor,
                                                           float* __restrict__ weight) {
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;
  if (i >= B * L) return;
  const int b = static_cast<int>(i / L);
  const float qx = __ldg(&query[3 * size_t(i)]), qy = __ldg(&query[3 * size_t(i) + 1]), qz = __ldg(&query[3 * size_t(i) + 2]);
  const int bx = static_cast<int>(floorf(qx - 0.5f)), by = static_cast<int>(floorf(qy - 0.5f)), bz = static_cast<int>(floorf(qz - 0.5f));
  const auto table = make_table<kKeyBits>(table_mem, slots);
  uint32_t nb[8];
  float w[8];
  float sum = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int x = bx + (k & 1), y = by + ((k >> 1) & 1), z = bz + ((k >> 2) & 1);
    nb[k] = kInvalid;
    w[k] = 0.f;
    if (x >= 0 && x < g.W && y >= 0 && y < g.H && z >= 0 && z < g.D) {
      const uint32_t row = table.find(g.template key<kKeyBits>(b, x, y, z));
      if (row != kInvalid) {
        nb[k] = row;
        w[k] = (1.f - fabsf(qx - x - 0.5f)) * (1.f - fabsf(qy - y - 0.5f)) * (1.f - fabsf(qz - z - 0.5f));
        sum += w[k];
      }
    }
  }
  const float inv = 1.f / fmaxf(sum, 1e-12f);
  uint4* no = reinterpret_cast<uint4*>(neighbor + 8 * size_t(i));
  float4* wo = reinterpret_cast<float4*>(weight + 8 * size_t(i));
  no[0] = make_uint4(nb[0], nb[1], nb[2], nb[3]);
  no[1] = make_uint4(nb[4], nb[5], nb[6], nb[7]);
  wo[0] = make_float4(w[0] * inv, w[1] * inv, w[2] * inv, w[3] * inv);
  wo[1] = make_float4(w[4] * inv, w[5] * inv, w[6] * inv, w[7] * inv);
}

template <typename T>
__device__ __forceinline__ void load4(const T* p, float (&v)[4]);
template <>
__device__ __forceinline__ void load4<float>(const float* p, float (&v)[4]) {
  const float4 t = __ldg(reinterpret_cast<const float4*>(p));
  v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
}
template <>
__device__ __forceinline__ void load4<__half>(const __half* p, float (&v)[4]) {
  const uint2 t = __ldg(reinterpret_cast<const uint2*>(p));
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&t.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&t.y));
  v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
}
template <>
__device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[4]) {
  const uint2 t = __ldg(reinterpret_cast<const uint2*>(p));
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t.x)),
               b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t.y));
  v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
}
template <typename T>
__device__ __forceinline__ void store4(T* p, const float (&v)[4]);
template <>
__device__ __forceinline__ void store4<float>(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
template <>
__device__ __forceinline__ void store4<__half>(__half* p, const float (&v)[4]) {
  const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
template <>
__device__ __forceinline__ void store4<__nv_bfloat16>(__nv_bfloat16* p, const float (&v)[4]) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

// out[m, :] = sum_k weight[m, k] * feats[indices[m, k], :] over the valid entries (weight == null: every weight 1).
// A thread owns four consecutive channels of one output row; the rows of a warp are consecutive, so the index and
// weight loads coalesce and every feature load is 8 or 16 bytes of a gathered row.
template <typename T>
__global__ void __launch_bounds__(256) weighted_gather_kernel(const T* __restrict__ feats, const uint32_t* __restrict__ indices,
                                                             const float* __restrict__ weight, T* __restrict__ out, int64_t M, int C,
                                                             int V) {
  const int c4 = C / 4;
  const int64_t e = blockIdx.x * int64_t(256) + threadIdx.x;
  if (e >= M * c4) return;
  const int64_t m = e / c4;
  const int c = static_cast<int>(e - m * c4) * 4;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int k = 0; k < V; ++k) {
    const uint32_t row = __ldg(&indices[m * V + k]);
    if (row == kInvalid) continue;
    const float w = weight != nullptr ? __ldg(&weight[m * V + k]) : 1.f;
    float v[4];
    load4<T>(feats + size_t(row) * C + c, v);
    acc[0] += w * v[0], acc[1] += w * v[1], acc[2] += w * v[2], acc[3] += w * v[3];
  }
  store4<T>(out + m * C + c, acc);
}

// grad_feats_f32[indices[m, k], :] += weight[m, k] * grad_out[m, :]   (fp32 atomics; the caller zeroes the buffer)
template <typename T>
__global__ void __launch_bounds__(256) weighted_scatter_kernel(const T* __restrict__ grad_out, const uint32_t* __restrict__ indices,
                                                              const float* __restrict__ weight, float* __restrict__ grad_feats, int64_t M,
                                                              int C, int V) {
  const int c4 = C / 4;
  const int64_t e = blockIdx.x * int64_t(256) + threadIdx.x;
  if (e >= M * c4) return;
  const int64_t m = e / c4;
  const int c = static_cast<int>(e - m * c4) * 4;
  float g[4];
  load4<T>(grad_out + m * C + c, g);
  for (int k = 0; k < V; ++k) {
    const uint32_t row = __ldg(&indices[m * V + k]);
    if (row == kInvalid) continue;
    const float w = weight != nullptr ? __ldg(&weight[m * V + k]) : 1.f;
    float* dst = grad_feats + size_t(row) * C + c;
    atomicAdd(dst + 0, w * g[0]);
    atomicAdd(dst + 1, w * g[1]);
    atomicAdd(dst + 2, w * g[2]);
    atomicAdd(dst + 3, w * g[3]);
  }
}

// ------------------------------------------------------------------ fused sample
// Points around one voxel grid, features blended in one kernel.  A warp takes four points at a time: its 32 lanes look up
// the 4 x 8 corners at once, and the map goes to memory only where a backward pass will want it; then the points' feature
// rows are gathered with 16-byte loads.  Narrow rows share the warp: kGroup lanes per point.
// Bound at 10^6 points, C = 256 fp16, RES = 256: the rows' way out of L2 (1.6 GB of them at random places of an 84 MB
// matrix, and the 0.5 GB of results): 375 us against 84 + 620 us for a map kernel and a gather that walked the eight
// corners one after the other.  Occupancies from 32 to 48 warps, two to four rows in flight and lookups ahead or not
// all gave 367 to 397 us.
// kNearest: one corner, the voxel that contains the point; the four points of a warp are looked up by four lanes.
template <typename T, int kVec>
struct Pack;  // kVec consecutive elements as one load
template <typename T>
struct Pack<T, 8> { using Raw = uint4; };
template <typename T>
struct Pack<T, 4> { using Raw = typename std::conditional<sizeof(T) == 4, uint4, uint2>::type; };
template <typename T, int kVec>
__device__ __forceinline__ void fma_pack(float (&acc)[kVec], const typename Pack<T, kVec>::Raw& raw, float w) {
  const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
  for (int i = 0; i < kVec; ++i) acc[i] += w * static_cast<float>(e[i]);
}
template <typename T, int kVec>
__device__ __forceinline__ typename Pack<T, kVec>::Raw round_pack(const float (&acc)[kVec]) {
  typename Pack<T, kVec>::Raw raw;
  T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
  for (int i = 0; i < kVec; ++i) e[i] = static_cast<T>(acc[i]);
  return raw;
}

constexpr int kSamplePoints = 4;  // points of a warp

template <typename T, int kVec, int kKeyBits, bool kNearest, int kGroup>
__global__ void __launch_bounds__(256, 4) sample_kernel(const T* __restrict__ feats, const float* __restrict__ query, uint32_t points, uint32_t L,
                                                     Grid3 g, void* table_mem, uint32_t slots, int C, T* __restrict__ out,
                                                     uint32_t* __restrict__ neighbor, float* __restrict__ weight) {
  using Raw = typename Pack<T, kVec>::Raw;
  constexpr int kCorners = kNearest ? 1 : 8;
  constexpr int kAtOnce = 32 / kGroup;  // points gathered side by side
  chain_release();
  chain_wait();
  const int lane = threadIdx.x & 31;
  const auto table = make_table<kKeyBits>(table_mem, slots);
  const bool looks = lane < kSamplePoints * kCorners;
  const int k = lane % kCorners;
  // A warp walks over groups of four points.  The next group's home slots and the query points of the one after are
  // loaded before the current group's rows, so a step waits for one latency, not for three in a row.
  auto load_query = [&](uint32_t group, float (&q)[3]) {
    const uint64_t i = uint64_t(group) * kSamplePoints + lane / kCorners;
    const bool ok = looks && i < points;
#pragma unroll
    for (int d = 0; d < 3; ++d) q[d] = ok ? __ldg(&query[3 * i + d]) : -4.f;  // -4: outside every grid
  };
  struct Probe {
    uint64_t key;
    unsigned long long word;  // the home slot
    float w;
    bool inside;
  };
  auto start_probe = [&](uint32_t group, const float (&q)[3]) {
    Probe pr;
    const uint32_t i = group * kSamplePoints + lane / kCorners;
    int x, y, z;
    if constexpr (kNearest) {
      x = static_cast<int>(q[0]), y = static_cast<int>(q[1]), z = static_cast<int>(q[2]);
      pr.w = 1.f;
    } else {
      x = static_cast<int>(floorf(q[0] - 0.5f)) + (k & 1);
      y = static_cast<int>(floorf(q[1] - 0.5f)) + ((k >> 1) & 1);
      z = static_cast<int>(floorf(q[2] - 0.5f)) + ((k >> 2) & 1);
      pr.w = (1.f - fabsf(q[0] - x - 0.5f)) * (1.f - fabsf(q[1] - y - 0.5f)) * (1.f - fabsf(q[2] - z - 0.5f));
    }
    pr.inside = x >= 0 && x < g.W && y >= 0 && y < g.H && z >= 0 && z < g.D;
    pr.key = 0, pr.word = 0;
    if (pr.inside) {
      pr.key = g.template key<kKeyBits>(static_cast<int>(i / L), x, y, z);
      pr.word = table.start(pr.key);
    }
    return pr;
  };
  const uint32_t groups = (points + kSamplePoints - 1) / kSamplePoints, stride = gridDim.x * 8u;
  uint32_t group = blockIdx.x * 8u + (threadIdx.x >> 5);
  float ahead[3];
  load_query(group, ahead);
  Probe next = start_probe(group, ahead);
  load_query(group + stride, ahead);
  const int nv = C / kVec;
#pragma unroll 1
  for (; group < groups; group += stride) {
    const uint32_t p0 = group * kSamplePoints;
    const uint32_t nb = next.inside ? table.finish(next.key, next.word) : kInvalid;
    float w = nb != kInvalid ? next.w : 0.f;
    next = start_probe(group + stride, ahead);
    load_query(group + 2 * stride, ahead);
    if constexpr (!kNearest) {
      // corner order of the sum as in the map kernel: the weights of a point are the same bits either way
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) sum += __shfl_sync(0xffffffffu, w, (lane & 24) + j);
      w *= 1.f / fmaxf(sum, 1e-12f);
    }
    if (neighbor != nullptr && looks && p0 + lane / kCorners < points) {
      neighbor[size_t(p0) * kCorners + lane] = nb;
      if constexpr (!kNearest) weight[size_t(p0) * kCorners + lane] = w;
    }
    // Only corners that exist are walked (about three of eight near a surface), kBatch rows in flight per step: walking all
    // eight under predicates took twice the instructions and, at 80 registers, ran with a third of the warps.
    constexpr int kBatch = kNearest ? 1 : 4;
    const unsigned valid = __ballot_sync(0xffffffffu, nb != kInvalid);
#pragma unroll 1
    for (int i = 0; i < kSamplePoints; i += kAtOnce < kSamplePoints ? kAtOnce : kSamplePoints) {
      const int local = (i + (kAtOnce == 1 ? 0 : lane / kGroup)) % kSamplePoints;
      const bool mine = p0 + local < points;
      const unsigned corners = (valid >> (local * kCorners)) & ((1u << kCorners) - 1u);
      const int steps = kGroup == 32 ? __popc(corners) : __reduce_max_sync(0xffffffffu, __popc(corners));
      for (int c0 = 0; c0 < nv; c0 += kGroup) {
        const int c = c0 + lane % kGroup;
        const bool col = mine && c < nv;
        float acc[kVec];
#pragma unroll
        for (int j = 0; j < kVec; ++j) acc[j] = 0.f;
        unsigned left = corners;
        for (int t = 0; t < steps; t += kBatch) {
          Raw raw[kBatch];
          float ws[kBatch];
          bool ok[kBatch];
#pragma unroll
          for (int u = 0; u < kBatch; ++u) {
            ok[u] = left != 0u;
            const int src = local * kCorners + (ok[u] ? __ffs(left) - 1 : 0);
            left &= left - 1u;
            const uint32_t row = __shfl_sync(0xffffffffu, nb, src);
            ws[u] = __shfl_sync(0xffffffffu, w, src);
            if (ok[u] && col) raw[u] = __ldg(reinterpret_cast<const Raw*>(feats + size_t(row) * C) + c);
          }
#pragma unroll
          for (int u = 0; u < kBatch; ++u)
            if (ok[u]) fma_pack<T, kVec>(acc, raw[u], ws[u]);
        }
        if (col) __stcs(reinterpret_cast<Raw*>(out + size_t(p0 + local) * C) + c, round_pack<T, kVec>(acc));
      }
    }
  }
}

// ------------------------------------------------------------------ gradient w.r.t. the features
// grad_feats[r, :] = sum over the (point, corner) entries e with indices[e] == r of weight[e] * grad_out[point(e), :]
//
// As a gather: the entries are first grouped by voxel (count, place the groups, fill), then one warp per voxel reads the
// gradient rows of its entries with 16-byte loads, sums in fp32 registers and writes the row once in the feature type.
// Against fp32 atomics into a buffer that is zeroed before and converted after (10^6 points, C = 256 fp16 on the RES=256
// shell: 2.05 ms + 28 + 35 us, all of it atomic traffic of 4 bytes per channel and corner) the gradient rows cross L2
// as 2-byte values, and consecutive voxels share the points between them, so a row comes from HBM once.
__global__ void __launch_bounds__(256) group_count_kernel(const uint32_t* __restrict__ indices, uint32_t entries, uint32_t* __restrict__ count) {
  chain_release();
  chain_wait();
  for (uint64_t e = blockIdx.x * uint64_t(256) + threadIdx.x; e < entries; e += uint64_t(gridDim.x) * 256) {
    const uint32_t row = __ldg(&indices[e]);
    if (row != kInvalid) atomicAdd(&count[row], 1u);
  }
}
// Lists longer than `limit` entries are cut into pieces that warps take on their own, so that a voxel that is hit far more
// often than the others (queries padded with one repeated point, a cluster of them) does not leave the sum to one warp.
struct CutLists {
  uint32_t limit, piece;  // limit = ~0: nothing is cut
  uint32_t* total;        // zeroed: pieces listed
  uint2* pieces;          // (row, first piece of the row)
  uint32_t* done;         // pieces of the row that are summed, at the row's first piece
  float* slab;            // [pieces, C] their sums
};
// At most 1024: the warp that ends last adds a row's parts up.
__host__ __device__ __forceinline__ uint32_t pieces_of(uint32_t len, uint32_t piece) { return min((len - 1u) / piece + 1u, 1024u); }

// start[r] = where the entries of voxel r go (the fill moves it on to their end).  The groups of 1024 consecutive voxels
// stand together, in order; such blocks take their places as they come (one atomic each), which no result depends on.
__global__ void __launch_bounds__(1024) group_place_kernel(const uint32_t* __restrict__ count, uint32_t n, uint32_t* __restrict__ start,
                                                           uint32_t* __restrict__ total, CutLists cut) {
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_base;
  chain_release();
  chain_wait();
  const uint32_t i = blockIdx.x * 1024u + threadIdx.x;
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const uint32_t x = i < n ? count[i] : 0u;
  uint32_t inc = x;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += y;
  }
  if (lane == 31) s_warp[wi] = inc;
  __syncthreads();
  if (wi == 0) {
    uint32_t ws = s_warp[lane];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, ws, d);
      if (lane >= d) ws += y;
    }
    s_warp[lane] = ws;
    if (lane == 31) s_base = atomicAdd(total, ws);
  }
  __syncthreads();
  if (i < n) start[i] = s_base + (wi ? s_warp[wi - 1] : 0u) + inc - x;
  const uint32_t k = x > cut.limit ? pieces_of(x, cut.piece) : 0u;
  uint32_t first = 0;
  if (k != 0u) {
    first = atomicAdd(cut.total, k);
    cut.done[first] = 0u;
  }
  for (unsigned todo = __ballot_sync(0xffffffffu, k != 0u); todo != 0u; todo &= todo - 1u) {
    const int l = __ffs(todo) - 1;
    const uint32_t row = __shfl_sync(0xffffffffu, i, l), at = __shfl_sync(0xffffffffu, first, l), many = __shfl_sync(0xffffffffu, k, l);
    for (uint32_t j = lane; j < many; j += 32u) cut.pieces[at + j] = make_uint2(row, at);
  }
}
__global__ void __launch_bounds__(256) group_fill_kernel(const uint32_t* __restrict__ indices, const float* __restrict__ weight, uint32_t entries,
                                                         int V, uint32_t* __restrict__ start, uint2* __restrict__ grouped) {
  chain_release();
  chain_wait();
  for (uint64_t e = blockIdx.x * uint64_t(256) + threadIdx.x; e < entries; e += uint64_t(gridDim.x) * 256) {
    const uint32_t row = __ldg(&indices[e]);
    if (row == kInvalid) continue;
    const float w = weight != nullptr ? __ldg(&weight[e]) : 1.f;
    grouped[atomicAdd(&start[row], 1u)] = make_uint2(static_cast<uint32_t>(e / V), __float_as_uint(w));
  }
}
// Sum over the entries base, base + step, ... (32 at a time) of a list, for the row's packs c0 + lane % kGroup: the lane
// groups of the warp take the entries in turn, and every lane ends with the whole sum.  Whole warps call it.
template <typename T, int kVec, int kGroup>
__device__ __forceinline__ void warp_sum(const T* __restrict__ grad_out, const uint2* list, uint32_t base, uint32_t step, uint32_t len, int C, int c,
                                         float (&acc)[kVec]) {
  using Raw = typename Pack<T, kVec>::Raw;
  constexpr int kSide = 32 / kGroup;
  const int lane = threadIdx.x & 31, side = lane / kGroup;
  const bool col = c < C / kVec;
#pragma unroll
  for (int i = 0; i < kVec; ++i) acc[i] = 0.f;
  for (; base < len; base += step) {
    const uint32_t here = min(32u, len - base);
    const uint2 e = lane < here ? __ldg(&list[base + lane]) : make_uint2(0, 0);
#pragma unroll 4
    for (uint32_t j0 = 0; j0 < here; j0 += kSide) {
      const uint32_t j = j0 + side;
      const uint32_t m = __shfl_sync(0xffffffffu, e.x, j & 31);
      const float w = __uint_as_float(__shfl_sync(0xffffffffu, e.y, j & 31));
      if (j < here && col) fma_pack<T, kVec>(acc, __ldg(reinterpret_cast<const Raw*>(grad_out + size_t(m) * C) + c), w);
    }
  }
#pragma unroll
  for (int d = kGroup; d < 32; d <<= 1)
#pragma unroll
    for (int i = 0; i < kVec; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], d);
}

// One piece of a list that is cut, by one warp; the warp that ends a row's last piece adds the parts up, in their order.
template <typename T, int kVec, int kGroup>
__device__ __forceinline__ void sum_piece(const T* __restrict__ grad_out, const uint2* __restrict__ grouped, const uint32_t* __restrict__ end,
                                          const uint32_t* __restrict__ count, int C, const CutLists& cut, uint32_t p, T* __restrict__ grad_feats) {
  const int lane = threadIdx.x & 31, nv = C / kVec;
  const uint2 d = __ldg(&cut.pieces[p]);
  const uint32_t len = __ldg(&count[d.x]), many = pieces_of(len, cut.piece), j = p - d.y;
  const uint32_t from = static_cast<uint32_t>(uint64_t(len) * j / many), to = static_cast<uint32_t>(uint64_t(len) * (j + 1u) / many);
  const uint2* list = grouped + (__ldg(&end[d.x]) - len);
  float acc[kVec];
  for (int c0 = 0; c0 < nv; c0 += kGroup) {
    const int c = c0 + lane % kGroup;
    warp_sum<T, kVec, kGroup>(grad_out, list, from, 32u, to, C, c, acc);
    if (lane < kGroup && c < nv)
#pragma unroll
      for (int i = 0; i < kVec; ++i) __stcg(&cut.slab[size_t(p) * C + c * kVec + i], acc[i]);
  }
  __threadfence();
  __syncwarp();
  uint32_t before = 0;
  if (lane == 0) before = atomicAdd(&cut.done[d.y], 1u);
  if (__shfl_sync(0xffffffffu, before, 0) != many - 1u) return;
  __threadfence();
  const float4* parts = reinterpret_cast<const float4*>(cut.slab + size_t(d.y) * C);
  for (int c = lane; c < C / 4; c += 32) {
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (uint32_t q = 0; q < many; ++q) {
      const float4 x = __ldcg(&parts[size_t(q) * (C / 4) + c]);
      sum[0] += x.x, sum[1] += x.y, sum[2] += x.z, sum[3] += x.w;
    }
    reinterpret_cast<typename Pack<T, 4>::Raw*>(grad_feats + size_t(d.x) * C)[c] = round_pack<T, 4>(sum);
  }
}

// kGroup lanes cover a voxel's row (or 32 packs of it at a time).  kWarps = 0: every group has a voxel of its own, 32 /
// kGroup of them per warp -- with narrow rows and few entries per voxel a warp per voxel spends its life on three
// dependent loads (RES=467, C=16, 2.4 entries per voxel: most of 275 us).  kWarps = 1: a warp per voxel, its groups take
// the entries in turn.  kWarps = 8: the warps of a CTA share a voxel, where voxels have many entries.  The first
// `piece_ctas` CTAs take the pieces of the lists that are cut.
// Cut lists, 10^6 points on 165 k voxels, us without and with: every tenth point the same one, C = 64 fp16 14256 -> 470,
// C = 256 50852 -> 905; all of them the same, C = 64 166387 -> 2484; none repeated 383 -> 381 and 843 -> 840 (RES=256
// shell, forward and backward, C = 16 to 512: 0.1 to 0.4 % more).  The register limits keep the walkers at the occupancy
// that they have without the pieces' code: at 6 CTAs per SM instead of 8 the same passes took 4 to 6 % longer.
template <typename T, int kVec, int kWarps, int kGroup>
__global__ void __launch_bounds__(256, kWarps == 8 ? 5 : kWarps == 0 && sizeof(T) == 2 && kVec == 8 ? 6 : 8) group_sum_kernel(const T* __restrict__ grad_out, const uint2* __restrict__ grouped,
                                                        const uint32_t* __restrict__ end, const uint32_t* __restrict__ count, uint32_t n, int C,
                                                        T* __restrict__ grad_feats, CutLists cut, uint32_t piece_ctas) {
  using Raw = typename Pack<T, kVec>::Raw;
  constexpr int kSide = 32 / kGroup;
  __shared__ float s_acc[kWarps > 1 ? kWarps : 1][kWarps > 1 ? 32 * kVec : 1];
  chain_release();
  chain_wait();
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const int nv = C / kVec;
  const int side = lane / kGroup;
  if (blockIdx.x < piece_ctas) {
    const uint32_t total = *cut.total;
    for (uint32_t p = blockIdx.x * 8u + wi; p < total; p += piece_ctas * 8u)
      sum_piece<T, kVec, kGroup>(grad_out, grouped, end, count, C, cut, p, grad_feats);
    return;
  }
  const uint32_t block = blockIdx.x - piece_ctas;
  if constexpr (kWarps == 0) {
    const uint32_t row = (block * 8u + wi) * kSide + side;
    if (row >= n) return;
    const uint32_t len = __ldg(&count[row]);
    if (len > cut.limit) return;
    const uint2* list = grouped + (len ? __ldg(&end[row]) - len : 0u);
    for (int c = lane % kGroup; c < nv; c += kGroup) {
      float acc[kVec];
#pragma unroll
      for (int i = 0; i < kVec; ++i) acc[i] = 0.f;
      uint32_t j = 0;
      for (; j + 4 <= len; j += 4) {
        uint2 e[4];
        Raw raw[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) e[u] = __ldg(&list[j + u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) raw[u] = __ldg(reinterpret_cast<const Raw*>(grad_out + size_t(e[u].x) * C) + c);
#pragma unroll
        for (int u = 0; u < 4; ++u) fma_pack<T, kVec>(acc, raw[u], __uint_as_float(e[u].y));
      }
      for (; j < len; ++j) {
        const uint2 e = __ldg(&list[j]);
        fma_pack<T, kVec>(acc, __ldg(reinterpret_cast<const Raw*>(grad_out + size_t(e.x) * C) + c), __uint_as_float(e.y));
      }
      reinterpret_cast<Raw*>(grad_feats + size_t(row) * C)[c] = round_pack<T, kVec>(acc);
    }
  } else {
    const uint32_t row = kWarps > 1 ? block : block * 8u + wi;
    if (row >= n) return;  // whole warps; with kWarps > 1 whole CTAs
    const uint32_t len = __ldg(&count[row]);
    if (len > cut.limit) return;
    const uint2* list = grouped + (len ? __ldg(&end[row]) - len : 0u);
    const int share = kWarps > 1 ? wi : 0;
    for (int c0 = 0; c0 < nv; c0 += kGroup) {
      const int c = c0 + lane % kGroup;
      float acc[kVec];
      warp_sum<T, kVec, kGroup>(grad_out, list, share * 32u, kWarps * 32u, len, C, c, acc);
      if constexpr (kWarps > 1) {
#pragma unroll
        for (int i = 0; i < kVec; ++i) s_acc[wi][lane * kVec + i] = acc[i];
        __syncthreads();
        if (wi == 0) {
#pragma unroll
          for (int i = 0; i < kVec; ++i) {
            acc[i] = 0.f;
#pragma unroll
            for (int k = 0; k < kWarps; ++k) acc[i] += s_acc[k][lane * kVec + i];
          }
        }
        __syncthreads();
      }
      if ((kWarps == 1 || wi == 0) && side == 0 && c < nv) reinterpret_cast<Raw*>(grad_feats + size_t(row) * C)[c] = round_pack<T, kVec>(acc);
    }
  }
}

// lanes for a row of nv packs: the next power of two, 8 .. 32
static int group_lanes(int nv) { return nv <= 8 ? 8 : nv <= 16 ? 16 : 32; }

template <typename T, int kVec, int kKeyBits, bool kNearest>
static cudaError_t launch_sample(const void* feats, const float* query, uint32_t points, uint32_t L, Grid3 g, void* table, uint32_t slots, int C,
                                 void* out, uint32_t* neighbor, float* weight, cudaStream_t s) {
  const int lanes = group_lanes(C / kVec);
  auto kernel = lanes == 8    ? sample_kernel<T, kVec, kKeyBits, kNearest, 8>
                : lanes == 16 ? sample_kernel<T, kVec, kKeyBits, kNearest, 16>
                              : sample_kernel<T, kVec, kKeyBits, kNearest, 32>;
  // eight CTAs per SM at most: more would only shorten the walks that hide the lookups
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>(ceil_div(points, 8 * kSamplePoints), int64_t(device_sm_count()) * 8));
  return launch_chained(kernel, dim3(grid), dim3(256), 0, s, static_cast<const T*>(feats),
                        query, points, L, g, table, slots, C, static_cast<T*>(out), neighbor, weight);
}
template <typename T, int kVec>
static cudaError_t launch_sample(int key_bits, bool nearest, const void* feats, const float* query, uint32_t points, uint32_t L, Grid3 g, void* table,
                                 uint32_t slots, int C, void* out, uint32_t* neighbor, float* weight, cudaStream_t s) {
  if (key_bits == 32)
    return nearest ? launch_sample<T, kVec, 32, true>(feats, query, points, L, g, table, slots, C, out, neighbor, weight, s)
                   : launch_sample<T, kVec, 32, false>(feats, query, points, L, g, table, slots, C, out, neighbor, weight, s);
  return nearest ? launch_sample<T, kVec, 64, true>(feats, query, points, L, g, table, slots, C, out, neighbor, weight, s)
                 : launch_sample<T, kVec, 64, false>(feats, query, points, L, g, table, slots, C, out, neighbor, weight, s);
}

// How the voxels' lists are summed, for rows of nv packs, and where lists are cut.  A piece takes a warp about as long as a
// list just below the limit takes whoever walks that (20 to 40 us), so a cut list does not end after the rest.
struct GroupPlan {
  int warps, lanes;
  uint32_t limit, piece;
};
static GroupPlan group_plan(uint32_t entries, uint32_t n, int nv) {
  const uint32_t mean = entries / n;  // places of entries, of which a part is used
  if (mean >= 128) return {8, group_lanes(nv), 8192, 1024};  // few warps would walk long lists otherwise
  if (nv <= 16 && mean < 32) return {0, nv <= 2 ? 2 : nv <= 4 ? 4 : nv <= 8 ? 8 : 16, 256, 128};
  return {1, group_lanes(nv), 1024, 512};
}

template <typename T, int kVec>
static cudaError_t launch_group_sum(const GroupPlan& g, const void* grad_out, const uint2* grouped, const uint32_t* start, const uint32_t* count,
                                    uint32_t n, int C, void* grad_feats, const CutLists& cut, uint32_t piece_ctas, cudaStream_t s) {
  void (*kernel)(const T*, const uint2*, const uint32_t*, const uint32_t*, uint32_t, int, T*, CutLists, uint32_t);
  int64_t rows_ctas = ceil_div(n, 8);
  if (g.warps == 8) {
    kernel = g.lanes == 8 ? group_sum_kernel<T, kVec, 8, 8> : g.lanes == 16 ? group_sum_kernel<T, kVec, 8, 16> : group_sum_kernel<T, kVec, 8, 32>;
    rows_ctas = n;
  } else if (g.warps == 0) {
    kernel = g.lanes == 2 ? group_sum_kernel<T, kVec, 0, 2> : g.lanes == 4 ? group_sum_kernel<T, kVec, 0, 4>
             : g.lanes == 8 ? group_sum_kernel<T, kVec, 0, 8> : group_sum_kernel<T, kVec, 0, 16>;
    rows_ctas = ceil_div(n, 8 * (32 / g.lanes));
  } else {
    kernel = g.lanes == 8 ? group_sum_kernel<T, kVec, 1, 8> : g.lanes == 16 ? group_sum_kernel<T, kVec, 1, 16> : group_sum_kernel<T, kVec, 1, 32>;
  }
  return launch_chained(kernel, dim3(static_cast<unsigned>(piece_ctas + rows_ctas)), dim3(256), 0, s, static_cast<const T*>(grad_out), grouped, start,
                        count, n, C, static_cast<T*>(grad_feats), cut, piece_ctas);
}

struct GroupScratch {
  size_t count_off, total_off, zero_bytes, start_off, grouped_off, bytes;
};
static GroupScratch group_scratch(int64_t entries, int64_t n) {
  GroupScratch g;
  g.count_off = 0;
  g.total_off = align256(n * 4);  // [0] places handed out [1] pieces listed
  g.zero_bytes = g.total_off + 256;
  g.start_off = g.zero_bytes;
  g.grouped_off = g.start_off + align256(n * 4);
  g.bytes = g.grouped_off + align256(entries * 8);
  return g;
}
// what cutting needs behind that
struct CutScratch {
  int64_t pieces;  // at most; 0 where no list can exceed the limit
  size_t pieces_off, done_off, slab_off, end;
};
static CutScratch cut_scratch(const GroupScratch& g, const GroupPlan& plan, int64_t entries, int C) {
  CutScratch c{};
  // a list of len > limit entries has at most len / piece + 1 pieces, and there are fewer than entries / limit such lists
  c.pieces = entries > plan.limit ? entries / plan.piece + entries / plan.limit + 1 : 0;
  c.pieces_off = g.bytes;
  c.done_off = c.pieces_off + align256(c.pieces * 8);
  c.slab_off = c.done_off + align256(c.pieces * 4);
  c.end = c.slab_off + align256(c.pieces * C * 4);
  return c;
}
static int pack_width(int C, int dtype) { return elem_bytes(dtype) == 2 && C % 8 == 0 ? 8 : 4; }

static int check_table(const void* table, int64_t slots, int key_bits) {
  if (key_bits != 32 && key_bits != 64) return FGB_E_DTYPE;
  if (slots < 1 || slots >= (int64_t(1) << 31)) return FGB_E_SIZE;
  if (!table) return FGB_E_NULL;
  if (reinterpret_cast<uintptr_t>(table) & 7) return FGB_E_ALIGN;
  return FGB_OK;
}

static int elem_code_ok(int dtype) { return dtype == FGB_F16 || dtype == FGB_BF16 || dtype == FGB_F32_TF32 || dtype == FGB_F32_IEEE; }

}  // namespace fgb

extern "C" int fgb_hash_insert_3d_idx_as_val(const int32_t* coords, int64_t n, int W, int H, int D, void* table, int64_t slots,
                                             int key_bits, int32_t* status, void* stream) {
  using namespace fgb;
  if (n < 0 || n >= (int64_t(1) << 32) - 1 || W <= 0 || H <= 0 || D <= 0) return FGB_E_SIZE;
  int rc = check_table(table, slots, key_bits);
  if (rc != FGB_OK) return rc;
  if (slots < n) return FGB_E_SIZE;
  if (n > 0 && !coords) return FGB_E_NULL;
  if (reinterpret_cast<uintptr_t>(coords) & 15) return FGB_E_ALIGN;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t words = static_cast<size_t>(fgb_hash_table_bytes(slots, key_bits)) / 4;
  const unsigned grid = static_cast<unsigned>(std::min<size_t>((words + 2047) / 2048, 148 * 16));
  launch(fill_words_kernel, grid > 0 ? grid : 1, 256, 0, s, static_cast<uint32_t*>(table), words, 0xFFFFFFFFu);
  if (n == 0) return launch_status();
  const Grid3 g{W, H, D};
  const unsigned blocks = static_cast<unsigned>(ceil_div(n, kMapBlock));
  if (key_bits == 32)
    launch(hash_insert_kernel<32>, blocks, kMapBlock, 0, s, reinterpret_cast<const int4*>(coords), static_cast<uint32_t>(n), g, table,
                                                       static_cast<uint32_t>(slots), status, nullptr);
  else
    launch(hash_insert_kernel<64>, blocks, kMapBlock, 0, s, reinterpret_cast<const int4*>(coords), static_cast<uint32_t>(n), g, table,
                                                       static_cast<uint32_t>(slots), status, nullptr);
  return launch_status();
}

extern "C" int fgb_hash_lookup_3d(const int32_t* query_coords, int64_t m, int W, int H, int D, void* table, int64_t slots, int key_bits,
                                  uint32_t* out_rows, void* stream) {
  using namespace fgb;
  if (m < 0 || m >= (int64_t(1) << 32) - 1 || W <= 0 || H <= 0 || D <= 0) return FGB_E_SIZE;
  int rc = check_table(table, slots, key_bits);
  if (rc != FGB_OK) return rc;
  if (m == 0) return FGB_OK;
  if (!query_coords || !out_rows) return FGB_E_NULL;
  if (reinterpret_cast<uintptr_t>(query_coords) & 15) return FGB_E_ALIGN;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const Grid3 g{W, H, D};
  const unsigned blocks = static_cast<unsigned>(ceil_div(m, 256));
  if (key_bits == 32)
    launch(hash_lookup_3d_kernel<32>, blocks, 256, 0, s, reinterpret_cast<const int4*>(query_coords), static_cast<uint32_t>(m), g, table,
                                                    static_cast<uint32_t>(slots), out_rows);
  else
    launch(hash_lookup_3d_kernel<64>, blocks, 256, 0, s, reinterpret_cast<const int4*>(query_coords), static_cast<uint32_t>(m), g, table,
                                                    static_cast<uint32_t>(slots), out_rows);
  return launch_status();
}

extern "C" int fgb_grid_sample_neighbor_map(const float* query, int64_t B, int64_t L, int W, int H, int D, void* table, int64_t slots,
                                            int key_bits, int trilinear, uint32_t* neighbor, float* weight, void* stream) {
  using namespace fgb;
  if (B < 0 || L < 0 || B * L >= (int64_t(1) << 28) || W <= 0 || H <= 0 || D <= 0) return FGB_E_SIZE;
  int rc = check_table(table, slots, key_bits);
  if (rc != FGB_OK) return rc;
  if (B * L == 0) return FGB_OK;
  if (!query || !neighbor || (trilinear && !weight)) return FGB_E_NULL;
  if (trilinear && ((reinterpret_cast<uintptr_t>(neighbor) | reinterpret_cast<uintptr_t>(weight)) & 15)) return FGB_E_ALIGN;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const Grid3 g{W, H, D};
  const unsigned blocks = static_cast<unsigned>(ceil_div(B * L, 256));
  const uint32_t b = static_cast<uint32_t>(B), l = static_cast<uint32_t>(L), sl = static_cast<uint32_t>(slots);
  if (trilinear) {
    if (key_bits == 32) launch(trilinear_map_kernel<32>, blocks, 256, 0, s, query, b, l, g, table, sl, neighbor, weight);
    else launch(trilinear_map_kernel<64>, blocks, 256, 0, s, query, b, l, g, table, sl, neighbor, weight);
  } else {
    if (key_bits == 32) launch(nearest_map_kernel<32>, blocks, 256, 0, s, query, b, l, g, table, sl, neighbor);
    else launch(nearest_map_kernel<64>, blocks, 256, 0, s, query, b, l, g, table, sl, neighbor);
  }
  return launch_status();
}

extern "C" int fgb_indice_weighted_sum_fwd(const void* feats, const uint32_t* indices, const float* weight, void* out, int64_t M,
                                           int C, int V, int dtype, void* stream) {
  using namespace fgb;
  if (!elem_code_ok(dtype)) return FGB_E_DTYPE;
  if (M < 0 || C <= 0 || V < 1 || V > 64) return FGB_E_SIZE;
  if (C % 4) return FGB_E_ALIGN;
  if (M == 0) return FGB_OK;
  if (!feats || !indices || !out) return FGB_E_NULL;
  if ((reinterpret_cast<uintptr_t>(feats) | reinterpret_cast<uintptr_t>(out)) & 15) return FGB_E_ALIGN;
  const int64_t blocks = ceil_div(M * (C / 4), 256);
  if (blocks > 0x7FFFFFFF) return FGB_E_SIZE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const unsigned g = static_cast<unsigned>(blocks);
  if (dtype == FGB_F16)
    launch(weighted_gather_kernel<__half>, g, 256, 0, s, static_cast<const __half*>(feats), indices, weight, static_cast<__half*>(out), M, C, V);
  else if (dtype == FGB_BF16)
    launch(weighted_gather_kernel<__nv_bfloat16>, g, 256, 0, s, static_cast<const __nv_bfloat16*>(feats), indices, weight,
                                                            static_cast<__nv_bfloat16*>(out), M, C, V);
  else
    launch(weighted_gather_kernel<float>, g, 256, 0, s, static_cast<const float*>(feats), indices, weight, static_cast<float*>(out), M, C, V);
  return launch_status();
}

extern "C" int fgb_indice_weighted_sum_bwd(const void* grad_out, const uint32_t* indices, const float* weight, float* grad_feats_f32,
                                           int64_t M, int64_t N, int C, int V, int dtype, void* stream) {
  using namespace fgb;
  if (!elem_code_ok(dtype)) return FGB_E_DTYPE;
  if (M < 0 || N < 0 || C <= 0 || V < 1 || V > 64) return FGB_E_SIZE;
  if (C % 4) return FGB_E_ALIGN;
  if (N > 0 && !grad_feats_f32) return FGB_E_NULL;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (N > 0) {
    int rc = cuda_status(cudaMemsetAsync(grad_feats_f32, 0, static_cast<size_t>(N) * C * sizeof(float), s));
    if (rc != FGB_OK) return rc;
  }
  if (M == 0 || N == 0) return FGB_OK;
  if (!grad_out || !indices) return FGB_E_NULL;
  if ((reinterpret_cast<uintptr_t>(grad_out) | reinterpret_cast<uintptr_t>(grad_feats_f32)) & 15) return FGB_E_ALIGN;
  const int64_t blocks = ceil_div(M * (C / 4), 256);
  if (blocks > 0x7FFFFFFF) return FGB_E_SIZE;
  const unsigned g = static_cast<unsigned>(blocks);
  if (dtype == FGB_F16)
    launch(weighted_scatter_kernel<__half>, g, 256, 0, s, static_cast<const __half*>(grad_out), indices, weight, grad_feats_f32, M, C, V);
  else if (dtype == FGB_BF16)
    launch(weighted_scatter_kernel<__nv_bfloat16>, g, 256, 0, s, static_cast<const __nv_bfloat16*>(grad_out), indices, weight, grad_feats_f32, M,
                                                             C, V);
  else
    launch(weighted_scatter_kernel<float>, g, 256, 0, s, static_cast<const float*>(grad_out), indices, weight, grad_feats_f32, M, C, V);
  return launch_status();
}

extern "C" int fgb_grid_sample_fused(const int32_t* coords, int64_t n, const void* feats, const float* query, int64_t B, int64_t L, int W, int H,
                                     int D, int C, int dtype, int trilinear, void* table, int64_t slots, int key_bits, int32_t* table_status,
                                     void* out, uint32_t* neighbor, float* weight, void* stream) {
  using namespace fgb;
  if (!elem_code_ok(dtype)) return FGB_E_DTYPE;
  if (n < 0 || n >= (int64_t(1) << 32) - 1 || B < 0 || L < 0 || B * L >= (int64_t(1) << 28) || W <= 0 || H <= 0 || D <= 0 || C <= 0) return FGB_E_SIZE;
  if (C % 4) return FGB_E_ALIGN;
  int rc = check_table(table, slots, key_bits);
  if (rc != FGB_OK) return rc;
  if (slots < n) return FGB_E_SIZE;
  if (B * L == 0) return FGB_OK;
  if ((n > 0 && (!coords || !feats)) || !query || !out || (neighbor != nullptr && trilinear && !weight)) return FGB_E_NULL;
  if ((reinterpret_cast<uintptr_t>(coords) | reinterpret_cast<uintptr_t>(feats) | reinterpret_cast<uintptr_t>(out)) & 15) return FGB_E_ALIGN;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(table, 0xFF, static_cast<size_t>(fgb_hash_table_bytes(slots, key_bits)), s);
  if (e != cudaSuccess) return cuda_status(e);
  const Grid3 g{W, H, D};
  const uint32_t sl = static_cast<uint32_t>(slots), points = static_cast<uint32_t>(B * L), l = static_cast<uint32_t>(L);
  if (n > 0) {
    const dim3 blocks(static_cast<unsigned>(ceil_div(n, kMapBlock)));
    const int4* c4 = reinterpret_cast<const int4*>(coords);
    const uint32_t* always = nullptr;
    e = key_bits == 32 ? launch_chained(hash_insert_kernel<32>, blocks, dim3(kMapBlock), 0, s, c4, static_cast<uint32_t>(n), g, table, sl, table_status, always)
                       : launch_chained(hash_insert_kernel<64>, blocks, dim3(kMapBlock), 0, s, c4, static_cast<uint32_t>(n), g, table, sl, table_status, always);
    if (e != cudaSuccess) return cuda_status(e);
  }
  const bool nearest = trilinear == 0;
  if (dtype == FGB_F16)
    e = C % 8 == 0 ? launch_sample<__half, 8>(key_bits, nearest, feats, query, points, l, g, table, sl, C, out, neighbor, weight, s)
                   : launch_sample<__half, 4>(key_bits, nearest, feats, query, points, l, g, table, sl, C, out, neighbor, weight, s);
  else if (dtype == FGB_BF16)
    e = C % 8 == 0 ? launch_sample<__nv_bfloat16, 8>(key_bits, nearest, feats, query, points, l, g, table, sl, C, out, neighbor, weight, s)
                   : launch_sample<__nv_bfloat16, 4>(key_bits, nearest, feats, query, points, l, g, table, sl, C, out, neighbor, weight, s);
  else
    e = launch_sample<float, 4>(key_bits, nearest, feats, query, points, l, g, table, sl, C, out, neighbor, weight, s);
  return e != cudaSuccess ? cuda_status(e) : launch_status();
}

extern "C" int64_t fgb_indice_weighted_sum_grad_bytes(int64_t M, int64_t N, int V) {
  if (M < 0 || N < 0 || N >= (int64_t(1) << 32) - 1 || V < 1 || V > 64 || M * V >= (int64_t(1) << 32)) return FGB_E_SIZE;
  return static_cast<int64_t>(fgb::group_scratch(M * V, N).bytes);
}

extern "C" int64_t fgb_indice_weighted_sum_grad_full_bytes(int64_t M, int64_t N, int C, int V, int dtype) {
  using namespace fgb;
  const int64_t bytes = fgb_indice_weighted_sum_grad_bytes(M, N, V);
  if (!elem_code_ok(dtype)) return FGB_E_DTYPE;
  if (bytes < 0 || C <= 0) return FGB_E_SIZE;
  if (C % 4) return FGB_E_ALIGN;
  if (N == 0) return bytes;
  const GroupPlan plan = group_plan(static_cast<uint32_t>(M * V), static_cast<uint32_t>(N), C / pack_width(C, dtype));
  return static_cast<int64_t>(cut_scratch(group_scratch(M * V, N), plan, M * V, C).end);
}

extern "C" int fgb_indice_weighted_sum_grad(const void* grad_out, const uint32_t* indices, const float* weight, void* grad_feats, int64_t M,
                                            int64_t N, int C, int V, int dtype, void* workspace, int64_t workspace_bytes, void* stream) {
  using namespace fgb;
  if (!elem_code_ok(dtype)) return FGB_E_DTYPE;
  const int64_t bytes = fgb_indice_weighted_sum_grad_bytes(M, N, V);
  if (bytes < 0 || C <= 0) return FGB_E_SIZE;
  if (C % 4) return FGB_E_ALIGN;
  if (N == 0) return FGB_OK;
  if (!grad_feats || !workspace || (M > 0 && (!grad_out || !indices))) return FGB_E_NULL;
  if ((reinterpret_cast<uintptr_t>(grad_out) | reinterpret_cast<uintptr_t>(grad_feats)) & 15) return FGB_E_ALIGN;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return FGB_E_ALIGN;
  if (workspace_bytes < bytes) return FGB_E_WORKSPACE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const uint32_t entries = static_cast<uint32_t>(M * V), n = static_cast<uint32_t>(N);
  const GroupScratch G = group_scratch(entries, N);
  char* mem = static_cast<char*>(workspace);
  uint32_t* count = reinterpret_cast<uint32_t*>(mem + G.count_off);
  uint32_t* total = reinterpret_cast<uint32_t*>(mem + G.total_off);
  uint32_t* start = reinterpret_cast<uint32_t*>(mem + G.start_off);
  uint2* grouped = reinterpret_cast<uint2*>(mem + G.grouped_off);
  const GroupPlan plan = group_plan(entries, n, C / pack_width(C, dtype));
  const CutScratch K = cut_scratch(G, plan, entries, C);
  CutLists cut{0xFFFFFFFFu, plan.piece, total + 1, nullptr, nullptr, nullptr};
  uint32_t piece_ctas = 0;
  if (K.pieces > 0 && workspace_bytes >= static_cast<int64_t>(K.end)) {
    cut.limit = plan.limit;
    cut.pieces = reinterpret_cast<uint2*>(mem + K.pieces_off);
    cut.done = reinterpret_cast<uint32_t*>(mem + K.done_off);
    cut.slab = reinterpret_cast<float*>(mem + K.slab_off);
    piece_ctas = static_cast<uint32_t>(std::min<int64_t>(ceil_div(K.pieces, 8), int64_t(device_sm_count()) * 2));
  }
  LaunchErrors chain;
  chain.add(cudaMemsetAsync(mem, 0, G.zero_bytes, s));
  if (entries > 0) {
    const dim3 egrid(static_cast<unsigned>(std::min<int64_t>(ceil_div(entries, 256), 148 * 32)));
    chain.add(launch_chained(group_count_kernel, egrid, dim3(256), 0, s, indices, entries, count));
    chain.add(launch_chained(group_place_kernel, dim3(static_cast<unsigned>(ceil_div(N, 1024))), dim3(1024), 0, s, static_cast<const uint32_t*>(count), n,
                             start, total, cut));
    chain.add(launch_chained(group_fill_kernel, egrid, dim3(256), 0, s, indices, weight, entries, V, start, grouped));
  }
  if (dtype == FGB_F16)
    chain.add(C % 8 == 0 ? launch_group_sum<__half, 8>(plan, grad_out, grouped, start, count, n, C, grad_feats, cut, piece_ctas, s)
                         : launch_group_sum<__half, 4>(plan, grad_out, grouped, start, count, n, C, grad_feats, cut, piece_ctas, s));
  else if (dtype == FGB_BF16)
    chain.add(C % 8 == 0 ? launch_group_sum<__nv_bfloat16, 8>(plan, grad_out, grouped, start, count, n, C, grad_feats, cut, piece_ctas, s)
                         : launch_group_sum<__nv_bfloat16, 4>(plan, grad_out, grouped, start, count, n, C, grad_feats, cut, piece_ctas, s));
  else
    chain.add(launch_group_sum<float, 4>(plan, grad_out, grouped, start, count, n, C, grad_feats, cut, piece_ctas, s));
  return chain.first != cudaSuccess ? cuda_status(chain.first) : launch_status();
}
