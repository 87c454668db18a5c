// Neighbour cache of small inputs (up to 8192 rows) in two launches.
//
// At these sizes the general build is a chain of ten stream operations that each do a microsecond of work: the host
// spends 25 us on launching them and the device as long on passing from one to the next.  Here the map kernel's CTAs
// each insert ALL rows into a hash table in their own shared memory (8192 rows: 8 inserts per thread) and look their 256
// rows' neighbours up in it -- no table in memory, nothing to clear, no order to detect -- and one CTA then does all that
// follows from the codes: scan of the per-block counts, argsort, tile masks, schedule.
#include <algorithm>

#include "fgb_hash.cuh"
#include "fgb_map.cuh"

namespace fgb {

constexpr int kSmallThreads = 1024;
constexpr uint32_t kNoRow = 0xFFFFFFFFu;

struct SmallStencil {
  int K[3], D[3], V;
};

template <int kKeyBits>
__global__ void __launch_bounds__(kSmallThreads) small_map_kernel(const int4* __restrict__ coords, uint32_t n, Grid3 g, SmallStencil st,
                                                                  uint32_t slots /* power of two >= 2 n */, MapOut o) {
  using Key = typename std::conditional<kKeyBits == 32, uint32_t, unsigned long long>::type;
  extern __shared__ __align__(16) uint8_t s_mem[];
  Key* s_key = reinterpret_cast<Key*>(s_mem);                            // [n]
  uint32_t* s_table = reinterpret_cast<uint32_t*>(s_key + ((n + 3) & ~3u));  // [slots] row or kNoRow
  __shared__ uint32_t s_gray[kMapBlock];
  __shared__ uint32_t s_count[32];
  __shared__ int4 s_delta[32];
  chain_release();
  const int t = threadIdx.x;
  const int V = st.V;
  for (uint32_t i = t; i < slots; i += kSmallThreads) s_table[i] = kNoRow;
  if (t < kMapBlock) s_gray[t] = 0;
  if (t < 32) {
    s_count[t] = 0;
    const int kx = t / (st.K[1] * st.K[2]), ky = t / st.K[2] % st.K[1], kz = t % st.K[2];
    s_delta[t] = make_int4((kx - st.K[0] / 2) * st.D[0], (ky - st.K[1] / 2) * st.D[1], (kz - st.K[2] / 2) * st.D[2], 0);
  }
  chain_wait();
  for (uint32_t i = t; i < n; i += kSmallThreads) {
    const int4 c = __ldg(&coords[i]);
    s_key[i] = static_cast<Key>(g.template key<kKeyBits>(c.x, c.y, c.z, c.w));
  }
  __syncthreads();
  const uint32_t mask = slots - 1u;
  auto home = [&](Key k) -> uint32_t { return (kKeyBits == 32 ? fmix32(static_cast<uint32_t>(k)) : fmix64_hi(k)) & mask; };
  for (uint32_t i = t; i < n; i += kSmallThreads) {
    const Key k = s_key[i];
    for (uint32_t s = home(k);; s = (s + 1u) & mask) {  // at most n of the 2 n slots are taken: ends
      const uint32_t prev = atomicCAS(&s_table[s], kNoRow, i);
      if (prev == kNoRow || s_key[prev] == k) break;
    }
  }
  __syncthreads();
  const uint32_t n0 = blockIdx.x * kMapBlock, nv = min(static_cast<uint32_t>(kMapBlock), n - n0);
  const uint32_t items = nv * V;
  uint32_t* out = o.nbr + size_t(n0) * V;
  for (uint32_t item = t; item < items; item += kSmallThreads) {
    const uint32_t lv = item / V;
    const int v = static_cast<int>(item - lv * V);
    const int4 c = __ldg(&coords[n0 + lv]), d = s_delta[v];
    const int x = c.y + d.x, y = c.z + d.y, z = c.w + d.z;
    uint32_t val = kInvalid;
    if (v == (V >> 1)) {
      val = n0 + lv;
    } else if (x >= 0 && x < g.W && y >= 0 && y < g.H && z >= 0 && z < g.D) {
      const Key k = static_cast<Key>(g.template key<kKeyBits>(c.x, x, y, z));
      for (uint32_t s = home(k);; s = (s + 1u) & mask) {
        const uint32_t row = s_table[s];
        if (row == kNoRow) break;
        if (s_key[row] == k) {
          val = row;
          break;
        }
      }
    }
    out[item] = val;
    if (val != kInvalid) {
      atomicOr(&s_gray[lv], 1u << v);
      atomicAdd(&s_count[v], 1u);
    }
  }
  __syncthreads();
  if (t < nv) {
    o.gray[n0 + t] = static_cast<int32_t>(s_gray[t]);
    o.binary[n0 + t] = static_cast<int32_t>(gray_to_binary(s_gray[t]));
  }
  if (t < V) o.block_counts[size_t(t) * o.nblk + blockIdx.x] = s_count[t];
}

cudaError_t launch_small_map(const int32_t* coords, uint32_t n, int W, int H, int D, const int32_t* k, const int32_t* dil, int key_bits,
                             const MapOut& o, cudaStream_t s) {
  const SmallStencil st{{k[0], k[1], k[2]}, {dil[0], dil[1], dil[2]}, k[0] * k[1] * k[2]};
  uint32_t slots = 64;
  while (slots < 2 * n) slots <<= 1;
  const size_t smem = size_t((n + 3) & ~3u) * (key_bits / 8) + size_t(slots) * 4;
  static PerDeviceTable configured32, configured64;
  const int rc = key_bits == 32 ? ensure_dynamic_smem(configured32, small_map_kernel<32>, smem) : ensure_dynamic_smem(configured64, small_map_kernel<64>, smem);
  if (rc != FGB_OK) return cudaErrorInvalidConfiguration;
  auto kernel = key_bits == 32 ? small_map_kernel<32> : small_map_kernel<64>;
  return launch_chained(kernel, dim3(o.nblk), dim3(kSmallThreads), smem, s, reinterpret_cast<const int4*>(coords), n, Grid3{W, H, D}, st, slots, o);
}

// One CTA: argsort of the codes (least significant digit first, as fgb_sort.cu: stable ranks by warp match, per-warp digit
// counts, but all in shared memory), tile masks, schedule, and the scan of the per-block counts.
template <int kItems>
__global__ void __launch_bounds__(kSmallThreads) small_plan_kernel(PlanJob job_a, PlanJob job_b) {
  constexpr int kWarps = kSmallThreads / 32;
  const PlanJob& j = blockIdx.x == 0 ? job_a : job_b;
  extern __shared__ __align__(16) uint8_t s_mem[];
  uint32_t* s_keys = reinterpret_cast<uint32_t*>(s_mem);                         // [kItems * 1024]
  uint16_t* s_vals = reinterpret_cast<uint16_t*>(s_keys + kItems * kSmallThreads);  // [kItems * 1024]
  uint16_t* s_cnt = s_vals + kItems * kSmallThreads;                             // [kWarps][512]
  __shared__ uint32_t s_scan[kWarps];
  __shared__ uint32_t s_total[33];
  __shared__ ScheduleSmem s_sched;
  chain_release();
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  chain_wait();
  const uint32_t n = j.n;
  if (j.counts != nullptr) {
    // per-block counts of offset w -> offsets, in place (at most 32 blocks); totals -> segment table
    const uint32_t nblk = (n + kMapBlock - 1) / kMapBlock;
    if (w < j.V) {
      const uint32_t x = lane < nblk ? __ldcg(&j.counts[size_t(w) * nblk + lane]) : 0u;
      uint32_t inc = x;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += y;
      }
      if (lane < nblk) j.counts[size_t(w) * nblk + lane] = inc - x;
      if (lane == 31) s_total[w] = inc;
    }
    __syncthreads();
    if (w == 0) {
      const uint32_t x = lane < j.V ? s_total[lane] : 0u;
      uint32_t inc = x;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += y;
      }
      if (lane < j.V) j.seg[lane + 1] = inc;
      if (lane == 0) j.seg[0] = 0;
      if (lane == 31) {
        if (j.fin.build_status != nullptr) j.seg[j.V + 1] = 1u, j.seg[j.V + 2] = 0u;  // not by columns; nothing can run full
        tell_host(j.fin.host_words, j.fin.host_seq, inc, 1u, 0u);
      }
    }
  }
  // warp w holds keys [w * 32 * kItems, (w + 1) * 32 * kItems), item i of lane l is key w * 32 * kItems + i * 32 + l
  uint32_t key[kItems], val[kItems];
  uint16_t rank[kItems];
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    val[i] = w * (32 * kItems) + i * 32 + lane;
    key[i] = val[i] < n ? sort_key_of(static_cast<uint32_t>(__ldg(&j.codes[val[i]])), j.V) : 0u;
  }
  const int passes = sort_passes_of(j.V);
  const uint32_t lt = (1u << lane) - 1u;
  for (int pass = 0; pass < passes; ++pass) {
    for (int i = t; i < kWarps * kSortDigits / 2; i += kSmallThreads) reinterpret_cast<uint32_t*>(s_cnt)[i] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      // positions past the end keep their places: they are at the end of the order in every pass
      const bool ok = w * (32 * kItems) + i * 32 + lane < n;
      const uint32_t d = sort_digit_of(key[i], pass);
      const unsigned valid = __ballot_sync(0xffffffffu, ok);
      const unsigned peers = __match_any_sync(0xffffffffu, d) & valid;
      const int leader = __ffs(peers) - 1;
      uint32_t before = 0;
      if (ok && lane == leader) {
        before = s_cnt[w * kSortDigits + d];
        s_cnt[w * kSortDigits + d] = static_cast<uint16_t>(before + __popc(peers));
      }
      before = __shfl_sync(0xffffffffu, before, leader < 0 ? 0 : leader);
      rank[i] = static_cast<uint16_t>(before + __popc(peers & lt));
      __syncwarp();
    }
    __syncthreads();
    uint32_t total = 0;
    if (t < kSortDigits) {
#pragma unroll 8
      for (int ww = 0; ww < kWarps; ++ww) {
        const uint32_t c = s_cnt[ww * kSortDigits + t];
        s_cnt[ww * kSortDigits + t] = static_cast<uint16_t>(total);
        total += c;
      }
    }
    uint32_t inc = total;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += y;
    }
    if (lane == 31) s_scan[w] = inc;
    __syncthreads();
    if (t < kSortDigits) {
      uint32_t base = inc - total;
      for (int ww = 0; ww < w; ++ww) base += s_scan[ww];
#pragma unroll 8
      for (int ww = 0; ww < kWarps; ++ww) s_cnt[ww * kSortDigits + t] = static_cast<uint16_t>(s_cnt[ww * kSortDigits + t] + base);
    }
    __syncthreads();
    const bool last = pass == passes - 1;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      if (w * (32 * kItems) + i * 32 + lane >= n) continue;
      const uint32_t pos = s_cnt[w * kSortDigits + sort_digit_of(key[i], pass)] + rank[i];
      s_keys[pos] = key[i];
      s_vals[pos] = static_cast<uint16_t>(val[i]);
      if (last) j.sorted_idx[pos] = val[i];
    }
    __syncthreads();
    if (!last) {
#pragma unroll
      for (int i = 0; i < kItems; ++i) {
        const uint32_t p = w * (32 * kItems) + i * 32 + lane;
        key[i] = p < n ? s_keys[p] : 0u;
        val[i] = s_vals[p];
      }
    }
  }
  const uint32_t tiles = (n + 127) / 128;
  for (uint32_t tile = w; tile < tiles; tile += kWarps) {
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 128; i += 32) {
      const uint32_t r = tile * 128 + i + lane;
      if (r < n) m |= static_cast<uint32_t>(__ldg(&j.gray[s_vals[r]]));
    }
    m = __reduce_or_sync(0xffffffffu, m);
    if (lane == 0) j.tile_masks[tile] = m;
  }
  __threadfence();
  __syncthreads();
  block_schedule(s_sched, j.tile_masks, tiles, (tiles + 1) / 2, j.block_order);
}

template <int kItems>
static cudaError_t launch_plan(const PlanJob& a, const PlanJob* b, cudaStream_t s) {
  const size_t smem = size_t(kItems) * kSmallThreads * 6 + size_t(kSmallThreads / 32) * kSortDigits * 2;
  static PerDeviceTable configured;
  if (ensure_dynamic_smem(configured, small_plan_kernel<kItems>, smem) != FGB_OK) return cudaErrorInvalidConfiguration;
  return launch_chained(small_plan_kernel<kItems>, dim3(b != nullptr ? 2 : 1), dim3(kSmallThreads), smem, s, a, b != nullptr ? *b : a);
}
cudaError_t launch_small_plan(const PlanJob& a, const PlanJob* b, cudaStream_t s) {
  const uint32_t n = std::max(a.n, b != nullptr ? b->n : 0u);
  if (n <= 1024) return launch_plan<1>(a, b, s);
  if (n <= 2048) return launch_plan<2>(a, b, s);
  if (n <= 4096) return launch_plan<4>(a, b, s);
  return launch_plan<8>(a, b, s);
}

}  // namespace fgb
