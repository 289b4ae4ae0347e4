// gpu_build.cu -- the reference's S1 pass (RaytracerBVH.cpp:778-991) on the GPU.
//
// Same node layout and the same binary32 operations as the host builder
// (host_bvh.cpp), so the two emit identical 40-byte node arrays:
//   k_centroids      centroids ((v0+v1)+v2)/3, min/max fold from +-1e9
//                    (GetEnclosingAABB.comp:64-109); block reduction, then
//                    atomicMax on order-preserving integer images of floats
//   k_morton         the box's padding (:105-109), 30-bit codes
//                    (GenerateMortonCodesOfPrimitives.comp:52-93)
//   k_front          all of the above and the sort in one cluster, small builds
//   radix sort       stable LSD sort of (code, index), 4 passes of 8 bits like
//                    RadixSortSimple.comp:8-13: per-tile histograms, a scan, and
//                    a scatter whose ranks keep input order (warp multi-split)
//   k_tree           padded leaf boxes (ConstructHLBVH.comp:117-169), internal
//                    nodes (:72-209) and box unions, the second arriving child
//                    continuing upward (ConstructAABBsOfInternalNodes.comp:38-64)
//   k_mid, k_last,   the same for the nodes above k_tree's blocks
//   k_top
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstring>
#include <map>
#include <mutex>

#include "rt_internal.h"

namespace rtgb {

void set_error(const std::string& msg);

namespace {

constexpr int kT = 256;  // threads per block
constexpr int kBins = 256;

__device__ __forceinline__ uint32_t f2ord(float f) {  // order-preserving float -> uint
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// A vertex: one 16-byte load when the caller's array allows it (al16, uniform
// per launch; the records only promise 4 bytes), else three loads.
__device__ __forceinline__ void load_vertex(const float* p, bool al16, float v[3]) {
  if (al16) {
    const float4 f = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = f.x; v[1] = f.y; v[2] = f.z;
  } else {
    v[0] = __ldg(p); v[1] = __ldg(p + 1); v[2] = __ldg(p + 2);
  }
}

__device__ __forceinline__ bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0u; }

__device__ __forceinline__ void centroid(const RtTriangle64* __restrict__ tris, const RtSphere32* __restrict__ sph,
                                         uint32_t nt, uint32_t i, bool al16, float c[3]) {
  if (i < nt) {
    float v0[3], v1[3], v2[3];
    load_vertex(tris[i].v0, al16, v0);
    load_vertex(tris[i].v1, al16, v1);
    load_vertex(tris[i].v2, al16, v2);
    for (int k = 0; k < 3; ++k) c[k] = (v0[k] + v1[k] + v2[k]) / 3.0f;
  } else {
    const RtSphere32& s = sph[i - nt];
    for (int k = 0; k < 3; ++k) c[k] = s.center[k];
  }
}

// Centroids, kept for k_morton (12 of a primitive's 64 bytes to read again),
// and their box: words 0-2 of `box` the complements of the minima's integer
// images and 3-5 the maxima's, so that both are maxima over words that start at
// zero.  Bound by HBM: 4,194,304 triangles take 47 us here (6.8 TB/s) and 29 us
// in k_morton; reading the triangles twice, with scalar loads, took 88 and 72.
__global__ void __launch_bounds__(kT) k_centroids(const RtTriangle64* __restrict__ tris,
                                                  const RtSphere32* __restrict__ sph, uint32_t nt, uint32_t n,
                                                  float* __restrict__ cx, float* __restrict__ cy,
                                                  float* __restrict__ cz, uint32_t* __restrict__ box) {
  grid_wait();
  constexpr int kUnroll = 4;
  __shared__ float part[6][kT / 32];
  const bool al16 = aligned16(tris);
  float mn[3] = {1000000000.0f, 1000000000.0f, 1000000000.0f};
  float mx[3] = {-1000000000.0f, -1000000000.0f, -1000000000.0f};
  for (uint32_t b = blockIdx.x * (kT * kUnroll); b < n; b += gridDim.x * (kT * kUnroll)) {
    float c[kUnroll][3];
#pragma unroll
    for (int j = 0; j < kUnroll; ++j) {
      const uint32_t i = b + j * kT + threadIdx.x;
      if (i < n) centroid(tris, sph, nt, i, al16, c[j]);
    }
#pragma unroll
    for (int j = 0; j < kUnroll; ++j) {
      const uint32_t i = b + j * kT + threadIdx.x;
      if (i >= n) continue;
      cx[i] = c[j][0];
      cy[i] = c[j][1];
      cz[i] = c[j][2];
      for (int k = 0; k < 3; ++k) {
        mn[k] = fminf(mn[k], c[j][k]);
        mx[k] = fmaxf(mx[k], c[j][k]);
      }
    }
  }
  for (int k = 0; k < 3; ++k) {
    for (int o = 16; o > 0; o >>= 1) {
      mn[k] = fminf(mn[k], __shfl_down_sync(0xFFFFFFFFu, mn[k], o));
      mx[k] = fmaxf(mx[k], __shfl_down_sync(0xFFFFFFFFu, mx[k], o));
    }
    if ((threadIdx.x & 31u) == 0u) {
      part[k][threadIdx.x >> 5] = mn[k];
      part[3 + k][threadIdx.x >> 5] = mx[k];
    }
  }
  __syncthreads();
  if (threadIdx.x < 6u) {
    float v = part[threadIdx.x][0];
    for (int w = 1; w < kT / 32; ++w)
      v = threadIdx.x < 3u ? fminf(v, part[threadIdx.x][w]) : fmaxf(v, part[threadIdx.x][w]);
    atomicMax(&box[threadIdx.x], threadIdx.x < 3u ? ~f2ord(v) : f2ord(v));
  }
}

// The padding of GetEnclosingAABB.comp:105-109.
__device__ __forceinline__ void padded_box(const uint32_t* box, float mn[3], float mx[3]) {
  const float delta = 0.001f, padding = delta / 2.0f;
  for (int k = 0; k < 3; ++k) {
    mn[k] = ord2f(~box[k]);
    mx[k] = ord2f(box[3 + k]);
    if (mx[k] - mn[k] < delta) {
      mn[k] -= padding;
      mx[k] += padding;
    }
  }
}

__device__ __forceinline__ uint32_t f2u_sat(float f) { return __float2uint_rz(f); }

__device__ __forceinline__ uint32_t spread3(uint32_t v) {
  if (v == 1024u) v--;
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

__device__ __forceinline__ uint32_t morton(const float c[3], const float mn[3], const float mx[3], uint32_t mode) {
  uint32_t q[3];
  for (int k = 0; k < 3; ++k) {
    const float span = mx[k] - mn[k];
    const float off = mode == RT_BVH_REFERENCE ? c[k] / span : (c[k] - mn[k]) / span;
    q[k] = f2u_sat(off * 1024.0f);
  }
  return (spread3(q[2]) << 2) | (spread3(q[1]) << 1) | spread3(q[0]);
}

// Codes of one sort tile and their digit counts for the sort's first pass.
__global__ void __launch_bounds__(kT) k_morton(const float* __restrict__ cx, const float* __restrict__ cy,
                                               const float* __restrict__ cz, uint32_t n,
                                               const uint32_t* __restrict__ box, uint32_t mode,
                                               uint32_t* __restrict__ codes, uint32_t* __restrict__ hist,
                                               uint32_t tiles, uint32_t tile) {
  grid_wait();
  __shared__ uint32_t h[kBins];
  h[threadIdx.x] = 0u;
  float mn[3], mx[3];
  padded_box(box, mn, mx);
  __syncthreads();
  const uint32_t base = blockIdx.x * tile;
#pragma unroll 4
  for (uint32_t j = threadIdx.x; j < tile; j += kT) {
    const uint32_t i = base + j;
    if (i < n) {
      const float c[3] = {cx[i], cy[i], cz[i]};
      const uint32_t code = morton(c, mn, mx, mode);
      codes[i] = code;
      atomicAdd(&h[code & 255u], 1u);
    }
  }
  __syncthreads();
  hist[threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// ---- stable LSD radix sort, 8-bit digits ----
// A tile is 256 x ITEMS keys.  Per pass: k_rs_hist counts each tile's digits
// ([bin][tile]), k_rs_scan turns each bin's row into exclusive offsets (one
// block a bin) and leaves the bin's total, and k_rs_scatter adds the totals of
// lower bins, ranks its keys and writes them.  Bound by latency below about
// 10^5 keys and by L2 above (keys and indices of 4 M primitives, 67 MB with
// both copies, stay in L2).  us per pass at 4,194,304 keys, before and now: hist
// 11 / 7, scan 182 / 3.5 (it was one block over all 262,144 counts), scatter 91 /
// 40 (50 with __match_any_sync, which stalled the warps, or at 127 registers).
constexpr int kItemsLarge = 16;  // 4096-key tiles: 64-byte runs per digit on average
constexpr int kItemsSmall = 4;   // 1024-key tiles: four times the blocks
// Tiles of kItemsSmall up to here: at 1 M keys the large tiles are down to 256
// blocks, under two per SM.
constexpr uint32_t kSmallSort = 1u << 20;

constexpr uint32_t tile_keys(uint32_t n) { return kT * (n <= kSmallSort ? kItemsSmall : kItemsLarge); }

__global__ void __launch_bounds__(kT) k_rs_hist(const uint32_t* __restrict__ keys, uint32_t n, uint32_t shift,
                                                uint32_t* __restrict__ hist, uint32_t tiles, uint32_t tile) {
  grid_wait();
  __shared__ uint32_t h[kBins];
  h[threadIdx.x] = 0u;
  __syncthreads();
  const uint32_t base = blockIdx.x * tile;
  if (base + tile <= n) {  // tiles start 16-byte aligned
    const uint4* k4 = reinterpret_cast<const uint4*>(keys + base);
#pragma unroll 4
    for (uint32_t j = threadIdx.x; j < tile / 4u; j += kT) {
      const uint4 k = k4[j];
      atomicAdd(&h[(k.x >> shift) & 255u], 1u);
      atomicAdd(&h[(k.y >> shift) & 255u], 1u);
      atomicAdd(&h[(k.z >> shift) & 255u], 1u);
      atomicAdd(&h[(k.w >> shift) & 255u], 1u);
    }
  } else {
    for (uint32_t i = base + threadIdx.x; i < n; i += kT) atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
  }
  __syncthreads();
  hist[threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// Exclusive scan of x over the block's kT threads; *total gets the sum.
__device__ __forceinline__ uint32_t block_scan(uint32_t x, uint32_t* warp_sums, uint32_t* total) {
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  uint32_t v = x;
#pragma unroll
  for (uint32_t off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, off);
    if (lane >= off) v += y;
  }
  if (lane == 31u) warp_sums[w] = v;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (uint32_t k = 0; k < kT / 32; ++k) {
    const uint32_t c = warp_sums[k];
    before += k < w ? c : 0u;
    all += c;
  }
  __syncthreads();  // warp_sums may be rewritten
  *total = all;
  return before + v - x;
}

// Block b: exclusive scan of bin b's tile counts in place, its total to totals[b].
__global__ void __launch_bounds__(kT) k_rs_scan(uint32_t* __restrict__ hist, uint32_t tiles,
                                                uint32_t* __restrict__ totals) {
  grid_wait();
  __shared__ uint32_t warp_sums[kT / 32];
  uint32_t* row = hist + (size_t)blockIdx.x * tiles;
  uint32_t carry = 0;
  for (uint32_t base = 0; base < tiles; base += 4u * kT) {
    const uint32_t i0 = base + 4u * threadIdx.x;
    uint32_t v[4], sum = 0, total;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = i0 + k < tiles ? row[i0 + k] : 0u;
      sum += v[k];
    }
    uint32_t run = carry + block_scan(sum, warp_sums, &total);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i0 + k < tiles) row[i0 + k] = run;
      run += v[k];
    }
    carry += total;
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// Each warp holds a contiguous stretch of 32 x ITEMS keys of the tile and ranks
// it in order, 32 keys at a time: equal digits within a step rank by lane
// (a ballot per digit bit), a per-warp count keeps earlier steps ahead.  The tile is
// put in digit order in shared memory first, so that a digit's keys leave as
// one run of consecutive addresses.  vals == nullptr: the value is the index
// (the first pass).
template <int ITEMS>
__global__ void __launch_bounds__(kT, 4) k_rs_scatter(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals,
                                                   uint32_t n, uint32_t shift, const uint32_t* __restrict__ offs,
                                                   const uint32_t* __restrict__ totals, uint32_t tiles,
                                                   uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out) {
  grid_wait();
  constexpr int kWarps = kT / 32, kTile = kT * ITEMS;
  __shared__ uint32_t cnt[kWarps][kBins];
  __shared__ uint32_t sk[kTile], sv[kTile];
  __shared__ uint32_t to[kBins];  // output position of the digit's first key less its position in the tile
  __shared__ uint32_t warp_sums[kWarps];
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5, b = threadIdx.x;  // kT == kBins
  for (int i = lane; i < kBins; i += 32) cnt[w][i] = 0u;
  const uint32_t base = blockIdx.x * kTile, first = base + w * 32u * ITEMS + lane;
  const uint32_t live = min((uint32_t)kTile, n - base);
  uint32_t k[ITEMS], rank[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const uint32_t i = first + 32u * j;
    k[j] = i < n ? keys[i] : 0u;
  }
  uint32_t all;
  const uint32_t bin_base = block_scan(totals[b], warp_sums, &all) + offs[b * tiles + blockIdx.x];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const bool ok = first + 32u * j < n;
    const uint32_t d = (k[j] >> shift) & 255u;
    uint32_t peers = __ballot_sync(0xFFFFFFFFu, ok);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const bool one = (d >> b) & 1u;
      const uint32_t ones = __ballot_sync(0xFFFFFFFFu, one);
      peers &= one ? ones : ~ones;
    }
    const uint32_t seen = ok ? cnt[w][d] : 0u;
    rank[j] = seen + (uint32_t)__popc(peers & ((1u << lane) - 1u));
    __syncwarp();
    if (ok && lane == (uint32_t)(__ffs(peers) - 1)) cnt[w][d] = seen + (uint32_t)__popc(peers);
    __syncwarp();
  }
  __syncthreads();
  {  // per digit: the warps' counts become offsets within the digit, then within the tile
    uint32_t run = 0;
#pragma unroll
    for (int ww = 0; ww < kWarps; ++ww) {
      const uint32_t c = cnt[ww][b];
      cnt[ww][b] = run;
      run += c;
    }
    const uint32_t start = block_scan(run, warp_sums, &all);
#pragma unroll
    for (int ww = 0; ww < kWarps; ++ww) cnt[ww][b] += start;
    to[b] = bin_base - start;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
    if (first + 32u * j < n) {
      const uint32_t at = cnt[w][(k[j] >> shift) & 255u] + rank[j];
      sk[at] = k[j];
      sv[at] = vals ? vals[first + 32u * j] : first + 32u * j;
    }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const uint32_t i = j * kT + threadIdx.x;
    if (i < live) {
      const uint32_t key = sk[i], pos = to[(key >> shift) & 255u] + i;
      keys_out[pos] = key;
      vals_out[pos] = sv[i];
    }
  }
}

// ---- small builds: centroids, codes and sort in one cluster ----
// Below kFrontMax primitives the twelve launches above are bound by their gaps
// and by a few blocks' latency.  Here eight blocks of one cluster hold all keys
// in their shared memory: block r sorted positions [r M, (r + 1) M).  The box is
// reduced and each pass's digit counts are exchanged through distributed shared
// memory, and the scatter of a pass writes straight into the other blocks'
// buffers; cluster barriers separate the steps, no global memory in between.
// us for the whole build by the launches / by this: 16,385 primitives 54 / 16,384
// 49, 20,482 54 / 55, 32,769 57 / 32,768 69; hence the line.
constexpr int kFrontBlocks = 8, kFrontThreads = 1024, kFrontItems = 2;
constexpr uint32_t kFrontMax = kFrontBlocks * kFrontThreads * kFrontItems;  // 16 bytes a key: 32 KB a block

size_t front_smem(uint32_t n) {
  const size_t m = (n + kFrontBlocks - 1) / kFrontBlocks;
  return 16 * m + (kFrontThreads / 32) * kBins * 2;
}

__global__ void __cluster_dims__(kFrontBlocks, 1, 1) __launch_bounds__(kFrontThreads)
    k_front(const RtTriangle64* __restrict__ tris, const RtSphere32* __restrict__ sph, uint32_t nt, uint32_t n,
            uint32_t mode, uint32_t* __restrict__ codes, uint32_t* __restrict__ order, uint32_t* __restrict__ clear,
            uint32_t clear_words) {
  grid_wait();
  namespace cg = cooperative_groups;
  constexpr int kWarps = kFrontThreads / 32;
  extern __shared__ uint32_t sm[];
  __shared__ uint32_t hist[kBins], base_of[kBins], warp_sums[kBins / 32], box[6], all_box[6];
  __shared__ float part[6][kWarps];
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t rank = cluster.block_rank(), t = threadIdx.x, lane = t & 31u, w = t >> 5;
  const uint32_t M = (n + kFrontBlocks - 1) / kFrontBlocks;
  const uint32_t begin = rank * M, m = begin < n ? min(M, n - begin) : 0u;
  uint32_t *key = sm, *idx = sm + M, *key2 = sm + 2u * M, *idx2 = sm + 3u * M;
  uint16_t* cnt = reinterpret_cast<uint16_t*>(sm + 4u * M);  // [warp][bin]
  for (uint32_t i = rank * kFrontThreads + t; i < clear_words; i += kFrontBlocks * kFrontThreads) clear[i] = 0u;
  // the box of the centroids (see k_centroids)
  const bool al16 = aligned16(tris);
  float mn[3] = {1000000000.0f, 1000000000.0f, 1000000000.0f};
  float mx[3] = {-1000000000.0f, -1000000000.0f, -1000000000.0f};
  for (uint32_t i = t; i < m; i += kFrontThreads) {
    float c[3];
    centroid(tris, sph, nt, begin + i, al16, c);
    for (int k = 0; k < 3; ++k) {
      mn[k] = fminf(mn[k], c[k]);
      mx[k] = fmaxf(mx[k], c[k]);
    }
  }
  for (int k = 0; k < 3; ++k) {
    for (int o = 16; o > 0; o >>= 1) {
      mn[k] = fminf(mn[k], __shfl_down_sync(0xFFFFFFFFu, mn[k], o));
      mx[k] = fmaxf(mx[k], __shfl_down_sync(0xFFFFFFFFu, mx[k], o));
    }
    if (lane == 0u) {
      part[k][w] = mn[k];
      part[3 + k][w] = mx[k];
    }
  }
  __syncthreads();
  if (t < 6u) {
    float v = part[t][0];
    for (int k = 1; k < kWarps; ++k) v = t < 3u ? fminf(v, part[t][k]) : fmaxf(v, part[t][k]);
    box[t] = t < 3u ? ~f2ord(v) : f2ord(v);
  }
  cluster.sync();
  if (t < 6u) {
    uint32_t v = 0u;
    for (int r = 0; r < kFrontBlocks; ++r) v = max(v, cluster.map_shared_rank(box, r)[t]);
    all_box[t] = v;
  }
  __syncthreads();
  padded_box(all_box, mn, mx);
  for (uint32_t i = t; i < m; i += kFrontThreads) {
    float c[3];
    centroid(tris, sph, nt, begin + i, al16, c);
    key[i] = morton(c, mn, mx, mode);
    idx[i] = begin + i;
  }
  // four passes of 8 bits; a warp owns a contiguous stretch of the block's keys
  const uint32_t items = (M + kFrontThreads - 1) / kFrontThreads, first = w * 32u * items + lane;
  for (int pass = 0; pass < 4; ++pass) {
    const uint32_t shift = 8u * (uint32_t)pass;
    for (uint32_t i = t; i < kWarps * kBins / 2; i += kFrontThreads) reinterpret_cast<uint32_t*>(cnt)[i] = 0u;
    __syncthreads();
    uint16_t rank_of[kFrontItems];
    uint16_t* mine = cnt + w * kBins;
#pragma unroll
    for (int j = 0; j < kFrontItems; ++j) {
      if ((uint32_t)j >= items) break;
      const uint32_t i = first + 32u * j;
      const bool ok = i < m;
      const uint32_t d = ok ? (key[i] >> shift) & 255u : 0u;
      uint32_t peers = __ballot_sync(0xFFFFFFFFu, ok);
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const bool one = (d >> b) & 1u;
        const uint32_t ones = __ballot_sync(0xFFFFFFFFu, one);
        peers &= one ? ones : ~ones;
      }
      const uint32_t seen = mine[d];
      rank_of[j] = (uint16_t)(seen + (uint32_t)__popc(peers & ((1u << lane) - 1u)));
      __syncwarp();
      if (ok && lane == (uint32_t)(__ffs(peers) - 1)) mine[d] = (uint16_t)(seen + (uint32_t)__popc(peers));
      __syncwarp();
    }
    __syncthreads();
    if (t < kBins) {
      uint32_t run = 0u;
      for (int k = 0; k < kWarps; ++k) {
        const uint32_t c = cnt[k * kBins + t];
        cnt[k * kBins + t] = (uint16_t)run;
        run += c;
      }
      hist[t] = run;
    }
    cluster.sync();
    uint32_t total = 0u, before = 0u, scan = 0u;
    if (t < kBins) {
      for (uint32_t r = 0; r < (uint32_t)kFrontBlocks; ++r) {
        const uint32_t c = cluster.map_shared_rank(hist, r)[t];
        total += c;
        before += r < rank ? c : 0u;
      }
      scan = total;  // inclusive scan over the bins
#pragma unroll
      for (uint32_t off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, scan, off);
        if (lane >= off) scan += y;
      }
      if (lane == 31u) warp_sums[w] = scan;
    }
    __syncthreads();
    if (t < kBins) {
      for (uint32_t k = 0; k < w; ++k) scan += warp_sums[k];
      base_of[t] = scan - total + before;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kFrontItems; ++j) {
      if ((uint32_t)j >= items) break;
      const uint32_t i = first + 32u * j;
      if (i < m) {
        const uint32_t k = key[i], d = (k >> shift) & 255u;
        const uint32_t to = base_of[d] + mine[d] + rank_of[j], r = to / M;
        cluster.map_shared_rank(key2, r)[to - r * M] = k;
        cluster.map_shared_rank(idx2, r)[to - r * M] = idx[i];
      }
    }
    cluster.sync();
    uint32_t* x = key; key = key2; key2 = x;
    x = idx; idx = idx2; idx2 = x;
  }
  for (uint32_t i = t; i < m; i += kFrontThreads) {
    codes[begin + i] = key[i];
    order[begin + i] = idx[i];
  }
}

__device__ __forceinline__ void pad_axis(float& mn, float& mx) {
  const float delta = 0.001f, padding = delta / 2.0f;
  if (mx - mn < delta) {
    mn -= padding;
    mx += padding;
  }
}

// Padded box of primitive g (ConstructHLBVH.comp:117-169).
__device__ __forceinline__ void leaf_box(const RtTriangle64* __restrict__ tris, const RtSphere32* __restrict__ sph,
                                         uint32_t nt, uint32_t g, bool al16, float r[6]) {
  if (g < nt) {
    float a[3], b[3], c[3];
    load_vertex(tris[g].v0, al16, a);
    load_vertex(tris[g].v1, al16, b);
    load_vertex(tris[g].v2, al16, c);
    for (int k = 0; k < 3; ++k) {
      r[2 * k] = fminf(a[k], fminf(b[k], c[k]));
      r[2 * k + 1] = fmaxf(a[k], fmaxf(b[k], c[k]));
    }
  } else {
    const RtSphere32& s = sph[g - nt];
    for (int k = 0; k < 3; ++k) {
      const float l = s.center[k] - s.radius, h = s.center[k] + s.radius;
      r[2 * k] = fminf(l, h);
      r[2 * k + 1] = fmaxf(l, h);
    }
  }
  pad_axis(r[0], r[1]);
  pad_axis(r[2], r[3]);
  pad_axis(r[4], r[5]);
}

// Length of the common prefix of the augmented keys (code, index) of sorted
// neighbours i and i + 1 (the delta of ConstructHLBVH.comp:72-84).
__device__ __forceinline__ int delta_next(const uint32_t* __restrict__ codes, uint32_t i) {
  const uint32_t a = __ldg(&codes[i]), b = __ldg(&codes[i + 1u]);
  return a == b ? 32 + __clz((int)(i ^ (i + 1u))) : __clz((int)(a ^ b));
}

// Leaves, internal nodes and boxes in one pass, bottom up (after Apetrei, "Fast
// and Simple Agglomerative LBVH Construction", 2014), with Karras' numbering
// (ConstructHLBVH.comp:85-209): the node over sorted positions [l, r] is the
// left child of the node split after r if that split's common prefix is the
// longer one of its two outer neighbours', else the right child of the node
// split after l - 1; Karras numbers a left child by its last position, a right
// child by its first, and the root 0.  A thread starts at each leaf and climbs:
// of a split's two children the first to arrive leaves the far end of its range
// in the split's slot and stops, the second takes the range on.
//
// A block of k_tree owns kLeaves consecutive leaves.  Splits inside it meet in
// shared memory, and its records leave as whole lines.  The few nodes whose
// parent reaches over an edge of the block go to a list, from which k_mid and
// k_last or k_top climb on; climbing on through global slots in k_tree itself
// kept whole blocks resident for one thread's chain of atomics.  They replace a
// leaf pass, a pass of Karras searches and a bottom-up pass with a global atomic
// and two 40-byte record reads per node.  4,194,304 triangles: 666 us for those three; k_tree 311 us as
// one climb per thread, 260 with the climb cut in two, 195 with 8-byte stores,
// padded rows and one box array (bound by issue; 518 MB read, most of it the
// gather, and 289 MB written); k_top 65 us of serial atomics.
constexpr int kLeaves = 512;
constexpr int kFirstClimb = 4;
constexpr uint32_t kGroupBlocks = 128, kGroupLeaves = kGroupBlocks * kLeaves;  // blocks that share a list
constexpr uint32_t kGroupOpen = kGroupLeaves + kGroupBlocks;  // at most a node per leaf and one more per block
constexpr uint32_t kRight = 0x8000u;  // shared slot: the visitor was the right child
// Row of the boxes in shared memory: leaves, then internal nodes; five words of
// padding keep the ten words of neighbouring records in different banks.
constexpr int kBoxRow = 2 * kLeaves + 5;
constexpr uint32_t kLinked = 0x80000000u, kLeafLeft = 0x10000u, kLeafRight = 0x20000u;

__global__ void __launch_bounds__(kLeaves) k_tree(const RtTriangle64* __restrict__ tris,
                                                  const RtSphere32* __restrict__ sph, uint32_t nt, uint32_t n,
                                                  uint32_t mode, const uint32_t* __restrict__ codes,
                                                  const uint32_t* __restrict__ order, RtBVHNode40* __restrict__ nodes,
                                                  uint2* __restrict__ open, uint32_t* __restrict__ num_open) {
  grid_wait();
  open += (size_t)(blockIdx.x / kGroupBlocks) * kGroupOpen;  // the list of the block's group
  num_open += blockIdx.x / kGroupBlocks;
  // positions are relative to the block's first leaf
  __shared__ float bx[6][kBoxRow];
  __shared__ uint32_t link[kLeaves];   // internal node: its split | kLeafLeft | kLeafRight | kLinked (0: not here)
  __shared__ uint32_t prim[kLeaves];
  __shared__ uint32_t slot[kLeaves];   // split after i: 0, or a visitor's far end + 1 (and kRight)
  __shared__ uint32_t climb[kLeaves];  // nodes to climb on from: l | r << 16
  __shared__ int8_t gap[kLeaves + 1];  // delta of i - 1 and i; -1 at the ends of the whole order
  __shared__ uint32_t num_climb, num_edge, num_lone, open_at;
  __shared__ uint2 edge[2];
  const uint32_t t = threadIdx.x, base = blockIdx.x * kLeaves, i0 = base + t;
  const uint32_t live = min((uint32_t)kLeaves, n - base);
  slot[t] = 0u;
  link[t] = 0u;
  if (t <= live) gap[t] = i0 > 0u && i0 < n ? (int8_t)delta_next(codes, i0 - 1u) : (int8_t)-1;
  if (t == 0u) {
    if (live == kLeaves) gap[kLeaves] = base + kLeaves < n ? (int8_t)delta_next(codes, base + kLeaves - 1u) : (int8_t)-1;
    num_climb = num_edge = num_lone = 0u;
  }
  float box[6];
  if (t < live) {
    const uint32_t g = mode == RT_BVH_REFERENCE ? i0 : order[i0];
    leaf_box(tris, sph, nt, g, aligned16(tris), box);
    prim[t] = g;
#pragma unroll
    for (int k = 0; k < 6; ++k) bx[k][t] = box[k];
  }
  __syncthreads();
  // Half of the climbers stop at every level, and a warp climbs as long as its
  // last lane: after kFirstClimb levels the rest move together into few warps.
  uint32_t l = t, r = t;
  int gl = 0, gr = 0;  // the gaps before l and after r
  bool climbing = t < live && n > 1u;
  if (climbing) {
    gl = gap[t];
    gr = gap[t + 1u];
  }
  for (int part = 0; part < 2; ++part) {
    if (part == 1) {
      __syncthreads();
      if (climbing) climb[atomicAdd(&num_climb, 1u)] = l | r << 16;
      __syncthreads();
      climbing = t < num_climb;
      if (!climbing) break;
      l = climb[t] & 0xFFFFu;
      r = climb[t] >> 16;
      gl = gap[l];
      gr = gap[r + 1u];
#pragma unroll
      for (int k = 0; k < 6; ++k) box[k] = bx[k][kLeaves + (gr > gl ? r : l)];
    }
    for (int step = 0; climbing && (part == 1 || step < kFirstClimb); ++step) {
      const bool is_left = gr > gl;
      const uint32_t s = is_left ? r : l - 1u;  // the parent's split
      climbing = false;
      if (is_left ? r == kLeaves - 1u : l == 0u) {  // its other child is in another block
        edge[atomicAdd(&num_edge, 1u)] = make_uint2(base + l, base + r);  // one node at each edge at most
        break;
      }
      __threadfence_block();
      const uint32_t other = atomicExch(&slot[s], is_left ? l + 1u : (r + 1u) | kRight);
      if (other == 0u) break;
      __threadfence_block();
      slot[s] = 0u;  // both children have met
      const uint32_t end = (other & (kRight - 1u)) - 1u;
      uint32_t sib;
      if (is_left) {
        sib = end == s + 1u ? end : kLeaves + s + 1u;
        r = end;
        gr = gap[end + 1u];
      } else {
        sib = end == s ? s : kLeaves + s;
        l = end;
        gl = gap[end];
      }
      const bool root = (gl & gr) < 0;
      const uint32_t at = root ? 0u : (gr > gl ? r : l);  // this node's number
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const float b = bx[k][sib];
        box[k] = (k & 1) ? fmaxf(box[k], b) : fminf(box[k], b);
        bx[k][kLeaves + at] = box[k];
      }
      link[at] = s | (l == s ? kLeafLeft : 0u) | (r == s + 1u ? kLeafRight : 0u) | kLinked;
      climbing = !root;
    }
  }
  __syncthreads();
  {  // the block's records in address order, five 8-byte words each
    const uint32_t leaf_off = n - 1u;
    const bool al8 = (reinterpret_cast<uintptr_t>(nodes) & 7u) == 0u;  // the records only promise 4
    auto put = [&](uint32_t* p, uint32_t x, uint32_t y) {
      if (al8) {
        *reinterpret_cast<uint2*>(p) = make_uint2(x, y);
      } else {
        p[0] = x;
        p[1] = y;
      }
    };
    uint32_t* out_leaf = reinterpret_cast<uint32_t*>(nodes + leaf_off + base);
    uint32_t* out_inner = reinterpret_cast<uint32_t*>(nodes + base);
    for (uint32_t j = t; j < live * 5u; j += kLeaves) {
      const uint32_t i = j / 5u, w = j - 5u * i;
      uint32_t x = 0u, y = 0u;
      if (w < 3u) {
        x = __float_as_uint(bx[2u * w][i]);
        y = __float_as_uint(bx[2u * w + 1u][i]);
      } else if (w == 4u) {
        const uint32_t g = prim[i];
        x = g < nt ? g : g - nt;
        y = g < nt ? RT_PRIM_TRIANGLE : RT_PRIM_SPHERE;
      }
      put(out_leaf + 2u * j, x, y);
      const uint32_t k = link[i];
      if (k == 0u) continue;  // not an internal node that is complete here
      x = y = 0u;
      if (w < 3u) {
        x = __float_as_uint(bx[2u * w][kLeaves + i]);
        y = __float_as_uint(bx[2u * w + 1u][kLeaves + i]);
      } else if (w == 3u) {
        x = base + (k & 0xFFFFu);
        y = x + 1u;
        if (k & kLeafLeft) x += leaf_off;
        if (k & kLeafRight) y += leaf_off;
      }
      put(out_inner + 2u * j, x, y);
    }
  }
  // The nodes the next kernel climbs on from: those at the edges and the visitors that
  // met nobody in their shared slot.
  const uint32_t tag = slot[t];
  uint32_t mine = 0u;
  if (tag != 0u) mine = atomicAdd(&num_lone, 1u);
  __syncthreads();
  if (t == 0u && num_lone + num_edge) {
    open_at = atomicAdd(num_open, num_lone + num_edge);
    for (uint32_t k = 0; k < num_edge; ++k) open[open_at + k] = edge[k];
  }
  __syncthreads();
  if (tag != 0u) {
    const uint32_t end = base + (tag & (kRight - 1u)) - 1u;
    open[open_at + num_edge + mine] = (tag & kRight) ? make_uint2(i0 + 1u, end) : make_uint2(end, i0);
  }
}

__device__ __forceinline__ void read_box(const RtBVHNode40* nd, float r[6]) {
  const float* q = &nd->minX;
#pragma unroll
  for (int k = 0; k < 6; ++k) r[k] = __ldcg(q + k);  // from L2: another SM may have written it
}

__device__ __forceinline__ void write_inner(RtBVHNode40* out, const float box[6], uint32_t left, uint32_t right) {
  RtBVHNode40 nd;
  nd.minX = box[0]; nd.maxX = box[1]; nd.minY = box[2]; nd.maxY = box[3]; nd.minZ = box[4]; nd.maxZ = box[5];
  nd.left = left;
  nd.right = right;
  nd.primitiveIndex = 0u;
  nd.primitiveType = 0u;
  *out = nd;
}

// Climbs from node [l, r], whose record is written, as far as it is the second
// to arrive, through one global slot per split.
__device__ void climb_global(uint32_t l, uint32_t r, uint32_t n, const uint32_t* __restrict__ codes, uint32_t* slots,
                             RtBVHNode40* nodes) {
  const uint32_t leaf_off = n - 1u;
  uint32_t lc = 0u, rc = 0u;
  float box[6];
  for (bool written = true;; written = false) {
    const bool root = l == 0u && r == n - 1u;
    const bool is_left = l == 0u || (r != n - 1u && delta_next(codes, r) > delta_next(codes, l - 1u));
    const uint32_t number = root ? 0u : (l == r ? leaf_off + l : (is_left ? r : l));
    if (written)
      read_box(&nodes[number], box);
    else
      write_inner(&nodes[number], box, lc, rc);
    if (root) break;
    const uint32_t s = is_left ? r : l - 1u;
    __threadfence();
    const uint32_t other = atomicExch(&slots[s], (is_left ? l : r) + 1u);
    if (other == 0u) break;
    __threadfence();
    if (is_left) r = other - 1u;
    else l = other - 1u;
    lc = l == s ? leaf_off + s : s;
    rc = s + 1u == r ? leaf_off + r : s + 1u;
    float sib[6];
    read_box(&nodes[is_left ? rc : lc], sib);
#pragma unroll
    for (int k = 0; k < 6; ++k) box[k] = (k & 1) ? fmaxf(box[k], sib[k]) : fminf(box[k], sib[k]);
  }
}

// One block per group of kGroupBlocks blocks of k_tree: the listed nodes
// partition the group's positions (about nine per block of k_tree), a bitmap of
// their first positions ranks them, and k_tree's climb runs over those ranks in
// shared memory.  What reaches over the group's edges goes to the next list, for
// k_last.  A group with more than kMidItems nodes (long runs of equal codes) is
// left to k_top as it is, or, alone, climbs through the global slots here.
// k_top alone takes a global atomic, two fences and a record read per level: 45
// us for the top of the tree of 20,482 primitives, 14 with k_mid.
constexpr int kMidThreads = 1024;
constexpr uint32_t kMidItems = 1792, kMidWords = kGroupLeaves / 32;
static_assert(kMidWords <= 2 * kMidThreads, "two words of the bitmap per thread");
constexpr size_t kMidSmem = kMidItems * (12 * 4 + 4 + 4) + 8 + (kMidItems + 4) + kMidWords * 8;
constexpr uint32_t kMidOpen = kMidItems + 2;  // nodes that a group leaves at most
constexpr uint32_t kLongLists = 0x80000000u;  // in the count of those nodes: some group's list was too long

// The block's shared memory in k_mid and k_last.
struct MidShared {
  float* bx;       // [6][nodes by rank, then internal nodes by the rank that numbers them]
  uint32_t* slot;  // split after rank i: 0, or a visitor's far end + 1 (and kRight)
  uint32_t* pos;   // first position of rank i; the end after the last
  uint32_t* bits;
  uint32_t* before;  // ranks before a word of bits
  int8_t* gap;       // delta across the start of rank i
};
__device__ __forceinline__ MidShared mid_shared(uint32_t* sm) {
  MidShared m;
  m.bx = reinterpret_cast<float*>(sm);
  m.slot = sm + 12 * kMidItems;
  m.pos = m.slot + kMidItems;
  m.bits = m.pos + kMidItems + 2;
  m.before = m.bits + kMidWords;
  m.gap = reinterpret_cast<int8_t*>(m.before + kMidWords);
  return m;
}

// k_tree's climb over the ranks 0..count-1 (pos is set, slot is zero); nodes
// whose sibling lies outside go to `next`.
__device__ void climb_ranked(const MidShared& m, uint32_t count, uint32_t n, const uint32_t* __restrict__ codes,
                             RtBVHNode40* nodes, uint2* __restrict__ next, uint32_t* __restrict__ num_next) {
  float* bx = m.bx;
  uint32_t *slot = m.slot, *pos = m.pos;
  int8_t* gap = m.gap;
  const uint32_t t = threadIdx.x, leaf_off = n - 1u;
  for (uint32_t i = t; i <= count; i += kMidThreads)
    gap[i] = pos[i] > 0u && pos[i] < n ? (int8_t)delta_next(codes, pos[i] - 1u) : (int8_t)-1;
  __syncthreads();
  for (uint32_t i = t; i < count; i += kMidThreads) {
    uint32_t l = i, r = i;
    int gl = gap[i], gr = gap[i + 1u];
    float box[6];
    {
      const uint32_t first = pos[i], last = pos[i + 1u] - 1u;
      read_box(&nodes[first == last ? leaf_off + first : (gr > gl ? last : first)], box);
#pragma unroll
      for (int k = 0; k < 6; ++k) bx[k * 2u * kMidItems + i] = box[k];
    }
    for (;;) {
      const bool is_left = gr > gl;
      const uint32_t s = is_left ? r : l - 1u;
      if (is_left ? r == count - 1u : l == 0u) {  // the sibling is in another group
        next[atomicAdd(num_next, 1u) & ~kLongLists] = make_uint2(pos[l], pos[r + 1u] - 1u);
        break;
      }
      __threadfence_block();
      const uint32_t other = atomicExch(&slot[s], is_left ? l + 1u : (r + 1u) | kRight);
      if (other == 0u) break;
      __threadfence_block();
      slot[s] = 0u;
      const uint32_t far = (other & (kRight - 1u)) - 1u;
      uint32_t sib;
      if (is_left) {
        sib = far == s + 1u ? far : kMidItems + s + 1u;
        r = far;
        gr = gap[far + 1u];
      } else {
        sib = far == s ? s : kMidItems + s;
        l = far;
        gl = gap[far];
      }
      const bool root = (gl & gr) < 0, left = gr > gl;
      const uint32_t at = root ? 0u : (left ? r : l);
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const float b = bx[k * 2u * kMidItems + sib];
        box[k] = (k & 1) ? fmaxf(box[k], b) : fminf(box[k], b);
        bx[k * 2u * kMidItems + kMidItems + at] = box[k];
      }
      const uint32_t first = pos[l], cut = pos[s + 1u], last = pos[r + 1u] - 1u;
      write_inner(&nodes[root ? 0u : (left ? last : first)], box, first == cut - 1u ? leaf_off + first : cut - 1u,
                  cut == last ? leaf_off + last : cut);
      if (root) break;
    }
  }
  __syncthreads();
  for (uint32_t i = t; i < count; i += kMidThreads) {  // visitors that met nobody
    const uint32_t tag = slot[i];
    if (tag == 0u) continue;
    const uint32_t far = (tag & (kRight - 1u)) - 1u;
    const uint32_t l = (tag & kRight) ? i + 1u : far, r = (tag & kRight) ? far : i;
    next[atomicAdd(num_next, 1u) & ~kLongLists] = make_uint2(pos[l], pos[r + 1u] - 1u);
  }
}

__global__ void __launch_bounds__(kMidThreads) k_mid(uint32_t n, const uint32_t* __restrict__ codes,
                                                     const uint2* __restrict__ open,
                                                     const uint32_t* __restrict__ num_open, uint32_t* slots,
                                                     RtBVHNode40* nodes, uint2* __restrict__ next,
                                                     uint32_t* __restrict__ num_next) {
  grid_wait();
  extern __shared__ uint32_t sm[];
  __shared__ uint32_t warp_sums[kMidThreads / 32];
  const MidShared m = mid_shared(sm);
  uint32_t *slot = m.slot, *pos = m.pos, *bits = m.bits, *before = m.before;
  const uint32_t t = threadIdx.x, lane = t & 31u, w = t >> 5;
  const uint32_t base = blockIdx.x * kGroupLeaves, end = min(n, base + kGroupLeaves);
  const uint32_t count = num_open[blockIdx.x];
  open += (size_t)blockIdx.x * kGroupOpen;
  if (count > kMidItems) {
    if (gridDim.x == 1u)
      for (uint32_t i = t; i < count; i += kMidThreads) climb_global(open[i].x, open[i].y, n, codes, slots, nodes);
    else if (t == 0u)
      atomicOr(num_next, kLongLists);
    return;
  }
  const uint32_t words = (end - base + 31u) / 32u;
  for (uint32_t i = t; i < words; i += kMidThreads) bits[i] = 0u;
  for (uint32_t i = t; i < count; i += kMidThreads) slot[i] = 0u;
  __syncthreads();
  for (uint32_t i = t; i < count; i += kMidThreads) {
    const uint32_t l = open[i].x - base;
    atomicOr(&bits[l >> 5], 1u << (l & 31u));
  }
  __syncthreads();
  {
    const uint32_t i = 2u * t, c0 = i < words ? (uint32_t)__popc(bits[i]) : 0u,
                   c1 = i + 1u < words ? (uint32_t)__popc(bits[i + 1u]) : 0u;
    uint32_t v = c0 + c1;
#pragma unroll
    for (uint32_t off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, off);
      if (lane >= off) v += y;
    }
    if (lane == 31u) warp_sums[w] = v;
    __syncthreads();
    uint32_t b = v - c0 - c1;
    for (uint32_t k = 0; k < w; ++k) b += warp_sums[k];
    if (i < words) before[i] = b;
    if (i + 1u < words) before[i + 1u] = b + c0;
  }
  __syncthreads();
  for (uint32_t i = t; i < count; i += kMidThreads) {
    const uint32_t l = open[i].x - base;
    pos[before[l >> 5] + (uint32_t)__popc(bits[l >> 5] & ((1u << (l & 31u)) - 1u))] = base + l;
  }
  if (t == 0u) pos[count] = end;
  __syncthreads();
  climb_ranked(m, count, n, codes, nodes, next, num_next);
}

// The top of a tree of several groups: the nodes that k_mid's groups left, about
// ten each, ranked by counting, in one block.  Leaves the work to k_top when some
// group's list was too long.  They are never too many by themselves: they are one
// more than the nodes that reach over an edge between groups, and over each of the
// 47 edges of kLastGroups reach at most 36 (30 lengths of common prefix of two
// codes, six of two positions of one code), less the shared ones.
__device__ __forceinline__ bool fits_last(uint32_t num_next) { return num_next <= kMidItems; }

__global__ void __launch_bounds__(kMidThreads) k_last(uint32_t n, const uint32_t* __restrict__ codes,
                                                      uint2* __restrict__ next, uint32_t* __restrict__ num_next,
                                                      RtBVHNode40* nodes) {
  grid_wait();
  extern __shared__ uint32_t sm[];
  const MidShared m = mid_shared(sm);
  const uint32_t t = threadIdx.x, count = *num_next;
  if (!fits_last(count)) return;
  uint32_t* first = m.slot;  // unranked, until the ranks are known
  for (uint32_t i = t; i < count; i += kMidThreads) first[i] = next[i].x;
  __syncthreads();
  for (uint32_t i = t; i < count; i += kMidThreads) {
    const uint32_t l = first[i];
    uint32_t rank = 0u;
    for (uint32_t j = 0; j < count; ++j) rank += first[j] < l ? 1u : 0u;
    m.pos[rank] = l;
  }
  if (t == 0u) m.pos[count] = n;
  __syncthreads();
  for (uint32_t i = t; i < count; i += kMidThreads) m.slot[i] = 0u;
  __syncthreads();
  climb_ranked(m, count, n, codes, nodes, next, num_next);
}

// One global slot per split: all of k_tree's lists (`all`), or what k_last left.
// blockIdx.y: the group.
__global__ void __launch_bounds__(128) k_top(uint32_t n, const uint32_t* __restrict__ codes,
                                             const uint2* __restrict__ open, const uint32_t* __restrict__ num_open,
                                             const uint2* __restrict__ next, const uint32_t* __restrict__ num_next,
                                             bool all, uint32_t* slots, RtBVHNode40* nodes) {
  grid_wait();
  if (!all && fits_last(*num_next)) return;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  if (!all && blockIdx.y == 0u) {
    const uint32_t count = *num_next & ~kLongLists;
    for (uint32_t i = t; i < count; i += step) climb_global(next[i].x, next[i].y, n, codes, slots, nodes);
  }
  const uint32_t c = num_open[blockIdx.y];
  if (!all && c <= kMidItems) return;
  open += (size_t)blockIdx.y * kGroupOpen;
  for (uint32_t i = t; i < c; i += step) climb_global(open[i].x, open[i].y, n, codes, slots, nodes);
}

// Groups up to which k_mid and k_last finish the tree.  us for the whole build
// with them / with k_top over all lists: 262,144 primitives (4 groups) 91 / 102,
// 1,000,000 (16) 176 / 189, 2,000,000 (31) 275 / 289, 3,000,000 (46) 376 / 384,
// 4,194,304 (64) 501 / 489.
constexpr uint32_t kLastGroups = 48;

}  // namespace

// Cleared at the start: the centroid box (six words, two unused), the count of
// k_mid's list, those of k_tree's lists, then a slot per split.
constexpr size_t kClearWords = 9;

constexpr uint32_t tree_groups(uint32_t n) { return (n + kGroupLeaves - 1) / kGroupLeaves; }

size_t device_build_scratch_bytes(uint32_t n) {
  const uint32_t tiles = (n + tile_keys(n) - 1) / tile_keys(n);
  const size_t blocks = (n + kLeaves - 1) / kLeaves, groups = tree_groups(n);
  return 24 + kBins * 4 + (size_t)n * 4 * 4 + blocks * 8 + groups * kMidOpen * 8 + (size_t)kBins * tiles * 4 +
         (kClearWords + groups + (size_t)n) * 4;
}

// nodes: 2n-1 records; scratch: device_build_scratch_bytes(n).
cudaError_t launch_device_build(const RtTriangle64* tris, uint32_t nt, const RtSphere32* sph, uint32_t ns,
                                uint32_t mode, RtBVHNode40* nodes, void* scratch, cudaStream_t st) {
  const uint32_t n = nt + ns;
  if (n == 0) return cudaSuccess;
  char* p = static_cast<char*>(scratch);
  uint32_t* totals = reinterpret_cast<uint32_t*>(p);
  p += kBins * 4;
  uint32_t* ka = reinterpret_cast<uint32_t*>(p);
  p += (size_t)n * 4;
  uint32_t* va = reinterpret_cast<uint32_t*>(p);
  p += (size_t)n * 4;
  p = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15);
  // k_tree's list takes the sort's second buffers, which four passes leave
  // free: at most one entry per leaf and one more per block
  uint2* open = reinterpret_cast<uint2*>(p);
  uint32_t* kb = reinterpret_cast<uint32_t*>(p);
  p += (size_t)n * 4;
  uint32_t* vb = reinterpret_cast<uint32_t*>(p);
  p += (size_t)n * 4;
  const uint32_t blocks = (n + kLeaves - 1) / kLeaves, groups = tree_groups(n);
  p += (size_t)blocks * 8;
  uint2* next = reinterpret_cast<uint2*>((reinterpret_cast<uintptr_t>(p) + 7) & ~(uintptr_t)7);
  p = reinterpret_cast<char*>(next + (size_t)groups * kMidOpen);
  const uint32_t tile = tile_keys(n), tiles = (n + tile - 1) / tile;
  uint32_t* hist = reinterpret_cast<uint32_t*>(p);
  p += (size_t)kBins * tiles * 4;
  uint32_t* box = reinterpret_cast<uint32_t*>(p);
  uint32_t *num_next = box + kClearWords - 1, *num_open = num_next + 1, *slots = num_open + groups;
  const uint32_t cleared = 1u + groups + n;  // from num_next on

  const uint32_t sms = (uint32_t)device_sm_count();
  uint32_t *kin = ka, *vin = va, *kout = kb, *vout = vb;
  cudaError_t e;
  if (n <= kFrontMax) {
    const size_t smem = front_smem(n);
    e = cudaFuncSetAttribute(k_front, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)front_smem(kFrontMax));
    if (e != cudaSuccess) return e;
    e = launch_dependent(k_front, kFrontBlocks, kFrontThreads, smem, st, tris, sph, nt, n, mode, ka, va, num_next, cleared);
    if (e != cudaSuccess) return e;
  } else {
    e = cudaMemsetAsync(box, 0, (kClearWords - 1 + (size_t)cleared) * 4, st);
    if (e != cudaSuccess) return e;
    // the centroids take buffers that the sort's first pass does not read
    float *cx = reinterpret_cast<float*>(va), *cy = reinterpret_cast<float*>(kb), *cz = reinterpret_cast<float*>(vb);
    e = launch_dependent(k_centroids, std::min<uint32_t>((n + kT * 4 - 1) / (kT * 4), sms * 8u), kT, 0, st, tris, sph, nt,
                         n, cx, cy, cz, box);
    if (e == cudaSuccess)
      e = launch_dependent(k_morton, tiles, kT, 0, st, cx, cy, cz, n, box, mode, ka, hist, tiles, tile);
    for (int pass = 0; pass < 4 && e == cudaSuccess; ++pass) {
      const uint32_t shift = 8u * (uint32_t)pass;
      const uint32_t* v = pass ? vin : nullptr;
      if (pass) e = launch_dependent(k_rs_hist, tiles, kT, 0, st, kin, n, shift, hist, tiles, tile);
      if (e == cudaSuccess) e = launch_dependent(k_rs_scan, kBins, kT, 0, st, hist, tiles, totals);
      if (e == cudaSuccess)
        e = launch_dependent(tile == kT * kItemsSmall ? k_rs_scatter<kItemsSmall> : k_rs_scatter<kItemsLarge>, tiles, kT,
                             0, st, kin, v, n, shift, hist, totals, tiles, kout, vout);
      std::swap(kin, kout);
      std::swap(vin, vout);
    }
    if (e != cudaSuccess) return e;
  }
  e = launch_dependent(k_tree, blocks, kLeaves, 0, st, tris, sph, nt, n, mode, kin, vin, nodes, open, num_open);
  if (e == cudaSuccess && blocks > 1 && groups <= kLastGroups) {
    e = cudaFuncSetAttribute(k_mid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMidSmem);
    if (e == cudaSuccess)
      e = launch_dependent(k_mid, groups, kMidThreads, kMidSmem, st, n, kin, open, num_open, slots, nodes, next,
                           num_next);
    if (e == cudaSuccess && groups > 1)
      e = cudaFuncSetAttribute(k_last, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMidSmem);
    if (e == cudaSuccess && groups > 1)
      e = launch_dependent(k_last, 1, kMidThreads, kMidSmem, st, n, kin, next, num_next, nodes);
  }
  if (e == cudaSuccess && groups > 1)
    e = launch_dependent(k_top, dim3(16, groups), 128, 0, st, n, kin, open, num_open, next, num_next,
                         groups > kLastGroups, slots, nodes);
  return e;
}

}  // namespace rtgb

namespace rtgb {
namespace {

// Scratch of device builds comes from a pool of the library's own, one per
// context: the device's default pool gives its memory back at every
// synchronisation, and mapping it again cost a build after one 180 us (20,482
// triangles, build and wait: 247 us, 80 us with the pool).  It keeps at most
// kKeepBytes between builds -- scratch for 13 M primitives at 20.5 bytes each --
// and rt_stream_release hands that back.  Allocation and release are ordered on the
// caller's stream, as before.
//
// A pool goes with its context, and a later one may come at the same address
// (cudaDeviceReset); context ids are never used again, so a pool is found by the
// id alone.
constexpr uint64_t kKeepBytes = 256ull << 20;
std::mutex g_pool_mu;
std::map<unsigned long long, cudaMemPool_t> g_pools;

// Lets the calling thread make and trim the pool while it captures a stream: a
// capture refuses both otherwise, and is lost, although neither is part of it.
struct AllowInCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  AllowInCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~AllowInCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

cudaError_t context_id(int dev, unsigned long long* id) {
  using GetId = CUresult (*)(CUcontext, unsigned long long*);
  static const GetId get = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult r;
    const cudaError_t e = cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &r);
    return e == cudaSuccess && r == cudaDriverEntryPointSuccess ? reinterpret_cast<GetId>(f) : nullptr;
  }();
  if (!get) return cudaErrorNotSupported;
  if (get(nullptr, id) == CUDA_SUCCESS) return cudaSuccess;
  const cudaError_t e = cudaSetDevice(dev);  // a thread's first call, or one after a reset
  if (e != cudaSuccess) return e;
  return get(nullptr, id) == CUDA_SUCCESS ? cudaSuccess : cudaErrorDeviceUninitialized;
}

cudaError_t scratch_pool(cudaMemPool_t* out) {
  int dev = 0;
  unsigned long long id = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = context_id(dev, &id);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  auto it = g_pools.find(id);
  if (it == g_pools.end()) {
    const AllowInCapture allow;
    cudaMemPoolProps props;
    std::memset(&props, 0, sizeof(props));
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    if ((e = cudaMemPoolCreate(&pool, &props)) != cudaSuccess) return e;
    uint64_t keep = kKeepBytes;
    if ((e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess) {
      cudaMemPoolDestroy(pool);
      return e;
    }
    it = g_pools.emplace(id, pool).first;
  }
  *out = it->second;
  return cudaSuccess;
}

// The current context's pool; nullptr if no build has made one.
cudaMemPool_t existing_pool(int dev) {
  {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (g_pools.empty()) return nullptr;
  }
  unsigned long long id = 0;
  if (context_id(dev, &id) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  auto it = g_pools.find(id);
  return it == g_pools.end() ? nullptr : it->second;
}

}  // namespace

bool holds_build_scratch(int dev) { return existing_pool(dev) != nullptr; }

cudaError_t trim_build_scratch(int dev) {
  const cudaMemPool_t pool = existing_pool(dev);
  const AllowInCapture allow;
  return pool ? cudaMemPoolTrimTo(pool, 0) : cudaSuccess;
}

}  // namespace rtgb

using namespace rtgb;

extern "C" rt_status rt_build_bvh_device(const RtTriangle64* d_triangles, uint32_t num_triangles,
                                         const RtSphere32* d_spheres, uint32_t num_spheres, uint32_t bvh_mode,
                                         RtBVHNode40* d_nodes, void* stream) {
  const uint64_t n = (uint64_t)num_triangles + num_spheres;
  if ((num_triangles && !d_triangles) || (num_spheres && !d_spheres) || (n && !d_nodes) ||
      (bvh_mode != RT_BVH_SORTED && bvh_mode != RT_BVH_REFERENCE) || n > kMaxTriangles) {
    set_error("rt_build_bvh_device: bad argument");
    return RT_EINVAL;
  }
  if (n == 0) return RT_OK;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  void* scratch = nullptr;
  cudaMemPool_t pool = nullptr;
  cudaError_t e = scratch_pool(&pool);
  if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&scratch, device_build_scratch_bytes((uint32_t)n), pool, st);
  if (e != cudaSuccess) {
    set_error(std::string("rt_build_bvh_device: scratch: ") + cudaGetErrorString(e));
    return RT_ENOMEM;
  }
  e = launch_device_build(d_triangles, num_triangles, d_spheres, num_spheres, bvh_mode, d_nodes, scratch, st);
  cudaError_t e2 = cudaFreeAsync(scratch, st);
  if (e == cudaSuccess) e = e2;
  if (e != cudaSuccess) {
    set_error(std::string("rt_build_bvh_device: ") + cudaGetErrorString(e));
    return RT_ECUDA;
  }
  return RT_OK;
}
