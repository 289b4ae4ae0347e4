// gpu_build.cu -- the reference's S1 pass (RaytracerBVH.cpp:778-991) on the GPU.
//
// Same node layout and the same binary32 operations as the host builder
// (host_bvh.cpp), so the two emit identical 40-byte node arrays:
//   k_centroid_box   centroids ((v0+v1)+v2)/3, min/max fold from +-1e9
//                    (GetEnclosingAABB.comp:64-109); block reduction, then
//                    atomicMin/Max on order-preserving integer images of floats
//   k_pad_box        the padding of :105-109, one thread
//   k_morton         30-bit codes (GenerateMortonCodesOfPrimitives.comp:52-93)
//   radix sort       stable LSD sort of (code, index), 4 passes of 8 bits like
//                    RadixSortSimple.comp:8-13: per-tile histograms, a scan, and
//                    a scatter whose ranks keep input order (warp multi-split)
//   k_leaves         padded leaf boxes (ConstructHLBVH.comp:117-169)
//   k_karras         internal nodes: range and split (ConstructHLBVH.comp:72-209)
//   k_bottom_up      box unions, second arriving child continues upward
//                    (ConstructAABBsOfInternalNodes.comp:38-64)
#include <cuda_runtime.h>

#include <cstring>

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

__device__ __forceinline__ void centroid(const RtTriangle64* tris, const RtSphere32* sph, uint32_t nt, uint32_t i,
                                         float c[3]) {
  if (i < nt) {
    const RtTriangle64& t = tris[i];
    for (int k = 0; k < 3; ++k) c[k] = (t.v0[k] + t.v1[k] + t.v2[k]) / 3.0f;
  } else {
    const RtSphere32& s = sph[i - nt];
    for (int k = 0; k < 3; ++k) c[k] = s.center[k];
  }
}

__global__ void k_centroid_box(const RtTriangle64* tris, const RtSphere32* sph, uint32_t nt, uint32_t n,
                               uint32_t* box /* ord: min xyz, max xyz */) {
  float mn[3] = {1000000000.0f, 1000000000.0f, 1000000000.0f};
  float mx[3] = {-1000000000.0f, -1000000000.0f, -1000000000.0f};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float c[3];
    centroid(tris, sph, nt, i, c);
    for (int k = 0; k < 3; ++k) {
      mn[k] = fminf(mn[k], c[k]);
      mx[k] = fmaxf(mx[k], c[k]);
    }
  }
  for (int k = 0; k < 3; ++k)
    for (int o = 16; o > 0; o >>= 1) {
      mn[k] = fminf(mn[k], __shfl_down_sync(0xFFFFFFFFu, mn[k], o));
      mx[k] = fmaxf(mx[k], __shfl_down_sync(0xFFFFFFFFu, mx[k], o));
    }
  if ((threadIdx.x & 31u) == 0)
    for (int k = 0; k < 3; ++k) {
      atomicMin(&box[k], f2ord(mn[k]));
      atomicMax(&box[3 + k], f2ord(mx[k]));
    }
}

__global__ void k_pad_box(const uint32_t* ordbox, float* box) {
  const float delta = 0.001f, padding = delta / 2.0f;
  for (int k = 0; k < 3; ++k) {
    float mn = ord2f(ordbox[k]), mx = ord2f(ordbox[3 + k]);
    if (mx - mn < delta) {
      mn -= padding;
      mx += padding;
    }
    box[k] = mn;
    box[3 + k] = mx;
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

__global__ void k_morton(const RtTriangle64* tris, const RtSphere32* sph, uint32_t nt, uint32_t n, const float* box,
                         uint32_t mode, uint32_t* codes) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float c[3];
  centroid(tris, sph, nt, i, c);
  uint32_t q[3];
  for (int k = 0; k < 3; ++k) {
    const float span = box[3 + k] - box[k];
    const float off = mode == RT_BVH_REFERENCE ? c[k] / span : (c[k] - box[k]) / span;
    q[k] = f2u_sat(off * 1024.0f);
  }
  codes[i] = (spread3(q[2]) << 2) | (spread3(q[1]) << 1) | spread3(q[0]);
}

// ---- stable LSD radix sort, 8-bit digits ----
// A tile is 256 x ITEMS keys.  Per pass: k_rs_hist counts each tile's digits
// ([bin][tile]), k_rs_scan turns each bin's row into exclusive offsets (one
// block a bin) and leaves the bin's total, and k_rs_scatter adds the totals of
// lower bins, ranks its keys and writes them.  Bound by latency below about
// 10^5 keys and by L2 above (keys and indices of 4 M primitives, 67 MB with
// both copies, stay in L2).  The scan took 182 us a pass at 4,194,304 keys as
// one block over all 262,144 counts.  Whole build, before and after: 1,860 ->
// 1,094 us at 4,194,304 primitives, 187 -> 124 us at 20,482.
constexpr int kItemsLarge = 16;  // 4096-key tiles: 64-byte runs per digit on average
constexpr int kItemsSmall = 4;   // 1024-key tiles: four times the blocks
// Tiles of kItemsSmall up to here: at 1 M keys the large tiles are down to 256
// blocks, under two per SM.
constexpr uint32_t kSmallSort = 1u << 20;

constexpr uint32_t tile_keys(uint32_t n) { return kT * (n <= kSmallSort ? kItemsSmall : kItemsLarge); }

__global__ void __launch_bounds__(kT) k_rs_hist(const uint32_t* __restrict__ keys, uint32_t n, uint32_t shift,
                                                uint32_t* __restrict__ hist, uint32_t tiles, uint32_t tile) {
  __shared__ uint32_t h[kBins];
  h[threadIdx.x] = 0u;
  __syncthreads();
  const uint32_t base = blockIdx.x * tile;
#pragma unroll 4
  for (uint32_t j = threadIdx.x; j < tile; j += kT)
    if (base + j < n) atomicAdd(&h[(keys[base + j] >> shift) & 255u], 1u);
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
// (__match_any_sync), a per-warp count keeps earlier steps ahead.  The tile is
// put in digit order in shared memory first, so that a digit's keys leave as
// one run of consecutive addresses.  vals == nullptr: the value is the index
// (the first pass).
template <int ITEMS>
__global__ void __launch_bounds__(kT) k_rs_scatter(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals,
                                                   uint32_t n, uint32_t shift, const uint32_t* __restrict__ offs,
                                                   const uint32_t* __restrict__ totals, uint32_t tiles,
                                                   uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out) {
  constexpr int kWarps = kT / 32, kTile = kT * ITEMS;
  __shared__ uint32_t cnt[kWarps][kBins];
  __shared__ uint32_t sk[kTile], sv[kTile];
  __shared__ uint32_t to[kBins];  // output position of the digit's first key less its position in the tile
  __shared__ uint32_t warp_sums[kWarps];
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5, b = threadIdx.x;  // kT == kBins
  for (int i = lane; i < kBins; i += 32) cnt[w][i] = 0u;
  const uint32_t base = blockIdx.x * kTile, first = base + w * 32u * ITEMS + lane;
  const uint32_t live = min((uint32_t)kTile, n - base);
  uint32_t k[ITEMS], v[ITEMS], rank[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const uint32_t i = first + 32u * j;
    k[j] = i < n ? keys[i] : 0u;
    v[j] = i < n && vals ? vals[i] : i;
  }
  uint32_t all;
  const uint32_t bin_base = block_scan(totals[b], warp_sums, &all) + offs[b * tiles + blockIdx.x];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const bool ok = first + 32u * j < n;
    const uint32_t d = ok ? (k[j] >> shift) & 255u : 256u;
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
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
      sv[at] = v[j];
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

__device__ __forceinline__ void pad_axis(float& mn, float& mx) {
  const float delta = 0.001f, padding = delta / 2.0f;
  if (mx - mn < delta) {
    mn -= padding;
    mx += padding;
  }
}

__global__ void k_leaves(const RtTriangle64* tris, const RtSphere32* sph, uint32_t nt, uint32_t n, uint32_t mode,
                         const uint32_t* order, RtBVHNode40* nodes) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t g = mode == RT_BVH_REFERENCE ? k : order[k];
  RtBVHNode40 nd;
  if (g < nt) {
    const RtTriangle64& t = tris[g];
    nd.minX = fminf(t.v0[0], fminf(t.v1[0], t.v2[0]));
    nd.maxX = fmaxf(t.v0[0], fmaxf(t.v1[0], t.v2[0]));
    nd.minY = fminf(t.v0[1], fminf(t.v1[1], t.v2[1]));
    nd.maxY = fmaxf(t.v0[1], fmaxf(t.v1[1], t.v2[1]));
    nd.minZ = fminf(t.v0[2], fminf(t.v1[2], t.v2[2]));
    nd.maxZ = fmaxf(t.v0[2], fmaxf(t.v1[2], t.v2[2]));
    nd.primitiveIndex = g;
    nd.primitiveType = RT_PRIM_TRIANGLE;
  } else {
    const RtSphere32& s = sph[g - nt];
    float l[3], r[3];
    for (int a = 0; a < 3; ++a) {
      l[a] = s.center[a] - s.radius;
      r[a] = s.center[a] + s.radius;
    }
    nd.minX = fminf(l[0], r[0]);
    nd.maxX = fmaxf(l[0], r[0]);
    nd.minY = fminf(l[1], r[1]);
    nd.maxY = fmaxf(l[1], r[1]);
    nd.minZ = fminf(l[2], r[2]);
    nd.maxZ = fmaxf(l[2], r[2]);
    nd.primitiveIndex = g - nt;
    nd.primitiveType = RT_PRIM_SPHERE;
  }
  pad_axis(nd.minX, nd.maxX);
  pad_axis(nd.minY, nd.maxY);
  pad_axis(nd.minZ, nd.maxZ);
  nd.left = 0;
  nd.right = 0;
  nodes[(n - 1) + k] = nd;
}

__device__ __forceinline__ int delta(const uint32_t* codes, int n, int i, int j) {
  if (j < 0 || j > n - 1) return -1;
  const uint32_t ci = codes[i], cj = codes[j];
  if (ci == cj) return 32 + __clz((int)((uint32_t)i ^ (uint32_t)j));
  return __clz((int)(ci ^ cj));
}

__global__ void k_karras(const uint32_t* codes, uint32_t N, RtBVHNode40* nodes, uint32_t* parent, int* visits) {
  const int id = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int n = (int)N;
  if (id >= n - 1) return;
  const int dl = delta(codes, n, id, id - 1), dr = delta(codes, n, id, id + 1);
  const int dir = dr >= dl ? 1 : -1;
  const int dmin = min(dl, dr);
  int lmax = 2;
  while (delta(codes, n, id, id + lmax * dir) > dmin) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t > 0; t >>= 1)
    if (delta(codes, n, id, id + (l + t) * dir) > dmin) l += t;
  const int end = id + l * dir;
  const int first = min(id, end), last = max(id, end);
  const int common = delta(codes, n, first, last);
  int split = first, stride = last - first;
  do {
    stride = (stride + 1) >> 1;
    const int ns = split + stride;
    if (ns < last && delta(codes, n, first, ns) > common) split = ns;
  } while (stride > 1);
  const uint32_t leaf_off = N - 1;
  const uint32_t lc = (uint32_t)(split == first ? (int)leaf_off + split : split);
  const uint32_t rc = (uint32_t)(split + 1 == last ? (int)leaf_off + split + 1 : split + 1);
  RtBVHNode40 nd;
  nd.minX = nd.maxX = nd.minY = nd.maxY = nd.minZ = nd.maxZ = 0.0f;
  nd.left = lc;
  nd.right = rc;
  nd.primitiveIndex = 0;
  nd.primitiveType = 0;
  nodes[id] = nd;
  parent[lc] = (uint32_t)id;
  parent[rc] = (uint32_t)id;
  visits[id] = 0;
}

// Children's boxes are read with ld.global.cg (L2, not a stale L1 line).
__global__ void k_bottom_up(uint32_t N, RtBVHNode40* nodes, const uint32_t* parent, int* visits) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N || N < 2) return;
  uint32_t node = parent[(N - 1) + i];
  for (;;) {
    __threadfence();
    const int v = atomicAdd(&visits[node], 1);
    if (v < 1) return;
    RtBVHNode40* nd = &nodes[node];
    const uint32_t L = __ldcg(&nd->left), R = __ldcg(&nd->right);
    const float* a = reinterpret_cast<const float*>(&nodes[L]);
    const float* b = reinterpret_cast<const float*>(&nodes[R]);
    float r[6];
    for (int k = 0; k < 6; ++k) {
      const float x = __ldcg(&a[k]), y = __ldcg(&b[k]);
      r[k] = (k & 1) ? fmaxf(x, y) : fminf(x, y);
    }
    nd->minX = r[0]; nd->maxX = r[1]; nd->minY = r[2]; nd->maxY = r[3]; nd->minZ = r[4]; nd->maxZ = r[5];
    if (node == 0) return;
    node = parent[node];
  }
}

}  // namespace

size_t device_build_scratch_bytes(uint32_t n) {
  const uint32_t tiles = (n + tile_keys(n) - 1) / tile_keys(n);
  return 256 + kBins * 4 + (size_t)n * 4 * 4 + (size_t)kBins * tiles * 4 + (size_t)(2 * (size_t)n) * 4 * 2;
}

// nodes: 2n-1 records; scratch: device_build_scratch_bytes(n).
cudaError_t launch_device_build(const RtTriangle64* tris, uint32_t nt, const RtSphere32* sph, uint32_t ns,
                                uint32_t mode, RtBVHNode40* nodes, void* scratch, cudaStream_t st) {
  const uint32_t n = nt + ns;
  if (n == 0) return cudaSuccess;
  char* p = static_cast<char*>(scratch);
  uint32_t* ordbox = reinterpret_cast<uint32_t*>(p);
  float* box = reinterpret_cast<float*>(p + 64);
  p += 256;
  uint32_t* totals = reinterpret_cast<uint32_t*>(p);
  p += kBins * 4;
  uint32_t* ka = reinterpret_cast<uint32_t*>(p);
  p += (size_t)n * 4;
  uint32_t* va = reinterpret_cast<uint32_t*>(p);
  p += (size_t)n * 4;
  uint32_t* kb = reinterpret_cast<uint32_t*>(p);
  p += (size_t)n * 4;
  uint32_t* vb = reinterpret_cast<uint32_t*>(p);
  p += (size_t)n * 4;
  const uint32_t tile = tile_keys(n), tiles = (n + tile - 1) / tile;
  uint32_t* hist = reinterpret_cast<uint32_t*>(p);
  p += (size_t)kBins * tiles * 4;
  uint32_t* parent = reinterpret_cast<uint32_t*>(p);
  p += (size_t)(2 * (size_t)n) * 4;
  int* visits = reinterpret_cast<int*>(p);

  uint32_t init[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
  cudaError_t e = cudaMemcpyAsync(ordbox, init, sizeof(init), cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return e;
  const uint32_t gb = (n + kT - 1) / kT;
  k_centroid_box<<<std::min<uint32_t>(gb, 1024u), kT, 0, st>>>(tris, sph, nt, n, ordbox);
  k_pad_box<<<1, 1, 0, st>>>(ordbox, box);
  k_morton<<<gb, kT, 0, st>>>(tris, sph, nt, n, box, mode, ka);
  uint32_t *kin = ka, *vin = va, *kout = kb, *vout = vb;
  for (int pass = 0; pass < 4; ++pass) {
    const uint32_t shift = 8u * (uint32_t)pass;
    const uint32_t* v = pass ? vin : nullptr;
    k_rs_hist<<<tiles, kT, 0, st>>>(kin, n, shift, hist, tiles, tile);
    k_rs_scan<<<kBins, kT, 0, st>>>(hist, tiles, totals);
    if (tile == kT * kItemsSmall)
      k_rs_scatter<kItemsSmall><<<tiles, kT, 0, st>>>(kin, v, n, shift, hist, totals, tiles, kout, vout);
    else
      k_rs_scatter<kItemsLarge><<<tiles, kT, 0, st>>>(kin, v, n, shift, hist, totals, tiles, kout, vout);
    std::swap(kin, kout);
    std::swap(vin, vout);
  }
  k_leaves<<<gb, kT, 0, st>>>(tris, sph, nt, n, mode, vin, nodes);
  if (n > 1) {
    k_karras<<<gb, kT, 0, st>>>(kin, n, nodes, parent, visits);
    k_bottom_up<<<gb, kT, 0, st>>>(n, nodes, parent, visits);
  }
  return cudaGetLastError();
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
  cudaError_t e = cudaMallocAsync(&scratch, device_build_scratch_bytes((uint32_t)n), st);
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
