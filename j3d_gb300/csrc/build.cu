// build.cu -- GPU construction of the 4-wide BVH over an indexed triangle mesh.
//
// Replaces, in scene.cpp:20-23 (add_object), compute_triangle_normals,
// compute_bb (mesh.cpp:39-58) and `new jtk::qbvh(triangles, vertices)`.
//
// Pipeline (all on the context stream):
//   1. vertex bbox: two-pass min/max reduction (exact)
//   2. per triangle: normal (fixed fp32 order), AABB centroid -> 48-bit Morton
//      code over the vertex bbox
//   3. LSD radix sort of (Morton, triangle id), 8-bit digits, stable
//   4. leaf-ordered triangle array: 3 float4 per triangle (v0.w = id bits)
//   5. binary tree: by default binned-SAH splits top-down down to ranges of
//      at most J3DG_SAH_TOP triangles (section 5c), then PLOC clustering
//      within each range (section 5b), both by one block in shared memory
//      below kSmallTask triangles (section 5d); with J3DG_BUILD_LBVH the LBVH,
//      bottom-up in one pass
//      (Apetrei 2014, "Fast and Simple Agglomerative LBVH Construction"),
//      with a strict total order on the split keys (xor of neighbouring
//      codes, then i ^ (i+1), then i)
//   6. collapse to 4-wide nodes level by level: slots and leaves chosen by
//      the SAH cost programme of section 6b, which also tells every wide
//      node's place in depth-first order (LBVH: open the largest-area
//      child until four children, subtrees of <= leaf_size triangles become
//      leaves; then the wide nodes are renumbered depth-first, section 7).
// Child boxes are exact unions of triangle boxes, which the traversal's
// topology-independence argument requires.
#include <cuda_runtime.h>
#include <float.h>
#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "device_common.cuh"
#include "internal.h"

namespace j3dg {

static const int kMortonBitsPerAxis = 16;
static const int kRadixPasses = (3 * kMortonBitsPerAxis + 7) / 8;

// ------------------------------------------------------------- 1. bbox ----

__global__ void k_bbox_partial(const float* __restrict__ V, uint32_t nv, float* __restrict__ part) {
  float mn[3] = {3.4e38f, 3.4e38f, 3.4e38f}, mx[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float x = V[3 * (size_t)i + k];
      mn[k] = fminf(mn[k], x);
      mx[k] = fmaxf(mx[k], x);
    }
  }
  __shared__ float s[6][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    for (int o = 16; o > 0; o >>= 1) {
      mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
      mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
    }
  }
  if (lane == 0)
    for (int k = 0; k < 3; ++k) {
      s[k][warp] = mn[k];
      s[3 + k][warp] = mx[k];
    }
  __syncthreads();
  if (threadIdx.x < 6) {
    float v = s[threadIdx.x][0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
      v = threadIdx.x < 3 ? fminf(v, s[threadIdx.x][w]) : fmaxf(v, s[threadIdx.x][w]);
    part[6 * blockIdx.x + threadIdx.x] = v;
  }
}

// one block over at most 1024 partial boxes, one a thread (one warp walking
// them took 41 us)
__global__ void __launch_bounds__(1024) k_bbox_final(const float* __restrict__ part, int n, float* __restrict__ out) {
  __shared__ float s[6][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = min((int)threadIdx.x, n - 1);  // (a box read twice changes nothing)
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    float v = part[6 * b + k];
    for (int o = 16; o > 0; o >>= 1) {
      const float y = __shfl_xor_sync(0xffffffffu, v, o);
      v = k < 3 ? fminf(v, y) : fmaxf(v, y);
    }
    if (lane == 0) s[k][warp] = v;
  }
  __syncthreads();
  if (warp < 6) {
    float v = s[warp][lane];
    for (int o = 16; o > 0; o >>= 1) {
      const float y = __shfl_xor_sync(0xffffffffu, v, o);
      v = warp < 3 ? fminf(v, y) : fmaxf(v, y);
    }
    if (lane == 0) out[warp] = v;
  }
}

// ------------------------------------------------ 2. normals and Morton ----

// spreads the low 21 bits of x to every third bit (Morton interleave)
__device__ __forceinline__ uint64_t spread3(uint32_t x) {
  uint64_t v = x & 0x1fffffu;
  v = (v | (v << 32)) & 0x1f00000000ffffull;
  v = (v | (v << 16)) & 0x1f0000ff0000ffull;
  v = (v | (v << 8)) & 0x100f00f00f00f00full;
  v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
  v = (v | (v << 2)) & 0x1249249249249249ull;
  return v;
}

__global__ void k_tri_prep(const float* __restrict__ V, uint32_t nv, const uint32_t* __restrict__ T, uint32_t nt,
                           const float* __restrict__ bb, float4* __restrict__ normals, uint64_t* __restrict__ keys,
                           uint32_t* status) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nt) return;
  uint32_t a = T[3 * (size_t)i], b = T[3 * (size_t)i + 1], c = T[3 * (size_t)i + 2];
  if (a >= nv || b >= nv || c >= nv) {
    atomicOr(status, J3DG_DEV_BAD_INDEX);
    a = b = c = 0;
  }
  const float* A = V + 3 * (size_t)a;
  const float* B = V + 3 * (size_t)b;
  const float* C = V + 3 * (size_t)c;
  // jtk compute_triangle_normals: normalize(cross(V1 - V0, V2 - V0))
  float e1x = fs(B[0], A[0]), e1y = fs(B[1], A[1]), e1z = fs(B[2], A[2]);
  float e2x = fs(C[0], A[0]), e2y = fs(C[1], A[1]), e2z = fs(C[2], A[2]);
  float nx = fs(fm(e1y, e2z), fm(e1z, e2y));
  float ny = fs(fm(e1z, e2x), fm(e1x, e2z));
  float nz = fs(fm(e1x, e2y), fm(e1y, e2x));
  float len = __fsqrt_rn(dot3(nx, ny, nz, nx, ny, nz));
  if (len > 0.f) {
    nx = __fdiv_rn(nx, len);
    ny = __fdiv_rn(ny, len);
    nz = __fdiv_rn(nz, len);
  }
  normals[i] = make_float4(nx, ny, nz, 0.f);
  // Morton code of the AABB centroid over the vertex bbox
  const float scale = (float)(1u << kMortonBitsPerAxis);
  uint32_t q[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float lo = fminf(fminf(A[k], B[k]), C[k]), hi = fmaxf(fmaxf(A[k], B[k]), C[k]);
    float cen = (lo + hi) * 0.5f;
    float ext = bb[3 + k] - bb[k];
    float f = ext > 0.f ? (cen - bb[k]) / ext * scale : 0.f;
    f = fminf(fmaxf(f, 0.f), scale - 1.f);
    q[k] = (uint32_t)f;
  }
  keys[i] = (spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]);
}

// ------------------------------------------------------ 3. radix sort ----

// Least significant digit first, a kernel a digit: a block takes a tile, ranks
// its keys within their digits, and learns how many keys of each digit the
// tiles before it hold by looking back over what they have published
// (Adinets and Merrill 2022, "Onesweep: A Faster Least Significant Digit Radix
// Sort for GPUs"), so that a pass reads and writes the keys once; the totals
// of all digits come from one pass over the keys before.
//
// Measured (GB300), all six digits: 82k keys 60 us, 500k 84, 2M 159, 28.09M
// 1209 (of which the totals 8-75), where counting each tile's digits, scanning
// the counts of all tiles and then moving the keys, four kernels a digit, took
// 147 at 82k and 2250 at 28.09M. There a pass moves 674 MB in 189 us. Bound by
// the ranking (shared memory and votes) and the words looked back at; so a
// tile is as large as four blocks an SM carry: 16 keys a thread at 64
// registers (the values fetched once the keys have left theirs), against 1738
// us with 8 keys and 1740 with 16 and three blocks. match.any in place of the
// eight votes: 1988. Below 300k keys the tiles are too few for the SMs, and
// 4 keys a thread are faster (82k: 60 us against 72; 500k: 98 against 84).

static const int kSortItems = 16, kSortFew = 4;  // keys per thread
static const uint32_t kSortLarge = 300000u;      // from this many keys on
static const uint32_t kSortLook = 8;             // words looked at together

static const int kSortThreads = 256, kSortWarps = kSortThreads / 32;

// keys by every digit: totals[pass][256] (zero before)
__global__ void __launch_bounds__(512) k_radix_totals(const uint64_t* __restrict__ keys, uint32_t n,
                                                      uint32_t* __restrict__ totals) {
  __shared__ uint32_t h[kRadixPasses][256];
  for (uint32_t k = threadIdx.x; k < kRadixPasses * 256u; k += blockDim.x) (&h[0][0])[k] = 0;
  __syncthreads();
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += 4u * stride) {
    uint64_t k[4];
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
      const uint64_t i = (uint64_t)i0 + (uint64_t)j * stride;
      k[j] = i < n ? keys[i] : 0ull;
    }
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j)
      if ((uint64_t)i0 + (uint64_t)j * stride < n)
#pragma unroll
        for (int p = 0; p < kRadixPasses; ++p) atomicAdd(&h[p][(k[j] >> (8 * p)) & 255u], 1u);
  }
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < kRadixPasses * 256u; k += blockDim.x) {
    const uint32_t c = (&h[0][0])[k];
    if (c) atomicAdd(totals + k, c);
  }
}

// what a tile publishes per digit: its own count, then the count of all tiles
// up to it; one word, so no other memory is ordered by it
static const uint32_t kSortOwn = 1u << 30, kSortUpTo = 2u << 30, kSortCount = kSortOwn - 1u;
static_assert(J3DG_MAX_TRIANGLES <= kSortOwn, "a count beside the two flag bits");
static const uint32_t kSortPolls = 1u << 18;  // looks at a tile's word before the sort gives up (> 0.1 s)

template <int ITEMS>
struct SortMem {
  union {
    uint32_t count[kSortWarps][256];  // a warp's keys by digit, then the earlier warps'
    struct {
      uint64_t key[ITEMS * kSortThreads];
      uint32_t val[ITEMS * kSortThreads];
    };
  };
  uint32_t start[256];  // a digit's first key in the tile
  uint32_t place[256];  // ... its position in the output less that
  uint64_t wsum[kSortWarps];
  uint32_t tile;
};

// One digit (shift): keys and values (vin null: the positions) to kout (null:
// the keys are not needed any more) and vout. rows: 256 words a tile, zero
// before; tiles are taken in order (ticket, zero before), so those that a
// block waits for are running or done.
template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads, 4) k_radix_pass(const uint64_t* __restrict__ kin,
                                                             const uint32_t* __restrict__ vin,
                                                             uint64_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                             uint32_t n, int shift, const uint32_t* __restrict__ totals,
                                                             uint32_t* rows, uint32_t* ticket, uint32_t* status) {
  constexpr uint32_t kTile = ITEMS * kSortThreads;
  extern __shared__ __align__(16) uint8_t sort_raw[];
  SortMem<ITEMS>& s = *reinterpret_cast<SortMem<ITEMS>*>(sort_raw);
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, below = (1u << lane) - 1u;
  if (tid == 0) s.tile = atomicAdd(ticket, 1u);
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) s.count[w][tid] = 0u;
  const uint32_t total = totals[tid];
  __syncthreads();
  const uint32_t tile = s.tile;
  const uint64_t first = (uint64_t)tile * kTile;
  const uint32_t held = (uint32_t)min((uint64_t)kTile, (uint64_t)n - first);  // (the grid has a block per tile)
  // a warp's keys are consecutive, 32 at a time; past the end: the largest,
  // which come after the tile's others
  const uint32_t at = warp * (ITEMS * 32u) + lane;
  uint64_t key[ITEMS];
  uint32_t rank[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) key[j] = at + 32u * j < held ? kin[first + at + 32u * j] : ~0ull;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const uint32_t d = (uint32_t)(key[j] >> shift) & 255u;
    uint32_t peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const bool bit = (d >> b) & 1u;
      const uint32_t m = __ballot_sync(0xffffffffu, bit);
      peers &= bit ? m : ~m;
    }
    const uint32_t before = s.count[warp][d];
    __syncwarp();
    if ((peers & below) == 0u) s.count[warp][d] = before + __popc(peers);
    __syncwarp();
    rank[j] = before + __popc(peers & below);
  }
  __syncthreads();
  // thread d: digit d
  uint32_t own = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) {
    const uint32_t c = s.count[w][tid];
    s.count[w][tid] = own;
    own += c;
  }
  volatile uint32_t* const row = rows + (size_t)tile * 256u + tid;
  *row = own | (tile == 0u ? kSortUpTo : kSortOwn);
  // both exclusive scans over the digits in one: of the totals (high) and of
  // the tile's counts (low 16 bits)
  const uint64_t x = ((uint64_t)total << 16) | own;
  uint64_t incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += y;
  }
  if (lane == 31) s.wsum[warp] = incl;
  __syncthreads();
  uint64_t ex = incl - x;
#pragma unroll
  for (uint32_t w = 0; w < kSortWarps; ++w)
    if (w < warp) ex += s.wsum[w];
  const uint32_t start = (uint32_t)ex & 0xffffu;
  s.start[tid] = start;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const uint32_t d = (uint32_t)(key[j] >> shift) & 255u;
    rank[j] += s.start[d] + s.count[warp][d];
  }
  __syncthreads();  // the counts' memory becomes the tile's
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) s.key[rank[j]] = key[j];
  uint32_t val[ITEMS];  // (fetched here: the keys' registers are free)
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const uint32_t k = at + 32u * j;
    val[j] = k < held ? (vin ? vin[first + k] : (uint32_t)first + k) : 0u;
  }
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) s.val[rank[j]] = val[j];
  // the tiles before, several words at a time
  uint32_t earlier = 0;
  if (tile > 0u) {
    uint32_t t = tile, polls = 0;
    bool found = false;
    while (!found) {
      uint32_t v[kSortLook];
#pragma unroll
      for (uint32_t q = 0; q < kSortLook; ++q)
        v[q] = t > q ? *(volatile uint32_t*)(rows + (size_t)(t - 1u - q) * 256u + tid) : kSortUpTo + 0u;
#pragma unroll
      for (uint32_t q = 0; q < kSortLook; ++q) {
        if (found || v[q] < kSortOwn) break;  // nothing there yet: look again from it
        earlier += v[q] & kSortCount;
        --t;
        found = v[q] >= kSortUpTo;
      }
      if (!found && ++polls >= kSortPolls) {  // (a stuck tile: the places are wrong, none is out of range)
        atomicOr(status, J3DG_DEV_VISIT_CAP);
        break;
      }
    }
    *row = ((earlier + own) & kSortCount) | kSortUpTo;
  }
  s.place[tid] = (uint32_t)(ex >> 16) + earlier - start;
  __syncthreads();
  for (uint32_t i = tid; i < held; i += kSortThreads) {
    const uint64_t k = s.key[i];
    const uint32_t pos = s.place[(uint32_t)(k >> shift) & 255u] + i;
    if (pos < n) {
      if (kout) kout[pos] = k;
      vout[pos] = s.val[i];
    } else {
      atomicOr(status, J3DG_DEV_BAD_INDEX);
    }
  }
}

// ----------------------------------------------- 4. leaf-ordered triangles ----

__global__ void k_soup(const float* __restrict__ V, const uint32_t* __restrict__ T, const uint32_t* __restrict__ order,
                       uint32_t nt, uint32_t nv, float4* __restrict__ tris, uint32_t* status) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nt) return;
  uint32_t id = order ? order[i] : i;
  if (id >= nt) {
    atomicOr(status, J3DG_DEV_BAD_INDEX);
    id = 0;
  }
  uint32_t a = T[3 * (size_t)id], b = T[3 * (size_t)id + 1], c = T[3 * (size_t)id + 2];
  if (a >= nv || b >= nv || c >= nv) a = b = c = 0;
  tris[3 * (size_t)i] = make_float4(V[3 * (size_t)a], V[3 * (size_t)a + 1], V[3 * (size_t)a + 2], __uint_as_float(id));
  tris[3 * (size_t)i + 1] = make_float4(V[3 * (size_t)b], V[3 * (size_t)b + 1], V[3 * (size_t)b + 2], 0.f);
  tris[3 * (size_t)i + 2] = make_float4(V[3 * (size_t)c], V[3 * (size_t)c + 1], V[3 * (size_t)c + 2], 0.f);
}

// ------------------------------------------------------------- 5. LBVH ----

// A binary node. LBVH: node n splits between sorted leaves n and n + 1, the
// w fields are unused. The default builder keeps the two children's refs
// there (bit 31: a triangle, in Morton order), so that one 32-byte sector
// holds what the collapse follows.
struct BinNode {
  float4 lo, hi;
};
// ... and what the collapse's decisions need of it (default builder)
struct __align__(16) NodeMeta {
  uint32_t count;   // triangles
  uint32_t wide;    // wide nodes its subtree becomes unless it is a leaf
  uint32_t dec[2];  // the decisions of section 6b, a byte each
};
// a BinNode's children
__device__ __forceinline__ uint32_t left_ref(const float4& lo) { return __float_as_uint(lo.w); }
__device__ __forceinline__ uint32_t right_ref(const float4& hi) { return __float_as_uint(hi.w); }

__device__ __forceinline__ void leaf_box(const float4* __restrict__ tris, uint32_t i, float4& lo, float4& hi) {
  float4 a = tris[3 * (size_t)i], b = tris[3 * (size_t)i + 1], c = tris[3 * (size_t)i + 2];
  lo = make_float4(fminf(fminf(a.x, b.x), c.x), fminf(fminf(a.y, b.y), c.y), fminf(fminf(a.z, b.z), c.z), 0.f);
  hi = make_float4(fmaxf(fmaxf(a.x, b.x), c.x), fmaxf(fmaxf(a.y, b.y), c.y), fmaxf(fmaxf(a.z, b.z), c.z), 0.f);
}

// split order: smaller (xor, i ^ (i+1), i) merges first
__device__ __forceinline__ bool split_less(const uint64_t* __restrict__ k, uint32_t a, uint32_t b) {
  uint64_t xa = k[a] ^ k[a + 1], xb = k[b] ^ k[b + 1];
  if (xa != xb) return xa < xb;
  uint32_t sa = a ^ (a + 1), sb = b ^ (b + 1);
  if (sa != sb) return sa < sb;
  return a < b;
}

// child refs: bit 31 set = sorted leaf index, else binary node index
__global__ void k_lbvh(const uint64_t* __restrict__ keys, const float4* __restrict__ tris, uint32_t n,
                       uint2* __restrict__ child, BinNode* __restrict__ box, uint2* __restrict__ range,
                       uint32_t* __restrict__ other, uint32_t* __restrict__ root) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t l = i, r = i;
  uint32_t cur = 0x80000000u | i;
  float4 lo, hi;
  leaf_box(tris, i, lo, hi);
  for (;;) {
    uint32_t p, prev;
    bool as_left;
    if (l == 0 || (r != n - 1 && split_less(keys, r, l - 1))) {
      p = r;
      as_left = true;
      __stcg(&child[p].x, cur);
      __threadfence();
      prev = atomicExch(&other[p], l);
    } else {
      p = l - 1;
      as_left = false;
      __stcg(&child[p].y, cur);
      __threadfence();
      prev = atomicExch(&other[p], r);
    }
    if (prev == 0xffffffffu) return;  // first to arrive: the sibling finishes p
    __threadfence();
    if (as_left)
      r = prev;
    else
      l = prev;
    uint32_t sib = as_left ? __ldcg(&child[p].y) : __ldcg(&child[p].x);
    float4 slo, shi;
    if (sib & 0x80000000u) {
      leaf_box(tris, sib & 0x7fffffffu, slo, shi);
    } else {
      slo = __ldcg(&box[sib].lo);
      shi = __ldcg(&box[sib].hi);
    }
    lo = make_float4(fminf(lo.x, slo.x), fminf(lo.y, slo.y), fminf(lo.z, slo.z), 0.f);
    hi = make_float4(fmaxf(hi.x, shi.x), fmaxf(hi.y, shi.y), fmaxf(hi.z, shi.z), 0.f);
    __stcg(&box[p].lo, lo);
    __stcg(&box[p].hi, hi);
    __stcg(&range[p], make_uint2(l, r));
    cur = p;
    if (l == 0 && r == n - 1) {
      *root = p;
      return;
    }
  }
}

// --------------------------------------------------------- 6. collapse ----

struct CollapseItem {
  uint32_t bin;    // binary node index
  uint32_t wide;   // wide node index to fill
  uint32_t depth;
};

__device__ __forceinline__ float half_area(float4 lo, float4 hi) {
  float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
  return dx * dy + dy * dz + dz * dx;
}

// One binary node of the LBVH's 4-wide collapse: it becomes wide node
// it.wide, whose slots are its children, the largest-area child opened until
// four slots are filled (or every slot is small enough to be a leaf); the
// slots that stay internal get wide nodes (n_wide) and are queued for the
// next level (n_out). bound: the wide array's and the queue's size; an index
// past it raises J3DG_DEV_BAD_INDEX and is not written.
__device__ __forceinline__ void collapse_one(const uint2* __restrict__ child, const BinNode* __restrict__ box,
                                             const uint2* __restrict__ range, const float4* __restrict__ tris,
                                             const CollapseItem it, CollapseItem* __restrict__ qout,
                                             uint32_t* __restrict__ n_out, uint32_t* __restrict__ n_wide,
                                             float4* __restrict__ wide, uint32_t bound, uint32_t leaf_size,
                                             uint32_t* __restrict__ max_depth, uint32_t* __restrict__ status) {
  if (it.wide >= bound) {
    atomicOr(status, J3DG_DEV_BAD_INDEX);
    return;
  }
  uint32_t ref[4];
  float4 lo[4], hi[4];
  uint32_t cnt[4];
  int m = 0;
  auto load = [&](uint32_t r, int s) {
    ref[s] = r;
    if (r & 0x80000000u) {
      leaf_box(tris, r & 0x7fffffffu, lo[s], hi[s]);
      cnt[s] = 1;
    } else {
      lo[s] = box[r].lo;
      hi[s] = box[r].hi;
      uint2 rg = range[r];
      cnt[s] = rg.y - rg.x + 1;
    }
  };
  uint2 c = child[it.bin];
  load(c.x, 0);
  load(c.y, 1);
  m = 2;
  while (m < 4) {
    int best = -1;
    float ba = -1.f;
    for (int s = 0; s < m; ++s)
      if (cnt[s] > leaf_size) {
        float a = half_area(lo[s], hi[s]);
        if (a > ba) {
          ba = a;
          best = s;
        }
      }
    if (best < 0) break;
    uint2 cc = child[ref[best]];
    load(cc.y, m);
    load(cc.x, best);
    ++m;
  }
  float4* W = wide + 8 * (size_t)it.wide;
  float v[6][4];
  uint32_t out_ref[4];
  for (int s = 0; s < 4; ++s) {
    if (s < m) {
      v[0][s] = lo[s].x;
      v[1][s] = hi[s].x;
      v[2][s] = lo[s].y;
      v[3][s] = hi[s].y;
      v[4][s] = lo[s].z;
      v[5][s] = hi[s].z;
      if (cnt[s] <= leaf_size) {
        uint32_t first = (ref[s] & 0x80000000u) ? (ref[s] & 0x7fffffffu) : range[ref[s]].x;
        out_ref[s] = J3DG_LEAF_BIT | (first << 3) | (cnt[s] - 1u);
      } else {
        const uint32_t w = atomicAdd(n_wide, 1u);
        const uint32_t q = atomicAdd(n_out, 1u);
        if (w < bound && q < bound) {
          qout[q] = CollapseItem{ref[s], w, it.depth + 1};
        } else {
          atomicOr(status, J3DG_DEV_BAD_INDEX);
        }
        out_ref[s] = w;
      }
    } else {
      v[0][s] = v[2][s] = v[4][s] = 3.4e38f;
      v[1][s] = v[3][s] = v[5][s] = -3.4e38f;
      out_ref[s] = J3DG_EMPTY_REF;
    }
  }
  for (int k = 0; k < 6; ++k) W[k] = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
  W[6] = make_float4(__uint_as_float(out_ref[0]), __uint_as_float(out_ref[1]), __uint_as_float(out_ref[2]),
                     __uint_as_float(out_ref[3]));
  W[7] = make_float4(0.f, 0.f, 0.f, 0.f);
  atomicMax(max_depth, it.depth);
}

// One level of the collapse: the level's item count is read from the device
// (n_in_p) and the grid strides over it.
__global__ void k_collapse(const uint2* __restrict__ child, const BinNode* __restrict__ box,
                           const uint2* __restrict__ range, const float4* __restrict__ tris,
                           const CollapseItem* __restrict__ qin, const uint32_t* __restrict__ n_in_p,
                           CollapseItem* __restrict__ qout, uint32_t* __restrict__ n_out, uint32_t* __restrict__ n_wide,
                           float4* __restrict__ wide, uint32_t bound, uint32_t leaf_size, uint32_t* __restrict__ max_depth,
                           uint32_t* __restrict__ status) {
  const uint32_t n_in = *n_in_p;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n_in; t += gridDim.x * blockDim.x)
    collapse_one(child, box, range, tris, qin[t], qout, n_out, n_wide, wide, bound, leaf_size, max_depth, status);
}

// -------------------------------------------------------- 5b. PLOC ----
//
// Parallel locally-ordered clustering (Meister and Bittner 2018, "Parallel
// Locally-Ordered Clustering for Bounding Volume Hierarchy Construction") of
// a segment of at most J3DG_SAH_TOP triangles (section 5d runs it): the
// Morton-ordered leaves start as clusters; every cluster picks the cluster
// within kPlocRadius list positions whose union box has the smallest surface
// area (equal areas: the smaller position; with the pair order this is a
// total order, so the best pair is always mutual and every round merges);
// mutual pairs become a new binary node at the lower position; the list is
// compacted and the rounds repeat until one cluster is left. Subtrees are no
// longer Morton ranges, so the collapse below carries each subtree's first
// position in the new leaf order and writes the triangles there.

#ifndef J3DG_PLOC_RADIUS
#define J3DG_PLOC_RADIUS 8  // 2..64 measured on the torus frames: 8 visits the fewest nodes
#endif
static const int kPlocRadius = J3DG_PLOC_RADIUS;

__device__ __forceinline__ float merged_area(float4 alo, float4 ahi, float4 blo, float4 bhi) {
  const float dx = fmaxf(ahi.x, bhi.x) - fminf(alo.x, blo.x);
  const float dy = fmaxf(ahi.y, bhi.y) - fminf(alo.y, blo.y);
  const float dz = fmaxf(ahi.z, bhi.z) - fminf(alo.z, blo.z);
  const float a = dx * dy + dy * dz + dz * dx;
  return a == a ? a : FLT_MAX;  // boxes with NaN planes still get an order
}

// ------------------------------------------------ a build's loop state ----

static const uint32_t kMaxTopLevels = 1024;  // SAH levels of a tree, top and small together
static const uint32_t kMaxPlaceLevels = 128;

// In device memory. A level's kernels read their sizes from its entry and add
// to the next one's: level `base + k` for the k that the launch gives (the
// bases move only in the loops of a captured build). The first part is what
// the host reads.
struct BuildCtl {
  float bb[6];
  uint32_t n_wide, max_depth;
  uint32_t error;     // 1 SAH levels overran their bound, 2 PLOC, 4 placement / collapse
  uint32_t top_left;  // tasks that wait for more SAH levels than were launched
  uint32_t place[kMaxPlaceLevels + 1];  // subtrees to be placed, by level
  uint32_t root;                        // the binary tree's root
  uint32_t top_base, place_base;
  uint32_t place_jobs;                  // subtrees that a warp places
  uint32_t n_small, n_ranges;           // small tasks and finished ranges
  uint32_t next_job;                    // the next of them to be taken (k_small_tasks)
  struct Level {
    uint32_t tasks, items;
  };
  __align__(8) Level top[kMaxTopLevels + 1];
  // the LBVH's loops
  uint32_t lohi[2];  // the running pass's node range
  uint32_t n_in, n_out, place_levels;
  int32_t dfs_level;
  uint32_t level_end[kMaxPlaceLevels];  // wide nodes of level L end at level_end[L]
};
static const size_t kCtlHead = offsetof(BuildCtl, root);

// ------------------------------------------- 6b. cost-optimal collapse ----
//
// SAH cost of covering the subtree of binary node n with at most i = 1..4
// slots of a wide node (the dynamic programme of Ylitie, Karras and Laine
// 2017, "Efficient Incoherent Ray Traversal on GPUs Through Compressed Wide
// BVHs", section 3.1, for 4-wide nodes). A is half the surface area:
//   C(tri, i) = A(tri) c_t
//   C(n, 1)   = min(leaf: A(n) N(n) c_t if N(n) <= leaf_size,
//                   node: A(n) c_n + min_k C(left, k) + C(right, 4 - k))
//   C(n, i)   = min(C(n, i - 1), min_k C(left, k) + C(right, i - k))
// Children come before their parents: within a small task (section 5d) the
// costs are made as its nodes are; the top nodes follow level by level,
// deepest first. The decisions steer the collapse:
// dec.x = the k of the node case (bit 7 set: the leaf case is cheaper);
// dec.y, .z, .w for i = 2, 3, 4: 0 = as i - 1, else the k of the best split.

#ifndef J3DG_SAH_CTRI
#define J3DG_SAH_CTRI 0.5f  // cost of a triangle test relative to a node visit
#endif

// what the programme keeps of a subtree: C(n, 1..W), and how many wide nodes
// it becomes with 1..W slots (a triangle: none), from which every wide node's
// place in depth-first order follows before any is made
template <int W>
struct Covering {
  float cost[W + 1];
  uint32_t wide[W + 1];
  __device__ __forceinline__ void triangle(float half_area) {
#pragma unroll
    for (int i = 1; i <= W; ++i) {
      cost[i] = half_area * J3DG_SAH_CTRI;
      wide[i] = 0u;
    }
  }
};

// the programme's step at a node of half area A over N triangles from its
// children's coverings; M.dec: the W decision bytes (byte 0 = the k of the node
// case | 0x80 when the leaf case is cheaper; byte i - 1, i = 2..W: 0 = as
// i - 1, else the k of the best split)
template <int W>
__device__ __forceinline__ void collapse_step(const Covering<W>& l, const Covering<W>& r, float A, uint32_t N,
                                              uint32_t leaf_size, Covering<W>& c, NodeMeta& M) {
  float best = FLT_MAX;
  uint32_t bk = 1, bw = l.wide[1] + r.wide[W - 1];
#pragma unroll
  for (uint32_t k = 1; k < (uint32_t)W; ++k)
    if (l.cost[k] + r.cost[W - k] < best) {
      best = l.cost[k] + r.cost[W - k];
      bk = k;
      bw = l.wide[k] + r.wide[W - k];
    }
  const float node = A + best;  // c_n = 1
  const float leaf = N <= leaf_size ? A * (float)N * J3DG_SAH_CTRI : FLT_MAX;
  c.cost[1] = fminf(leaf, node);
  const bool is_leaf = leaf <= node && N <= J3DG_MAX_LEAF;  // (areas past the largest float: at equal costs)
  c.wide[1] = is_leaf ? 0u : 1u + bw;
  M.count = N;
  M.wide = 1u + bw;
  M.dec[0] = bk | (is_leaf ? 0x80u : 0u);
  M.dec[1] = 0u;
#pragma unroll
  for (uint32_t i = 2; i <= (uint32_t)W; ++i) {
    float v = c.cost[i - 1];
    uint32_t dk = 0, w = c.wide[i - 1];
#pragma unroll
    for (uint32_t k = 1; k < i; ++k)
      if (l.cost[k] + r.cost[i - k] < v) {
        v = l.cost[k] + r.cost[i - k];
        dk = k;
        w = l.wide[k] + r.wide[i - k];
      }
    c.cost[i] = v;
    c.wide[i] = w;
    M.dec[(i - 1) >> 2] |= dk << (8 * ((i - 1) & 3u));
  }
}

__device__ __forceinline__ uint32_t dec_byte(const NodeMeta& m, uint32_t i) {
  return (m.dec[i >> 2] >> (8 * (i & 3u))) & 0xffu;
}

struct PlaceItem {
  uint32_t bin;    // binary node index
  uint32_t wide;   // wide node index to fill
  uint32_t depth;
  uint32_t start;  // first leaf-order position of the subtree
};

// The collapse of k_collapse over a tree whose subtrees are not ranges of the
// sorted leaves: each slot carries its subtree's first position; leaves are
// written to tris_out at those positions in depth-first order (and the
// triangles' positions to slot_of). A wide node's place in depth-first order
// is its parent's, plus one, plus the wide nodes of the slots before it: the
// wide nodes are written where they stay.
//
// A lane makes a slot: it goes down from the wide node's binary node by the
// decisions, at most W steps of one load's latency each, and holds the slot's
// box when it arrives. The warp then writes its nodes and copies the
// triangles of its leaves from shared memory, whole lines at a time. Subtrees
// above kPlaceJob triangles go level by level; below, a warp places a whole
// subtree, so that what its nodes share (sectors of the binary tree, lines of
// the output) is used while it is near, and no queue in global memory is
// added to. With a lane per wide node (a stack of subtrees, a loop over its
// leaves' triangles: the latencies of some twenty loads) and levels down to
// the leaves the placement took 3.35 ms for 28.09M triangles (6.08M nodes),
// 365 us for 2M, 116 for 82k; a lane per slot, by levels, 3.31, 242 and 67;
// now 1.78 ms, 203 and 63.
template <int W>
struct PlaceMem {  // a warp's
  static constexpr int kRow = 8 * W + 4;  // a node's words, and a shift of the banks
  __align__(16) float node[32 / W * kRow];
  uint2 tri[32 * J3DG_MAX_LEAF];  // leaf triangles: from, to
};

// the wide nodes of `it` (lane / W of the warp's; valid: there is one);
// push(inner, count, item), for whole warps, takes the subtrees to be placed next
template <int W, class Push>
__device__ __forceinline__ void place_nodes(PlaceMem<W>& s, const BinNode* __restrict__ node,
                                            const NodeMeta* __restrict__ meta, const BinNode* __restrict__ tbox,
                                            const float4* __restrict__ tris, const PlaceItem it, const bool valid,
                                            uint32_t n_wide, float4* __restrict__ wide, float4* __restrict__ tris_out,
                                            uint32_t* __restrict__ slot_of, uint32_t nt, uint32_t* status, Push push) {
  static_assert(J3DG_NODE_F4(W) == 2 * W, "eight rows of W words");
  const uint32_t lane = threadIdx.x & 31u, slot = lane & (W - 1), group = lane / W;
  // to the slot-th of the subtrees that the decisions give
  uint32_t ref = it.bin, start = it.start, cnt = 1u, sub = 0u;  // sub: wide nodes in it (0: a leaf)
  bool has = valid;
  float4 lo = make_float4(3.4e38f, 3.4e38f, 3.4e38f, 0.f), hi = make_float4(-3.4e38f, -3.4e38f, -3.4e38f, 0.f);
  if (valid) {
    uint32_t i = W, at = slot;  // the slots that the subtree takes, ours among them
    for (int step = 0; step <= W; ++step) {
      if (ref & 0x80000000u) {  // a triangle takes one
        has = at == 0u;
        break;
      }
      const BinNode b = node[ref];
      const NodeMeta M = meta[ref];
      uint32_t k = 0;
      if (step == 0) {
        k = dec_byte(M, 0) & 0x7fu;
      } else {
        while (i > 1u && (k = dec_byte(M, i - 1u)) == 0u) --i;  // 0: as with a slot less
        if (at >= i || i <= 1u) {
          has = at == 0u;
          lo = b.lo;
          hi = b.hi;
          cnt = M.count;
          sub = (M.dec[0] & 0x80u) ? 0u : M.wide;
          break;
        }
      }
      const uint32_t l = left_ref(b.lo);
      if (at < k) {
        ref = l;
        i = k;
      } else {
        start += (l & 0x80000000u) ? 1u : meta[l].count;
        ref = right_ref(b.hi);
        at -= k;
        i -= k;
      }
    }
    if (has && (ref & 0x80000000u)) {
      const BinNode b = tbox[ref & 0x7fffffffu];
      lo = b.lo;
      hi = b.hi;
    }
  }
  if (!has) {
    sub = 0u;
    lo = make_float4(3.4e38f, 3.4e38f, 3.4e38f, 0.f);
    hi = make_float4(-3.4e38f, -3.4e38f, -3.4e38f, 0.f);
  }
  // the wide nodes before it
  uint32_t next = sub;
#pragma unroll
  for (int o = 1; o < W; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, next, o, W);
    if (slot >= (uint32_t)o) next += y;
  }
  next += it.wide + 1u - sub;
  const bool inner = sub != 0u;
  if (inner && next >= n_wide) atomicOr(status, J3DG_DEV_BAD_INDEX);  // (a malformed tree is stopped here)
  push(inner && next < n_wide, cnt, PlaceItem{ref, next, it.depth + 1, start});
  const uint32_t out_ref =
      inner ? next : (has ? J3DG_LEAF_BIT | (start << 3) | (cnt - 1u) : J3DG_EMPTY_REF);
  // the node: planes [6][W], refs [W], zeros
  {
    float* r = s.node + group * PlaceMem<W>::kRow + slot;
    r[0 * W] = lo.x;
    r[1 * W] = hi.x;
    r[2 * W] = lo.y;
    r[3 * W] = hi.y;
    r[4 * W] = lo.z;
    r[5 * W] = hi.z;
    r[6 * W] = __uint_as_float(out_ref);
    r[7 * W] = 0.f;
  }
  // the leaf's triangles, in depth-first order
  const uint32_t mine = has && !inner ? min(cnt, J3DG_MAX_LEAF) : 0u;
  uint32_t off = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, off, o);
    if (lane >= (uint32_t)o) off += y;
  }
  const uint32_t n_tri = __shfl_sync(0xffffffffu, off, 31);
  off -= mine;
  if (mine == 1u) {
    s.tri[off] = make_uint2(ref & 0x7fffffffu, start);
  } else if (mine) {
    uint32_t stk[J3DG_MAX_LEAF];
    int sp = 0;
    uint32_t k = 0;
    stk[sp++] = ref;
    while (sp > 0 && k < mine) {
      const uint32_t r = stk[--sp];
      if (r & 0x80000000u) {
        s.tri[off + k] = make_uint2(r & 0x7fffffffu, start + k);
        ++k;
      } else if (sp + 2 <= (int)J3DG_MAX_LEAF) {
        const BinNode b = node[r];
        stk[sp++] = right_ref(b.hi);
        stk[sp++] = left_ref(b.lo);
      } else {
        break;
      }
    }
    if (k < mine || sp > 0) atomicOr(status, J3DG_DEV_STACK_OVERFLOW);
    for (; k < mine; ++k) s.tri[off + k] = make_uint2(0xffffffffu, 0xffffffffu);
  }
  __syncwarp();
  // out: two float4 of the nodes a lane
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t y = lane + 32u * h, g = y / (2 * W), x = y % (2 * W);
    const uint32_t at = __shfl_sync(0xffffffffu, it.wide, (int)(g * W));
    const bool there = __shfl_sync(0xffffffffu, valid ? 1u : 0u, (int)(g * W));
    if (there) {
      if (at < n_wide)
        wide[2 * W * (size_t)at + x] = *reinterpret_cast<const float4*>(s.node + g * PlaceMem<W>::kRow + 4 * x);
      else
        atomicOr(status, J3DG_DEV_BAD_INDEX);
    }
  }
  for (uint32_t k = lane; k < 3u * n_tri; k += 32u) {
    const uint32_t e = k / 3u, part = k - 3u * e;
    const uint2 ft = s.tri[e];
    if (ft.x < nt && ft.y < nt) {
      const float4 v = tris[3 * (size_t)ft.x + part];
      tris_out[3 * (size_t)ft.y + part] = v;
      if (part == 0u) {
        const uint32_t id = __float_as_uint(v.w);
        if (id < nt)
          slot_of[id] = ft.y;
        else
          atomicOr(status, J3DG_DEV_BAD_INDEX);
      }
    } else {
      atomicOr(status, J3DG_DEV_BAD_INDEX);
    }
  }
  __syncwarp();  // the warp's memory is free for its next nodes
}

// ------------------------------------------------ 7. depth-first order ----
//
// The LBVH's collapse numbers wide nodes level by level, so the nodes on one
// ray's path from the root to a leaf lie far apart in memory (one per level,
// each level hundreds of MB wide at the bottom). Renumbering in depth-first
// order puts every subtree in one contiguous range: the deep part of a path,
// and the paths of neighbouring rays, then fall in the same few pages. Each
// level is a contiguous index range (a collapse launch allocates exactly the
// next level), so subtree sizes go bottom-up and new positions top-down, one
// launch per level. (The default builder knows every subtree's size before it
// makes the wide nodes, and places them in this order at once.)

template <int W>
__device__ __forceinline__ void child_refs(const float4* __restrict__ wide, uint32_t i, uint32_t (&r)[W]) {
  const float* f = reinterpret_cast<const float*>(wide + J3DG_NODE_F4(W) * (size_t)i) + 6 * W;
#pragma unroll
  for (int c = 0; c < W; ++c) r[c] = __float_as_uint(f[c]);
}

// size[i] = wide nodes in the subtree of i (children of level lo..hi are done)
template <int W>
__global__ void k_dfs_size(const float4* __restrict__ wide, const uint32_t* __restrict__ lohi,
                           uint32_t* __restrict__ size) {
  const uint32_t lo = lohi[0], hi = lohi[1];  // the level's nodes (device memory)
  for (uint32_t i = lo + blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += gridDim.x * blockDim.x) {
    uint32_t r[W], s = 1;
    child_refs<W>(wide, i, r);
#pragma unroll
    for (int c = 0; c < W; ++c)
      if (!(r[c] & J3DG_LEAF_BIT)) s += size[r[c]];  // the empty ref has the leaf bit
    size[i] = s;
  }
}

// children of the level's nodes take consecutive ranges after their parent
template <int W>
__global__ void k_dfs_place(const float4* __restrict__ wide, const uint32_t* __restrict__ lohi,
                            const uint32_t* __restrict__ size, uint32_t* __restrict__ pos) {
  const uint32_t lo = lohi[0], hi = lohi[1];  // the level's nodes (device memory)
  for (uint32_t i = lo + blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += gridDim.x * blockDim.x) {
    uint32_t r[W], next = pos[i] + 1;
    child_refs<W>(wide, i, r);
#pragma unroll
    for (int c = 0; c < W; ++c)
      if (!(r[c] & J3DG_LEAF_BIT)) {
        pos[r[c]] = next;
        next += size[r[c]];
      }
  }
}

template <int W>
__global__ void k_dfs_permute(const float4* __restrict__ wide, const uint32_t* __restrict__ n_p,
                              const uint32_t* __restrict__ pos, float4* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= *n_p) return;
  constexpr int F4 = J3DG_NODE_F4(W);
  const float4* src = wide + F4 * (size_t)i;
  float F[4 * F4];
#pragma unroll
  for (int k = 0; k < F4; ++k) {
    const float4 v = src[k];
    F[4 * k] = v.x, F[4 * k + 1] = v.y, F[4 * k + 2] = v.z, F[4 * k + 3] = v.w;
  }
#pragma unroll
  for (int c = 0; c < W; ++c) {
    const uint32_t r = __float_as_uint(F[6 * W + c]);
    if (!(r & J3DG_LEAF_BIT)) F[6 * W + c] = __uint_as_float(pos[r]);
  }
  float4* dst = out + F4 * (size_t)pos[i];
#pragma unroll
  for (int k = 0; k < F4; ++k) dst[k] = make_float4(F[4 * k], F[4 * k + 1], F[4 * k + 2], F[4 * k + 3]);
}

// the device-driven builder's fixed grids (grid-stride kernels)
static const uint32_t kStrideBlocks = 2048;

// one full wave of 128-thread blocks (16 per SM): the collapse kernels are
// chains of dependent loads per item, so every resident thread slot is used
static uint32_t wave_blocks128() {
  static uint32_t blocks = 0;
  if (!blocks) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    blocks = sms > 0 ? 16u * (uint32_t)sms : kStrideBlocks;
  }
  return blocks;
}

static const int kPlaceThreads = 128, kPlaceWarps = kPlaceThreads / 32;
// a subtree that one warp places: what waits of it are disjoint subtrees of
// two triangles and more, half as many at most
// (28.09M triangles, one wave of blocks: 32: 2.96 ms, 64: 2.22, 128: 1.89; the whole
// build with 256 0.46 ms longer than with 128)
static const uint32_t kPlaceJob = 128;

// level `base + k` of the placement: subtrees above kPlaceJob triangles to the
// next level, the others to the jobs; warp-uniform strides
template <int W>
__global__ void __launch_bounds__(kPlaceThreads) k_collapse_place(
    const BinNode* __restrict__ node, const NodeMeta* __restrict__ meta, const BinNode* __restrict__ tbox,
    const float4* __restrict__ tris, const PlaceItem* __restrict__ qin, PlaceItem* __restrict__ qout,
    PlaceItem* __restrict__ jobs, BuildCtl* __restrict__ c, uint32_t k, float4* __restrict__ wide,
    float4* __restrict__ tris_out, uint32_t* __restrict__ slot_of, uint32_t nt, uint32_t* status) {
  const uint32_t L = c->place_base + k;
  if (L >= kMaxPlaceLevels) return;
  __shared__ PlaceMem<W> mem[kPlaceWarps];
  const uint32_t n_in = min(c->place[L], nt), n_wide = c->n_wide, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t stride = gridDim.x * (kPlaceThreads / W), below = (1u << lane) - 1u;
  uint32_t depth = 0;
  for (uint32_t t0 = blockIdx.x * (kPlaceThreads / W) + warp * (32u / W); t0 < n_in; t0 += stride) {
    const uint32_t t = t0 + lane / W;
    const PlaceItem it = t < n_in ? qin[t] : PlaceItem{0u, 0u, 0u, 0u};
    depth = max(depth, it.depth);
    place_nodes<W>(mem[warp], node, meta, tbox, tris, it, t < n_in, n_wide, wide, tris_out, slot_of, nt, status,
                   [&](bool inner, uint32_t count, const PlaceItem& next) {
                     for (int job = 0; job < 2; ++job) {
                       const bool mine = inner && (count <= kPlaceJob) == (job == 1);
                       const uint32_t bal = __ballot_sync(0xffffffffu, mine);
                       if (!bal) continue;
                       uint32_t q = 0;
                       if (lane == 0u) q = atomicAdd(job ? &c->place_jobs : &c->place[L + 1], (uint32_t)__popc(bal));
                       q = __shfl_sync(0xffffffffu, q, 0) + __popc(bal & below);
                       if (!mine) continue;
                       if (q < (job ? nt / 2u : nt))  // (the arrays' ends: a malformed tree is stopped here)
                         (job ? jobs : qout)[q] = next;
                       else
                         atomicOr(status, J3DG_DEV_BAD_INDEX);
                     }
                   });
  }
  depth = __reduce_max_sync(0xffffffffu, depth);
  if (lane == 0u && depth > 0u) atomicMax(&c->max_depth, depth);
}

// the jobs, once the levels up to `base + k` have left nothing
template <int W>
__global__ void __launch_bounds__(kPlaceThreads) k_place_jobs(
    const BinNode* __restrict__ node, const NodeMeta* __restrict__ meta, const BinNode* __restrict__ tbox,
    const float4* __restrict__ tris, const PlaceItem* __restrict__ jobs, BuildCtl* __restrict__ c, uint32_t k,
    float4* __restrict__ wide, float4* __restrict__ tris_out, uint32_t* __restrict__ slot_of, uint32_t nt,
    uint32_t* status) {
  if (c->place[min(c->place_base + k, kMaxPlaceLevels)]) return;
  __shared__ PlaceMem<W> mem[kPlaceWarps];
  __shared__ PlaceItem wait[kPlaceWarps][kPlaceJob / 2];
  const uint32_t n_jobs = min(c->place_jobs, nt / 2u), n_wide = c->n_wide, lane = threadIdx.x & 31u,
                 warp = threadIdx.x >> 5, below = (1u << lane) - 1u;
  uint32_t depth = 0;
  for (uint32_t j = blockIdx.x * kPlaceWarps + warp; j < n_jobs; j += gridDim.x * kPlaceWarps) {
    uint32_t n = 1;  // waiting, the last ones first
    if (lane == 0u) wait[warp][0] = jobs[j];
    __syncwarp();
    while (n > 0u) {
      const uint32_t take = min(n, 32u / W), t = lane / W;
      const PlaceItem it = t < take ? wait[warp][n - 1u - t] : PlaceItem{0u, 0u, 0u, 0u};
      n -= take;
      depth = max(depth, it.depth);
      __syncwarp();
      place_nodes<W>(mem[warp], node, meta, tbox, tris, it, t < take, n_wide, wide, tris_out, slot_of, nt, status,
                     [&](bool inner, uint32_t, const PlaceItem& next) {
                       const uint32_t bal = __ballot_sync(0xffffffffu, inner), q = n + __popc(bal & below);
                       if (inner) {
                         if (q < kPlaceJob / 2u)
                           wait[warp][q] = next;
                         else
                           atomicOr(status, J3DG_DEV_BAD_INDEX);
                       }
                       n = min(n + __popc(bal), kPlaceJob / 2u);
                     });
    }
  }
  depth = __reduce_max_sync(0xffffffffu, depth);
  if (lane == 0u && depth > 0u) atomicMax(&c->max_depth, depth);
}

// -------------------------------------------------- 5c. SAH top levels ----
//
// Above J3DG_SAH_TOP triangles a node is split top-down by binned SAH (Wald
// 2007, "On fast Construction of SAH-based Bounding Volume Hierarchies"):
// every task (a range of the triangle order `ord`) bins its triangles'
// centroids into kTopBins bins per axis, one warp finds the split of least
// A_L N_L + A_R N_R from prefix and suffix unions of the bins (shuffles,
// lanes = bins), and a stable partition reorders the range. A stable
// partition of the Morton-sorted order keeps every range in Morton order, so
// each range of at most J3DG_SAH_TOP triangles (a segment) is then clustered
// by PLOC on its own (neighbours searched within the segment only).
// Tasks above kSmallTask triangles (small builds: kSmallTaskFew) are split
// level by level, each cut into items of at most `chunk` positions that a
// block bins and partitions; a smaller task is taken through the rest of its
// subtree by one block (section 5d).
//
// Binary nodes are numbered by position: the node that splits its range at
// position mid is node mid, and the nodes that PLOC makes in a segment take
// the segment's positions but the first: every position but position 0
// numbers one node, without a counter.

// Segment size below which PLOC takes over. Measured on the 28M-triangle torus
// frames (node visits per ray, ms per 1080p frame, ms of the build of that
// time): PLOC only 6.955 / 0.881 / 39; 4096: 6.402 / 0.862 / 67; 256: 6.256 /
// 0.855 / 76; 64: 6.200 / 0.851 / 87; 16: 6.193 / 0.852 / 112.
#ifndef J3DG_SAH_TOP
#define J3DG_SAH_TOP 64u
#endif
static_assert(J3DG_SAH_TOP > 0, "a segment has a triangle");
static const int kTopBins = 16;
static_assert(kTopBins <= 16, "bin codes keep 4 bits per axis");
// per bin: count, box lo / hi xyz (ordered-float encoded). The children's
// centroid ranges (the next level's bin ranges) are their boxes: every
// centroid lies in its triangle's box, and with triangles small against a
// task the two ranges differ by about one triangle
static const int kTopVals = 7;
static const uint32_t kNoTask = 0xffffffffu;
static const uint32_t kNoParent = 0xffffffffu;  // the parent of the root

struct TopTask {
  uint32_t begin, end;
  uint32_t parent;   // the node whose child it becomes (kNoParent: the root)
  uint32_t side;     // which child (bit 0) | the task's level << 1
  float4 clo, chi;  // centroid bounds
};

struct TopSplit {
  uint32_t axis;   // 3: split by position (no usable SAH split)
  uint32_t bin;    // bins 0..bin go left
  uint32_t nleft;
  uint32_t pad;
  uint32_t task[2];  // section 5d: the children's tasks of the next level (255: a finished range)
  uint32_t pad2[2];
  float4 lclo, lchi, rclo, rchi;  // children's centroid bounds
};

// triangle boxes by triangle, computed once for the SAH levels, and the order they start from
__global__ void k_top_boxes(const float4* __restrict__ tris, uint32_t n, BinNode* __restrict__ tbox,
                            uint32_t* __restrict__ ord) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 lo, hi;
  leaf_box(tris, i, lo, hi);
  tbox[i].lo = lo;
  tbox[i].hi = hi;
  ord[i] = i;
}

struct TopRange {  // a finished range: a segment for PLOC
  uint32_t begin, end, parent, side;  // parent and side as in TopTask
};

// the binary tree under construction
struct Tree {
  BinNode* node;
  NodeMeta* meta;
  uint32_t* up;      // a top node's parent (kNoParent: the root)
  uint32_t* done;    // a top node's finished children
  float* cost;       // coverings (W entries) of the top nodes and of the small tasks' roots
  uint32_t* wide;
  uint32_t* root;
  uint32_t* error;
};

// puts a finished subtree under its parent (or makes it the root)
__device__ __forceinline__ void link_child(const Tree& tr, uint32_t parent, uint32_t side, uint32_t ref) {
  if (parent == kNoParent)
    *tr.root = ref;
  else if (side & 1u)
    tr.node[parent].hi.w = __uint_as_float(ref);
  else
    tr.node[parent].lo.w = __uint_as_float(ref);
}

// float <-> uint32 with the same order (for atomic min / max)
__device__ __forceinline__ uint32_t f2o(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t o) { return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o); }

__device__ __forceinline__ int top_bin(float c, float lo, float hi) {
  const float ext = hi - lo;
  if (!(ext > 0.f)) return 0;
  const int b = (int)((c - lo) / ext * (float)kTopBins);
  return b < 0 ? 0 : (b >= kTopBins ? kTopBins - 1 : b);
}

// top_bin on three axes (packed 4 bits each, x lowest) by products with
// kTopBins / (hi - lo) instead of divisions: the two differ by under 4e-6, so
// away from a bin's edge the bin is the same; where an axis is within 1e-4 of
// an edge or out of the range (or NaN or infinite), the divisions decide
struct TopBinner {
  float lx, ly, lz, sx, sy, sz;
  __device__ __forceinline__ void set(const TopTask& T) {
    lx = T.clo.x, ly = T.clo.y, lz = T.clo.z;
    sx = (float)kTopBins / (T.chi.x - lx);
    sy = (float)kTopBins / (T.chi.y - ly);
    sz = (float)kTopBins / (T.chi.z - lz);
  }
  // q - 0.5 rounded to an integer is the floor of a q away from its edges;
  // the bits of 1.5 2^23 + that are the integer itself
  __device__ __forceinline__ static float floor_off(float q, uint32_t& b) {
    const float t = q - 0.5f, m = t + 12582912.f;
    b = __float_as_uint(m) - 0x4b400000u;
    return fabsf(t - (m - 12582912.f));
  }
  __device__ __forceinline__ uint32_t code(float cx, float cy, float cz, const TopTask& T) const {
    uint32_t bx, by, bz;
    const float ox = floor_off((cx - lx) * sx, bx), oy = floor_off((cy - ly) * sy, by),
                oz = floor_off((cz - lz) * sz, bz);
    if (!(ox < 0.4999f && oy < 0.4999f && oz < 0.4999f) || (bx | by | bz) >= (uint32_t)kTopBins) {
      bx = top_bin(cx, T.clo.x, T.chi.x);
      by = top_bin(cy, T.clo.y, T.chi.y);
      bz = top_bin(cz, T.clo.z, T.chi.z);
    }
    return bx | (by << 4) | (bz << 8);
  }
};

// Tasks up to this size leave the level loop for section 5d.
#ifndef J3DG_SMALL_TASK
#define J3DG_SMALL_TASK 960
#endif
static const uint32_t kSmallTask = J3DG_SMALL_TASK;
// ... of builds below kSmallFewBelow triangles, whose tasks are fewer than the
// SMs: two blocks of half the size are done sooner than one, and a level more
// costs less than that. Build and first frame with 480 / 960: 40k triangles
// 647 and 674 us, 120k 758 and 771, 250k 918 and 890; with 240 40k 654.
static const uint32_t kSmallTaskFew = 480, kSmallFewBelow = 130000;

__device__ __forceinline__ float box_half_area(float lx, float ly, float lz, float hx, float hy, float hz) {
  const float dx = hx - lx, dy = hy - ly, dz = hz - lz;
  return dx * dy + dy * dz + dz * dx;
}

// One warp: the split of least SAH cost A_L N_L + A_R N_R over the task's
// bins B ([axis][bin][kTopVals], in shared memory); writes the split,
// the node's box and its triangle count, and returns its left count
// (warp-uniform). Lanes b and b + 16 hold bin b of
// the axis in hand; prefix and suffix unions of the bins come from shuffles
// within the 16 lanes. Among equal costs the lowest (axis, bin) wins, the
// split a sweep over the axes and bins in order with a strict comparison
// takes. Bins with no triangle carry no box (their encoded fields would
// decode to NaN).
__device__ uint32_t warp_top_split(const uint32_t* B, const TopTask& T, TopSplit* split, const Tree& tr) {
  const uint32_t lane = threadIdx.x & 31u, b = lane & 15u;
  const uint32_t n = T.end - T.begin;
  float best = FLT_MAX;
  uint32_t best_idx = 0xffffffffu, best_lc = 0;
  float bl[3], bh[3], rl_best[3], rh_best[3];
  float nlo[3], nhi[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) bl[k] = bh[k] = rl_best[k] = rh_best[k] = nlo[k] = nhi[k] = 0.f;
  for (int ax = 0; ax < 3; ++ax) {
    const uint32_t* V = B + (ax * kTopBins + b) * kTopVals;
    const uint32_t c = V[0];
    float pl[3], ph[3], sl[3], sh[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      pl[k] = sl[k] = c ? o2f(V[1 + k]) : FLT_MAX;
      ph[k] = sh[k] = c ? o2f(V[4 + k]) : -FLT_MAX;
    }
    uint32_t pc = c, sc = c;
#pragma unroll
    for (int o = 1; o < kTopBins; o <<= 1) {  // inclusive prefix (bins 0..b) and suffix (bins b..15)
      const uint32_t yp = __shfl_up_sync(0xffffffffu, pc, o, kTopBins);
      const uint32_t ys = __shfl_down_sync(0xffffffffu, sc, o, kTopBins);
      float ypl[3], yph[3], ysl[3], ysh[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        ypl[k] = __shfl_up_sync(0xffffffffu, pl[k], o, kTopBins);
        yph[k] = __shfl_up_sync(0xffffffffu, ph[k], o, kTopBins);
        ysl[k] = __shfl_down_sync(0xffffffffu, sl[k], o, kTopBins);
        ysh[k] = __shfl_down_sync(0xffffffffu, sh[k], o, kTopBins);
      }
      if (b >= (uint32_t)o) {
        pc += yp;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          pl[k] = fminf(pl[k], ypl[k]);
          ph[k] = fmaxf(ph[k], yph[k]);
        }
      }
      if (b + (uint32_t)o < (uint32_t)kTopBins) {
        sc += ys;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          sl[k] = fminf(sl[k], ysl[k]);
          sh[k] = fmaxf(sh[k], ysh[k]);
        }
      }
    }
    // the right side of a split after bin b: the suffix from bin b + 1
    const uint32_t rc = __shfl_down_sync(0xffffffffu, sc, 1, kTopBins);
    float rl[3], rh[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      rl[k] = __shfl_down_sync(0xffffffffu, sl[k], 1, kTopBins);
      rh[k] = __shfl_down_sync(0xffffffffu, sh[k], 1, kTopBins);
    }
    if (ax == 0) {  // the node's box: the union of all bins of one axis
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        nlo[k] = __shfl_sync(0xffffffffu, sl[k], 0, kTopBins);
        nhi[k] = __shfl_sync(0xffffffffu, sh[k], 0, kTopBins);
      }
    }
    if (b + 1 < (uint32_t)kTopBins && pc != 0 && rc != 0) {
      const float cost = box_half_area(pl[0], pl[1], pl[2], ph[0], ph[1], ph[2]) * (float)pc +
                         box_half_area(rl[0], rl[1], rl[2], rh[0], rh[1], rh[2]) * (float)rc;
      if (cost < best) {
        best = cost;
        best_idx = (uint32_t)ax * kTopBins + b;
        best_lc = pc;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          bl[k] = pl[k];
          bh[k] = ph[k];
          rl_best[k] = rl[k];
          rh_best[k] = rh[k];
        }
      }
    }
  }
  // lowest (cost, axis, bin) over the warp
  float wc = best;
  uint32_t wi = best_idx;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float oc = __shfl_xor_sync(0xffffffffu, wc, o);
    const uint32_t oi = __shfl_xor_sync(0xffffffffu, wi, o);
    if (oc < wc || (oc == wc && oi < wi)) {
      wc = oc;
      wi = oi;
    }
  }
  // the left count: the winner's, or half for a split by position
  const uint32_t win = __ballot_sync(0xffffffffu, best_idx == wi);
  const uint32_t left = __shfl_sync(0xffffffffu, best_lc, __ffs(win) - 1);
  const uint32_t nleft = wi == 0xffffffffu ? n / 2 : left;
  if (wi == 0xffffffffu) {  // no usable SAH split: split by position
    if (lane == 0) {
      TopSplit S;
      S.axis = 3;
      S.bin = 0;
      S.nleft = n / 2;
      S.pad = 0;
      S.task[0] = S.task[1] = 0;
      S.pad2[0] = S.pad2[1] = 0;
      S.lclo = S.rclo = T.clo;
      S.lchi = S.rchi = T.chi;
      *split = S;
    }
  } else if (lane < (uint32_t)kTopBins && best_idx == wi) {
    TopSplit S;
    S.axis = wi / kTopBins;
    S.bin = wi % kTopBins;
    S.nleft = best_lc;
    S.pad = 0;
    S.task[0] = S.task[1] = 0;
    S.pad2[0] = S.pad2[1] = 0;
    S.lclo = make_float4(bl[0], bl[1], bl[2], 0.f);
    S.lchi = make_float4(bh[0], bh[1], bh[2], 0.f);
    S.rclo = make_float4(rl_best[0], rl_best[1], rl_best[2], 0.f);
    S.rchi = make_float4(rh_best[0], rh_best[1], rh_best[2], 0.f);
    *split = S;
  }
  if (lane == 0) {
    const uint32_t node = T.begin + nleft;
    tr.node[node].lo = make_float4(nlo[0], nlo[1], nlo[2], 0.f);
    tr.node[node].hi = make_float4(nhi[0], nhi[1], nhi[2], 0.f);
    tr.meta[node].count = n;
  }
  return nleft;
}

// Work of a level: items of at most `chunk` positions of one task. A task's
// items are consecutive; a task of one item is split and partitioned by the
// block that bins it.
struct TopItem {
  uint32_t task, first;  // the task's first item
  uint32_t begin, n;     // positions
};
static const int kLevelThreads = 256;
static const uint32_t kTopBinWords = 3 * kTopBins * kTopVals;
static const uint32_t kTopBinRow = kTopBinWords + 4;  // a task's bins in global memory, then its items done

__device__ __forceinline__ uint32_t top_bin_empty(uint32_t k) {  // word k of a task's empty bins
  const uint32_t v = k % kTopVals;
  return v == 0 ? 0u : (v < 4 ? 0xffffffffu : 0u);  // lo fields: max code, hi fields: 0
}

// the first level: the root task's items and empty bins
__global__ void k_top_items(TopItem* __restrict__ items, uint32_t* __restrict__ bins, uint32_t nt, uint32_t chunk) {
  const uint32_t n_items = (nt + chunk - 1) / chunk;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_items; i += gridDim.x * blockDim.x)
    items[i] = TopItem{0u, 0u, i * chunk, min(chunk, nt - i * chunk)};
  if (blockIdx.x == 0)
    for (uint32_t k = threadIdx.x; k < kTopBinRow; k += blockDim.x) bins[k] = k < kTopBinWords ? top_bin_empty(k) : 0u;
}

// adds a box of ordered-float codes (n of them) to a bin
__device__ __forceinline__ void bin_update(uint32_t* b, uint32_t n, const uint32_t (&v)[6]) {
  atomicAdd(b, n);
#pragma unroll
  for (int k = 0; k < 3; ++k) atomicMin(b + 1 + k, v[k]);
#pragma unroll
  for (int k = 3; k < 6; ++k) atomicMax(b + 1 + k, v[k]);
}

// ... in shared memory: most boxes lie within what the bin has gathered, and a
// look (broadcast to the lanes of one bin) costs less than an addition
// (one lane of a bin after the other): k_top_bin's levels of 28.09M triangles
// 6.84 -> 6.28 ms, k_small_tasks 6.52 -> 6.43
__device__ __forceinline__ void bin_update_shared(uint32_t* b, uint32_t n, const uint32_t (&v)[6]) {
  atomicAdd(b, n);
  volatile uint32_t* r = b;
  uint32_t x[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) x[k] = r[1 + k];
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (v[k] < x[k]) atomicMin(b + 1 + k, v[k]);
#pragma unroll
  for (int k = 3; k < 6; ++k)
    if (v[k] > x[k]) atomicMax(b + 1 + k, v[k]);
}

// the same to the three bins of a code
__device__ __forceinline__ void bin_update3(uint32_t* __restrict__ bins, uint32_t code, uint32_t n, const uint32_t (&v)[6]) {
#pragma unroll
  for (uint32_t ax = 0; ax < 3; ++ax)
    bin_update_shared(bins + (ax * kTopBins + ((code >> (4 * ax)) & 15u)) * kTopVals, n, v);
}

// a run of the binning: the code that a thread's last positions share and what
// they gathered (boxes without NaN, whose minima and maxima order as their
// codes do)
struct BinRun {
  uint32_t at;  // the code, or kNoTask
  uint32_t n;
  float v[6];
  __device__ __forceinline__ void flush(uint32_t* __restrict__ bins) const {
    if (at == kNoTask) return;
    const uint32_t c[6] = {f2o(v[0]), f2o(v[1]), f2o(v[2]), f2o(v[3]), f2o(v[4]), f2o(v[5])};
    bin_update3(bins, at, n, c);
  }
  __device__ __forceinline__ void add(uint32_t* __restrict__ bins, uint32_t code, const float (&x)[6]) {
    if (code != at) {
      flush(bins);
      at = code;
      n = 1;
#pragma unroll
      for (int k = 0; k < 6; ++k) v[k] = x[k];
    } else {
      ++n;
#pragma unroll
      for (int k = 0; k < 3; ++k) v[k] = fminf(v[k], x[k]);
#pragma unroll
      for (int k = 3; k < 6; ++k) v[k] = fmaxf(v[k], x[k]);
    }
  }
  // the runs of a whole warp at its end: one update per distinct code where
  // they are few (each costs a round of reductions), else one per lane
  __device__ __forceinline__ void flush_warp(uint32_t* __restrict__ bins) const {
    const uint32_t g = __match_any_sync(0xffffffffu, at), lane = threadIdx.x & 31u;
    const bool leader = lane == (uint32_t)__ffs(g) - 1u;
    if (__popc(__ballot_sync(0xffffffffu, leader)) > 8) {
      flush(bins);
      return;
    }
    const uint32_t c[6] = {f2o(v[0]), f2o(v[1]), f2o(v[2]), f2o(v[3]), f2o(v[4]), f2o(v[5])};
    uint32_t r[6];
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] = __reduce_min_sync(g, c[k]);
#pragma unroll
    for (int k = 3; k < 6; ++k) r[k] = __reduce_max_sync(g, c[k]);
    const uint32_t m = __reduce_add_sync(g, n);
    if (at != kNoTask && leader) bin_update3(bins, at, m, r);
  }
};

// the exclusive scan of per-pass, per-warp counts in s_cnt[K][8] (in place), by the first warp
template <int K>
__device__ __forceinline__ void scan_counts(uint32_t* s_cnt) {
  constexpr uint32_t n = K * (kLevelThreads / 32);
  static_assert(n <= 64, "two counts a lane");
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t x = lane < n ? s_cnt[lane] : 0u, y = lane + 32u < n ? s_cnt[lane + 32u] : 0u;
  uint32_t xi = x, yi = y;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, xi, o), v = __shfl_up_sync(0xffffffffu, yi, o);
    if (lane >= (uint32_t)o) {
      xi += u;
      yi += v;
    }
  }
  const uint32_t half = __shfl_sync(0xffffffffu, xi, 31);
  if (lane < n) s_cnt[lane] = xi - x;
  if (lane + 32u < n) s_cnt[lane + 32u] = half + yi - y;
}

// 1 if a position (the k-th of task T) goes left: its bin on the split axis
// (the bin codes that binning wrote: 4 bits per axis) is at most the split
// bin, or, for a split by position, it lies in the first nleft positions
__device__ __forceinline__ bool top_goes_left(uint32_t k, uint32_t code, const TopSplit& S) {
  return S.axis < 3 ? ((code >> (4 * S.axis)) & 15u) <= S.bin : k < S.nleft;
}

// Stable partition of an item's n positions (from position p0 of its task,
// which begins at `begin`): left0 of the task's earlier positions go left.
// Whole block; code and o: of the thread's positions, the j-th the item's
// (j kLevelThreads + tid)-th.
template <int K>
__device__ __forceinline__ void partition_item(const TopSplit& S, uint32_t begin, uint32_t p0, uint32_t n, uint32_t end,
                                               uint32_t left0, uint32_t* s_cnt, const uint32_t (&code)[K],
                                               const uint32_t (&o)[K], uint32_t* __restrict__ ord2, uint32_t* status) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  uint32_t f = 0;
#pragma unroll
  for (int j = 0; j < K; ++j) {
    const uint32_t k = (uint32_t)j * kLevelThreads + tid;
    const bool left = k < n && top_goes_left(p0 + k, code[j], S);
    f |= (left ? 1u : 0u) << j;
    const uint32_t c = __popc(__ballot_sync(0xffffffffu, left));
    if (lane == 0) s_cnt[j * (kLevelThreads / 32) + warp] = c;
  }
  __syncthreads();
  if (warp == 0) scan_counts<K>(s_cnt);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < K; ++j) {
    const uint32_t k = (uint32_t)j * kLevelThreads + tid;
    const bool left = (f >> j) & 1u;
    const uint32_t bal = __ballot_sync(0xffffffffu, left);
    if (k >= n) continue;
    const uint32_t l = left0 + s_cnt[j * (kLevelThreads / 32) + warp] + __popc(bal & ((1u << lane) - 1u));
    const uint32_t d = begin + (left ? l : S.nleft + (p0 + k - l));
    if (d < end)
      ord2[d] = o[j];
    else
      atomicOr(status, J3DG_DEV_BAD_INDEX);
  }
}

// where a level's tasks leave the next level's
struct NextLevel {
  TopTask* tasks;
  TopItem* items;
  uint32_t* bins;
  TopTask* small;
  TopRange* ranges;
  uint32_t cap_tasks, cap_small, cap_items, nt;
  uint32_t small_max;  // tasks up to this size are one block's
};

// One warp, after the split S of task T: the children, lanes 0 and 1 one
// each: a task of the next level above small_max triangles (with its items
// and, if they are several, empty bins), a small task above J3DG_SAH_TOP, else
// a finished range; the task's own node goes under its parent.
__device__ void warp_children(const TopTask& T, const TopSplit& S, uint32_t chunk, const NextLevel& N,
                              BuildCtl* __restrict__ c, uint32_t level, const Tree& tr, uint32_t* status) {
  const uint32_t lane = threadIdx.x & 31u, n = T.end - T.begin, nl = S.nleft;
  if (nl == 0 || nl >= n) {  // (a split leaves both sides something: bins with a triangle on both)
    if (lane == 0) {
      atomicOr(status, J3DG_DEV_BAD_INDEX);
      atomicOr(tr.error, 1u);
    }
    return;
  }
  const uint32_t node = T.begin + nl;
  const uint32_t b = (lane & 1u) ? node : T.begin, e = (lane & 1u) ? T.end : node, len = e - b;
  const uint32_t m = (len + chunk - 1) / chunk;
  uint32_t q = kNoTask, i0 = 0;
  if (lane < 2) {
    const uint32_t tag = lane | (((T.side >> 1) + 1u) << 1);
    if (len > J3DG_SAH_TOP) {
      const bool again = len > N.small_max;
      if (again) {  // the task and its items in one atomic
        const unsigned long long at = atomicAdd(reinterpret_cast<unsigned long long*>(&c->top[level + 1]),
                                                1ull | ((unsigned long long)m << 32));
        q = (uint32_t)at;
        i0 = (uint32_t)(at >> 32);
      } else {
        q = atomicAdd(&c->n_small, 1u);
      }
      if (q >= (again ? N.cap_tasks : N.cap_small) ||
          (again && (i0 + m > N.cap_items || level + 1u >= kMaxTopLevels))) {
        atomicOr(tr.error, 1u);
        q = kNoTask;
      } else {
        TopTask C;
        C.begin = b;
        C.end = e;
        C.parent = node;
        C.side = tag;
        C.clo = lane ? S.rclo : S.lclo;
        C.chi = lane ? S.rchi : S.lchi;
        (again ? N.tasks : N.small)[q] = C;
        if (!again) q = kNoTask;
      }
    } else {
      const uint32_t r = atomicAdd(&c->n_ranges, 1u);
      if (r < N.nt)
        N.ranges[r] = TopRange{b, e, node, tag};
      else
        atomicOr(tr.error, 1u);
    }
  }
  if (lane == 2) {
    tr.up[node] = T.parent;
    tr.done[node] = 0u;
    link_child(tr, T.parent, T.side, node);
  }
  for (int side = 0; side < 2; ++side) {
    const uint32_t qs = __shfl_sync(0xffffffffu, q, side), is = __shfl_sync(0xffffffffu, i0, side);
    const uint32_t ms = __shfl_sync(0xffffffffu, m, side), bs = __shfl_sync(0xffffffffu, b, side);
    const uint32_t ls = __shfl_sync(0xffffffffu, len, side);
    if (qs == kNoTask) continue;
    for (uint32_t k = lane; k < ms; k += 32u) N.items[is + k] = TopItem{qs, is, bs + k * chunk, min(chunk, ls - k * chunk)};
    if (ms > 1u)
      for (uint32_t k = lane; k < kTopBinRow; k += 32u)
        N.bins[(size_t)qs * kTopBinRow + k] = k < kTopBinWords ? top_bin_empty(k) : 0u;
  }
}

// Bins the items of a level. The item's boxes are staged in shared memory
// (neighbouring threads fetch neighbouring positions), then every thread bins
// a run of consecutive positions: in Morton order they mostly share their
// bins, so a run is gathered in registers and its bin updated when it ends.
// The bins of a task of several items are merged in global memory, and each
// item leaves its counts of bins 0..b per axis (icum, one row per axis and
// bin), from which its lefts follow for any split; the last of a task's items
// to be binned splits it. A task of one item is split and partitioned here.
//
// Bound: 32 B of box and 4 of order in, 2 or 4 out per triangle; staging them
// alone takes 8.9 ps a triangle (2.1M triangles in one task, 4.7 TB/s), the
// whole kernel 13.4, at 3000-triangle tasks 21. One update of the bins per
// run, and of all three axes together, is what counts: a run per axis took
// 17.6, the same with a bin's values encoded for every triangle and runs read
// across the banks 19.6. The pass that binned whole chunks of positions, with
// one warp reduction per 32 triangles and global atomics where a chunk held
// two tasks, took 0.43 ms a level at 28.09M triangles and, with the passes for
// flags, scan and scatter, 0.66; this kernel, the split and the scatter took
// 0.52, and 0.42 with the looks at the bins and the scatter's earlier fetches.
// Builds of 82k / 2M / 28.09M triangles with their first frame: 1449 ->
// 1230, 4201 -> 3729, 28412 -> 26443 us.
// the place of an item's k-th box in shared memory: threads read runs of 2, 4
// or 8 positions, and the low bits are mixed so that the threads of a half
// warp meet in no bank (a run of 8 boxes of 8 bytes spans half the banks)
__device__ __forceinline__ uint32_t top_slot(uint32_t k) { return (k & ~15u) | ((k ^ (k >> 4)) & 15u); }

template <int K>
struct TopBinMem {
  float2 box[3][K * kLevelThreads];
  __align__(16) uint16_t code[K * kLevelThreads];
  uint32_t bins[kTopBinWords];
  uint32_t cnt[64];
  uint32_t last;
  TopSplit split;
};
#ifndef J3DG_LEVEL_BLOCKS
#define J3DG_LEVEL_BLOCKS 4
#endif
// Smaller builds split a task where its last item was binned: a level is two
// launches (82k triangles: 12 + 4 us a level, against 7 + 6 + 3 and their
// gaps). Where a block bins many items, waiting for each one's additions to
// the task's bins before counting it costs more than a launch: 28.09M
// triangles 8.2 ms in the binning, against 6.9 and 0.2 for the splits.
template <int K>
constexpr bool kSplitWhereBinned = K < 8;

// K positions a thread: items of K * kLevelThreads; level `base + k`
template <int K>
__global__ void __launch_bounds__(kLevelThreads, J3DG_LEVEL_BLOCKS) k_top_bin(
    const uint32_t* __restrict__ ord, uint32_t* __restrict__ ord2, const BinNode* __restrict__ tbox,
    const TopItem* __restrict__ items, const TopTask* __restrict__ tasks, BuildCtl* __restrict__ c, uint32_t level_k,
    uint32_t* __restrict__ bins, uint16_t* __restrict__ code, uint32_t* __restrict__ icum,
    TopSplit* __restrict__ splits, const NextLevel next, const Tree tr, uint32_t* status) {
  constexpr uint32_t chunk = K * kLevelThreads;
  extern __shared__ __align__(16) uint8_t top_raw[];
  TopBinMem<K>& s = *reinterpret_cast<TopBinMem<K>*>(top_raw);
  uint32_t* const sb = s.bins;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t level = c->top_base + level_k, cap_items = next.cap_items;
  if (tid == 0) s.last = c->error;  // (other blocks may raise it meanwhile: one answer for the block)
  __syncthreads();
  if (level >= kMaxTopLevels || s.last) return;
  const uint32_t n_items = min(c->top[level].items, cap_items);
  for (uint32_t it = blockIdx.x; it < n_items; it += gridDim.x) {  // uniform over the block
    const TopItem I = items[it];
    const TopTask T = tasks[I.task];
    if (tid < 3 * kTopBins)
#pragma unroll
      for (int v = 0; v < kTopVals; ++v) sb[tid * kTopVals + v] = top_bin_empty(v);
    constexpr int kFlight = K < 4 ? K : 4;
#pragma unroll
    for (int j0 = 0; j0 < K; j0 += kFlight) {  // four boxes in flight per thread
      uint32_t t[kFlight];
#pragma unroll
      for (int j = 0; j < kFlight; ++j) {
        const uint32_t k = (uint32_t)(j0 + j) * kLevelThreads + tid;
        t[j] = k < I.n ? ord[I.begin + k] : 0u;
      }
      float4 lo[kFlight], hi[kFlight];
#pragma unroll
      for (int j = 0; j < kFlight; ++j) {  // (a position past the item reads triangle 0's box and drops it)
        lo[j] = tbox[t[j]].lo;
        hi[j] = tbox[t[j]].hi;
      }
#pragma unroll
      for (int j = 0; j < kFlight; ++j) {
        const uint32_t q = top_slot((uint32_t)(j0 + j) * kLevelThreads + tid);
        s.box[0][q] = make_float2(lo[j].x, hi[j].x);
        s.box[1][q] = make_float2(lo[j].y, hi[j].y);
        s.box[2][q] = make_float2(lo[j].z, hi[j].z);
      }
    }
    __syncthreads();
    {
      TopBinner B;
      B.set(T);
      BinRun r;
      r.at = kNoTask;
      r.n = 0;
#pragma unroll
      for (int k = 0; k < 6; ++k) r.v[k] = 0.f;
      const uint32_t k1 = min(I.n, tid * K + K);
      for (uint32_t k = tid * K; k < k1; ++k) {
        const uint32_t q = top_slot(k);
        const float2 x = s.box[0][q], y = s.box[1][q], z = s.box[2][q];
        const float v[6] = {x.x, y.x, z.x, x.y, y.y, z.y};
        const float cx = 0.5f * (x.x + x.y), cy = 0.5f * (y.x + y.y), cz = 0.5f * (z.x + z.y);
        const uint32_t cd = B.code(cx, cy, cz, T);
        s.code[k] = (uint16_t)cd;
        const float sum = cx + cy + cz;
        if (!(sum == sum)) {  // a NaN (or infinities of both signs): by the codes' order, which ranks NaN too
          const uint32_t c[6] = {f2o(v[0]), f2o(v[1]), f2o(v[2]), f2o(v[3]), f2o(v[4]), f2o(v[5])};
          bin_update3(sb, cd, 1u, c);
          continue;
        }
        r.add(sb, cd, v);
      }
      __syncwarp();
      r.flush_warp(sb);
    }
    __syncthreads();
    if (T.end - T.begin <= chunk) {
      // the whole task is here
      if (warp == 0) {
        warp_top_split(sb, T, &s.split, tr);
      }
      __syncthreads();
      uint32_t cd[K], o[K];
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const uint32_t k = (uint32_t)j * kLevelThreads + tid;
        o[j] = k < I.n ? ord[I.begin + k] : 0u;
        cd[j] = k < I.n ? s.code[k] : 0u;
      }
      partition_item<K>(s.split, T.begin, 0u, I.n, T.end, 0u, s.cnt, cd, o, ord2, status);
      if (warp == 0) {
        if constexpr (kSplitWhereBinned<K>)
          warp_children(T, s.split, chunk, next, c, level, tr, status);
        else if (lane == 0)
          splits[I.task] = s.split;
      }
    } else {
      // the codes in one store a thread (2 K bytes, by item), the bins to the task's
      constexpr int kWords = K / 2;
      const uint32_t* cs = reinterpret_cast<const uint32_t*>(s.code) + tid * kWords;
      uint32_t* cg = reinterpret_cast<uint32_t*>(code) + ((size_t)it * kLevelThreads + tid) * kWords;
      if constexpr (K == 8)
        *reinterpret_cast<uint4*>(cg) = *reinterpret_cast<const uint4*>(cs);
      else if constexpr (K == 4)
        *reinterpret_cast<uint2*>(cg) = *reinterpret_cast<const uint2*>(cs);
      else
        *cg = *cs;
      if (tid < 3 * kTopBins) {
        const uint32_t* b = sb + tid * kTopVals;
        uint32_t* g = bins + (size_t)I.task * kTopBinRow + tid * kTopVals;
        if (b[0]) {
          const uint32_t v[6] = {b[1], b[2], b[3], b[4], b[5], b[6]};
          bin_update(g, b[0], v);
        }
        uint32_t cum = 0;
        for (uint32_t k = tid & ~15u; k <= tid; ++k) cum += sb[k * kTopVals];
        icum[(size_t)tid * cap_items + it] = cum;
      }
      if constexpr (kSplitWhereBinned<K>) {  // the last of the task's items splits it
        __syncthreads();
        uint32_t* const row = bins + (size_t)I.task * kTopBinRow;
        if (tid == 0) {
          __threadfence();
          const bool last = atomicAdd(row + kTopBinWords, 1u) == (T.end - T.begin + chunk - 1) / chunk - 1u;
          __threadfence();
          s.last = last ? 1u : 0u;
        }
        __syncthreads();
        if (s.last) {
          for (uint32_t k = tid; k < kTopBinWords; k += kLevelThreads) sb[k] = __ldcg(row + k);
          __syncthreads();
          if (warp == 0) {
            warp_top_split(sb, T, &s.split, tr);
            __syncwarp();
            if (lane == 0) splits[I.task] = s.split;
            warp_children(T, s.split, chunk, next, c, level, tr, status);
          }
        }
      }
    }
    __syncthreads();  // the block's memory is free for the next item
  }
}

// ... where not: a warp per task, the splits of the tasks of several items and
// everyone's children
__global__ void __launch_bounds__(128) k_top_split(const TopTask* __restrict__ tasks, uint32_t chunk,
                                                   const uint32_t* __restrict__ bins, TopSplit* __restrict__ splits,
                                                   BuildCtl* __restrict__ c, uint32_t level_k, const NextLevel next,
                                                   const Tree tr, uint32_t* status) {
  __shared__ uint32_t s_bins[4][kTopBinWords];
  __shared__ TopSplit s_split[4];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, level = c->top_base + level_k;
  if (level >= kMaxTopLevels) return;
  const uint32_t n_tasks = min(c->top[level].tasks, next.cap_tasks);
  for (uint32_t t = blockIdx.x * 4u + warp; t < n_tasks; t += gridDim.x * 4u) {  // whole warps
    const TopTask T = tasks[t];
    if (T.end - T.begin > chunk) {
      for (uint32_t k = lane; k < kTopBinWords; k += 32u) s_bins[warp][k] = bins[(size_t)t * kTopBinRow + k];
      __syncwarp();
      warp_top_split(s_bins[warp], T, &s_split[warp], tr);
      __syncwarp();
      if (lane == 0) splits[t] = s_split[warp];
    } else if (lane == 0) {
      s_split[warp] = splits[t];
    }
    __syncwarp();
    warp_children(T, s_split[warp], chunk, next, c, level, tr, status);
    __syncwarp();
  }
}

// the stable partition of the tasks of several items: an item's lefts go
// after those of the task's earlier items (a row of icum)
template <int K>
__global__ void __launch_bounds__(kLevelThreads) k_top_scatter(
    const uint32_t* __restrict__ ord, uint32_t* __restrict__ ord2, const TopItem* __restrict__ items,
    const TopTask* __restrict__ tasks, const BuildCtl* __restrict__ c, uint32_t level_k, uint32_t cap_items,
    const uint16_t* __restrict__ code, const uint32_t* __restrict__ icum, const TopSplit* __restrict__ splits,
    uint32_t* status) {
  constexpr uint32_t chunk = K * kLevelThreads;
  __shared__ uint32_t s_cnt[64], s_sum[kLevelThreads / 32];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t level = c->top_base + level_k;
  if (level >= kMaxTopLevels || c->error) return;
  const uint32_t n_items = min(c->top[level].items, cap_items);
  for (uint32_t it = blockIdx.x; it < n_items; it += gridDim.x) {  // uniform over the block
    const TopItem I = items[it];
    const TopTask T = tasks[I.task];
    if (T.end - T.begin <= chunk) continue;  // partitioned where it was binned
    // the positions' codes and order, whatever the split is: their fetch goes
    // on beside that of the split and of the sums that hang on it (28.09M
    // triangles, 18 levels: 2.30 -> 1.32 ms; a level of one task moves 281 MB
    // in 90 us)
    uint32_t cd[K], o[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const uint32_t k = (uint32_t)j * kLevelThreads + tid;
      o[j] = k < I.n ? ord[I.begin + k] : 0u;
      cd[j] = k < I.n ? code[(size_t)it * chunk + k] : 0u;
    }
    const TopSplit S = splits[I.task];
    uint32_t before = 0;  // lefts of the task's earlier items
    if (S.axis < 3) {
      const uint32_t* row = icum + (size_t)(S.axis * kTopBins + S.bin) * cap_items;
      for (uint32_t k = I.first + tid; k < it; k += kLevelThreads) before += row[k];
      before = __reduce_add_sync(0xffffffffu, before);
      if (lane == 0) s_sum[warp] = before;
    }
    __syncthreads();
    uint32_t left0;
    if (S.axis < 3) {
      left0 = 0;
#pragma unroll
      for (int w = 0; w < kLevelThreads / 32; ++w) left0 += s_sum[w];
    } else {
      left0 = min(S.nleft, I.begin - T.begin);
    }
    partition_item<K>(S, T.begin, I.begin - T.begin, I.n, T.end, left0, s_cnt, cd, o, ord2, status);
    __syncthreads();  // the counts are read before the next item resets them
  }
}

// -------------------------------------------------- 5d. small tasks ----
//
// One block takes a task of at most kSmallTask triangles through the rest of
// its subtree in shared memory: the SAH levels down to segments (the same
// bins, splits and stable partitions as the level loop's), PLOC in every
// segment, and the cost programme of every node it makes. Done level by
// level over the whole mesh, these levels were bound by launches on small
// meshes (82k triangles: 17 PLOC rounds, 6 SAH levels and 23 cost passes of
// 2-5 us kernels) and by passes over memory on large ones (28M triangles:
// about 12 of the build's 30 ms).
//
// The boxes stay in shared memory; the levels permute 16-bit indices to
// them. In a level every thread bins a run of consecutive positions with
// shared atomics: the lanes of a warp are then some positions apart, so that
// fewer of them meet in one bin than with neighbouring positions, which in
// Morton order mostly share their bins.
//
// Then the boxes are put in the final order and all segments are clustered
// together, as one list: the clusters of 20 segments and more fill the lanes
// that a segment on its own (44 triangles on average, a few after three
// rounds) would leave idle. Each cluster carries a node number that no node
// below it uses, at first its position: a merge makes the node of the higher
// cluster's number and keeps the lower one's, so a segment's nodes take its
// positions but the first, and what is left at the end tells the segment.
// The cost of a cluster sits beside it, so the programme reads no memory.
//
// Measured (GB300): this kernel 6.2 ms for 28.09M triangles where the levels,
// rounds and cost passes it replaces took 11.5; builds of 82k / 2M / 28M
// triangles with their first frame 1.88 -> 1.45, 5.10 -> 4.20 and 33.0 -> 28.4
// ms. It is bound by instruction issue and latency (40 % of issue slots), so
// a block of 192 threads with four blocks an SM (24 warps, 85 registers) is
// the best of 64-512 threads and tasks of 512-2048 triangles: 0.424 ms for 2M
// triangles in 700-triangle tasks, against 0.444 at 256 threads (64
// registers, spills), 0.472 at 128, and 0.68 for 2048-triangle tasks.

#ifndef J3DG_SMALL_THREADS
#define J3DG_SMALL_THREADS 192
#endif
#ifndef J3DG_SMALL_BLOCKS
#define J3DG_SMALL_BLOCKS 4
#endif
#ifndef J3DG_SMALL_BINS
#define J3DG_SMALL_BINS 8
#endif
static const int kSmallThreads = J3DG_SMALL_THREADS;
static const int kSmallWarps = kSmallThreads / 32;
static const int kSmallPer = (J3DG_SMALL_TASK + kSmallThreads - 1) / kSmallThreads;  // positions per thread
static const uint32_t kSmallBins = J3DG_SMALL_BINS;  // local tasks binned at once
static const uint32_t kSmallTasks = kSmallTask / (J3DG_SAH_TOP + 1u) + 1u;  // tasks of one local level
static_assert(kSmallPer <= 32 && kSmallPer * kSmallWarps <= 64, "flag bits and list counts per thread");
static_assert(kSmallTask <= 4096u && kSmallTasks < 255u && kSmallTasks <= kSmallThreads,
              "12-bit positions, 8-bit local tasks, one thread per task");
static_assert(J3DG_SAH_TOP <= 128u && kPlocRadius <= 8, "cluster sizes in a byte, neighbours within a warp's pass");

struct SmallTaskMem {   // while the levels run
  uint16_t ord[2][kSmallTask];
  uint16_t code[kSmallTask];
  uint8_t tk[2][kSmallTask];
  uint32_t bins[kSmallBins * kTopBinWords];
};
template <int W>
struct SmallClusterMem {  // while the segments are clustered
  float cost[W][kSmallTask];   // a cluster's covering: costs, and wide nodes (at most 63)
  uint8_t wide[W][kSmallTask];
  uint16_t spare[kSmallTask];  // the cluster's unused node number
  uint8_t cnt[kSmallTask];     // its triangles
  uint8_t nn[kSmallTask];      // its nearest neighbour's offset + kPlocRadius, or 255
};
template <int W>
struct SmallMem {
  union {
    float2 box[3][kSmallTask];     // lo, hi per axis
    uint16_t wide16[W][kSmallTask];  // after the clustering: wide nodes of the segments' roots and the nodes above
  };
  uint32_t ref[kSmallTask];      // triangle, then cluster reference
  uint16_t seg[kSmallTask];      // each position's segment: its first position
  uint16_t par[kSmallTask];      // at a segment's first position: its parent node << 1 | side, later its cluster
  union {
    SmallTaskMem t;
    SmallClusterMem<W> c;
  };
  union {
    struct {  // while the levels run
      TopTask task[2][kSmallTasks];
      TopSplit split[kSmallTasks];
      uint32_t pre[kSmallTasks];  // left flags before each task's first position
    };
    float edge[kSmallWarps][kPlocRadius][kPlocRadius];  // clustering: areas that reach into the next warp's clusters
  };
  uint32_t wsum[64];
  uint32_t n_task[2], n_seg, n_rec, job, bad;
};

template <int W>
static size_t small_smem() {
  return sizeof(SmallMem<W>);
}

// the SAH levels of the task in s.task[0][0] (n triangles from global
// position b0); leaves the order in s.t.ord[return value], the segments in
// s.seg and s.par and a record (begin | mid << 16, end | level << 16) per
// node in rec
template <int W>
__device__ int small_levels(SmallMem<W>& s, uint32_t b0, uint32_t n, uint2* __restrict__ rec,
                            const Tree& tr, uint32_t* status) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t K = (n + kSmallThreads - 1) / kSmallThreads, p0 = min(n, tid * K), p1 = min(n, p0 + K);
  int cur = 0;
  for (uint32_t level = 0;; ++level) {
    const uint32_t nlt = s.n_task[cur];
    if (nlt == 0) return cur;
    if ((s.task[cur][0].side >> 1) >= kMaxTopLevels) {  // every task of a local level has its level
      if (tid == 0) atomicOr(tr.error, 1u);
      __syncthreads();
      if (tid == 0) s.bad = 1u;
      __syncthreads();
      return cur;
    }
    if (tid == 0) s.n_task[cur ^ 1] = 0;
    for (uint32_t base = 0; base < nlt; base += kSmallBins) {
      const uint32_t m = min(kSmallBins, nlt - base);
      for (uint32_t k = tid; k < m * kTopBinWords; k += kSmallThreads) {
        const uint32_t v = k % kTopVals;
        s.t.bins[k] = v == 0 ? 0u : (v < 4 ? 0xffffffffu : 0u);
      }
      __syncthreads();
      {
        uint32_t last = kNoTask;
        TopBinner B;
        B.lx = B.ly = B.lz = B.sx = B.sy = B.sz = 0.f;
        const uint32_t q0 = min(n, (lane * kSmallWarps + warp) * K), q1 = min(n, q0 + K);  // lanes far apart
        for (uint32_t p = q0; p < q1; ++p) {
          const uint32_t t = (uint32_t)s.t.tk[cur][p] - base;  // 255: no task
          if (t >= m) continue;
          if (t != last) {
            B.set(s.task[cur][base + t]);
            last = t;
          }
          const uint32_t i = s.t.ord[cur][p];
          const float2 fx = s.box[0][i], fy = s.box[1][i], fz = s.box[2][i];
          const uint32_t v[6] = {f2o(fx.x), f2o(fy.x), f2o(fz.x), f2o(fx.y), f2o(fy.y), f2o(fz.y)};
          const uint32_t cd = B.code(0.5f * (fx.x + fx.y), 0.5f * (fy.x + fy.y), 0.5f * (fz.x + fz.y),
                                     s.task[cur][base + t]);
          s.t.code[p] = (uint16_t)cd;
          bin_update3(s.t.bins + t * kTopBinWords, cd, 1u, v);
        }
      }
      __syncthreads();
      for (uint32_t t = warp; t < m; t += kSmallWarps)
        warp_top_split(s.t.bins + t * kTopBinWords, s.task[cur][base + t], &s.split[base + t], tr);
      __syncthreads();
    }
    // the children's tasks
    if (tid < nlt) {
      const TopTask T = s.task[cur][tid];
      TopSplit& S = s.split[tid];
      const uint32_t mid = T.begin + S.nleft;  // the node's number too
      link_child(tr, T.parent, T.side, mid);
      // at most kSmallTask - 1 nodes: their records fit the task's own range
      const uint32_t r = atomicAdd(&s.n_rec, 1u);
      rec[b0 + r] = make_uint2((T.begin - b0) | ((mid - b0) << 16), (T.end - b0) | (level << 16));
#pragma unroll
      for (uint32_t side = 0; side < 2; ++side) {
        const uint32_t b = side ? mid : T.begin, e = side ? T.end : mid;
        S.task[side] = 255u;
        if (e - b > J3DG_SAH_TOP) {
          const uint32_t q = atomicAdd(&s.n_task[cur ^ 1], 1u);
          TopTask& C = s.task[cur ^ 1][q];
          C.begin = b;
          C.end = e;
          C.parent = mid;
          C.side = side | (((T.side >> 1) + 1u) << 1);
          C.clo = side ? S.rclo : S.lclo;
          C.chi = side ? S.rchi : S.lchi;
          S.task[side] = q;
        } else {
          s.par[b - b0] = (uint16_t)(((mid - b0) << 1) | side);
          atomicAdd(&s.n_seg, 1u);
        }
      }
    }
    // stable partition: lefts before each position by one scan
    uint32_t f = 0, cnt = 0;
    for (uint32_t p = p0; p < p1; ++p) {
      const uint32_t t = s.t.tk[cur][p];
      if (t >= nlt) continue;
      if (top_goes_left(b0 + p - s.task[cur][t].begin, s.t.code[p], s.split[t])) {
        f |= 1u << (p - p0);
        ++cnt;
      }
    }
    uint32_t inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= (uint32_t)o) inc += y;
    }
    if (lane == 31) s.wsum[warp] = inc;
    __syncthreads();
    uint32_t run = inc - cnt;
    for (uint32_t w = 0; w < warp; ++w) run += s.wsum[w];
    {
      uint32_t at = run;
      for (uint32_t p = p0; p < p1; ++p) {
        const uint32_t t = s.t.tk[cur][p];
        if (t < nlt && s.task[cur][t].begin - b0 == p) s.pre[t] = at;
        at += (f >> (p - p0)) & 1u;
      }
    }
    __syncthreads();
    for (uint32_t p = p0; p < p1; ++p) {
      const uint32_t t = s.t.tk[cur][p], left = (f >> (p - p0)) & 1u;
      uint32_t d = p, next = 255u;
      if (t < nlt) {
        const uint32_t begin = s.task[cur][t].begin - b0, l = run - s.pre[t], mid = begin + s.split[t].nleft;
        d = left ? begin + l : mid + (p - begin - l);
        next = s.split[t].task[left ? 0 : 1];
        run += left;
        if (d >= n) {
          atomicOr(status, J3DG_DEV_BAD_INDEX);
          continue;
        }
        if (next == 255u) s.seg[d] = (uint16_t)(left ? begin : mid);
      }
      s.t.ord[cur ^ 1][d] = s.t.ord[cur][p];
      s.t.tk[cur ^ 1][d] = (uint8_t)next;
    }
    __syncthreads();  // the level's tasks and splits are read before the next level writes them
    cur ^= 1;
  }
}

__device__ __forceinline__ float merged_area2(const float2 (&a)[3], const float2 (&b)[3]) {
  return merged_area(make_float4(a[0].x, a[1].x, a[2].x, 0.f), make_float4(a[0].y, a[1].y, a[2].y, 0.f),
                     make_float4(b[0].x, b[1].x, b[2].x, 0.f), make_float4(b[0].y, b[1].y, b[2].y, 0.f));
}
__device__ __forceinline__ float half_area2(const float2 (&a)[3]) {
  return half_area(make_float4(a[0].x, a[1].x, a[2].x, 0.f), make_float4(a[0].y, a[1].y, a[2].y, 0.f));
}

// PLOC over the block's m clusters (one list, neighbours within a segment
// only) until n_seg are left, one a segment, in segment order
template <int W>
__device__ uint32_t small_cluster(SmallMem<W>& s, uint32_t b0, uint32_t m, uint32_t n_seg, uint32_t leaf_size,
                                  const Tree& tr) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, below = (1u << lane) - 1u;
  while (m > n_seg) {
    const uint32_t passes = (m + kSmallThreads - 1) / kSmallThreads;
    // nearest neighbours: each warp's clusters are consecutive, 32 at a time.
    // A pair's area is made once, by its lower cluster (right[o]: with the
    // cluster o positions on), and handed to the higher one, which lies in
    // the same pass or, where the lane index wraps, in the next; the areas
    // that reach into the next warp's clusters go through shared memory.
    // Candidates are compared in increasing position: the first of equal
    // areas wins.
    const uint32_t lo = warp * passes * 32u;
    uint32_t first_bo = 255u;
    float first_best = INFINITY;
    {
      float before[kPlocRadius + 1];
#pragma unroll
      for (int o = 1; o <= kPlocRadius; ++o) before[o] = INFINITY;
      for (uint32_t i0 = lo; i0 < min(m, lo + passes * 32u); i0 += 32u) {
        const uint32_t i = i0 + lane;
        const bool act = i < m;
        // how many of the following clusters are of the cluster's segment
        // (up to the radius): by the segments' first clusters
        const uint32_t sg = act ? s.seg[i] : 0xffffu;
        const uint32_t sg2 = i + 32u < m ? s.seg[i + 32u] : 0xffffu;
        const uint32_t sn = __shfl_sync(0xffffffffu, lane == 0 ? sg2 : sg, (lane + 1u) & 31u);
        const uint32_t sn2 = __shfl_down_sync(0xffffffffu, sg2, 1);
        // bit l: the cluster after i0 + l starts another segment
        const uint64_t ends = (uint64_t)__ballot_sync(0xffffffffu, sn != sg) |
                              ((uint64_t)__ballot_sync(0xffffffffu, sn2 != sg2) << 32);
        const uint32_t run = act ? min((uint32_t)kPlocRadius, (uint32_t)__ffsll(ends >> lane | 1ull << 31) - 1u) : 0u;
        float2 a[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) a[k] = act ? s.box[k][i] : make_float2(0.f, 0.f);
        float right[kPlocRadius + 1], best = INFINITY;
        uint32_t bo = 255u;
#pragma unroll
        for (int o = kPlocRadius; o >= 1; --o) {
          right[o] = INFINITY;
          if ((uint32_t)o <= run) {
            float2 b[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) b[k] = s.box[k][i + o];
            right[o] = merged_area2(a, b);
          }
          const float left = __shfl_sync(0xffffffffu, lane + o < 32u ? right[o] : before[o], (lane - o) & 31u);
          if (left < best) {
            best = left;
            bo = kPlocRadius - o;
          }
          before[o] = right[o];
        }
#pragma unroll
        for (int o = 1; o <= kPlocRadius; ++o)
          if (right[o] < best) {
            best = right[o];
            bo = kPlocRadius + o;
          }
        if (i0 == lo) {
          first_best = best;
          first_bo = bo;
        } else if (act) {
          s.c.nn[i] = (uint8_t)bo;
        }
      }
      if (lane >= 32u - kPlocRadius)
#pragma unroll
        for (int o = 1; o <= kPlocRadius; ++o) s.edge[warp][lane - (32u - kPlocRadius)][o - 1] = before[o];
    }
    __syncthreads();
    if (lo + lane < m) {
      if (lane < (uint32_t)kPlocRadius && lo) {
        // the clusters of the warp before, which come first: they win ties
        float best = INFINITY;
        uint32_t bo = 255u;
#pragma unroll
        for (int o = kPlocRadius; o >= 1; --o)
          if ((uint32_t)o > lane) {
            const float left = s.edge[warp - 1][kPlocRadius + lane - o][o - 1];
            if (left < best) {
              best = left;
              bo = kPlocRadius - o;
            }
          }
        if (best <= first_best && bo != 255u) first_bo = bo;
      }
      s.c.nn[lo + lane] = (uint8_t)first_bo;
    }
    __syncthreads();
    // survivors before each pass's warp
    uint32_t flags = 0;  // 2 bits per pass: keep, create
    for (uint32_t pass = 0; pass < passes; ++pass) {
      if (pass * kSmallThreads + warp * 32u >= m) {  // past the list: the warp has nothing
        if (lane == 0) s.wsum[pass * kSmallWarps + warp] = 0;
        continue;
      }
      const uint32_t i = pass * kSmallThreads + tid;
      bool keep = false, create = false;
      if (i < m) {
        const uint32_t o = s.c.nn[i];
        const bool mutual = o != 255u && s.c.nn[i + o - kPlocRadius] == 2u * kPlocRadius - o;
        create = mutual && o > (uint32_t)kPlocRadius;
        keep = !mutual || create;
      }
      flags |= ((keep ? 1u : 0u) | (create ? 2u : 0u)) << (2u * pass);
      const uint32_t k = __popc(__ballot_sync(0xffffffffu, keep));
      if (lane == 0) s.wsum[pass * kSmallWarps + warp] = k;
    }
    __syncthreads();
    if (warp == 0) {
      const uint32_t c = passes * kSmallWarps;
      const uint32_t x = lane < c ? s.wsum[lane] : 0u, y = lane + 32u < c ? s.wsum[lane + 32u] : 0u;
      uint32_t xi = x, yi = y;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, xi, o), v = __shfl_up_sync(0xffffffffu, yi, o);
        if (lane >= (uint32_t)o) {
          xi += u;
          yi += v;
        }
      }
      const uint32_t half = __shfl_sync(0xffffffffu, xi, 31);
      if (lane < c) s.wsum[lane] = xi - x;
      if (lane + 32u < c) s.wsum[lane + 32u] = half + yi - y;
      if (lane == 31) s.job = half + yi;  // the survivors
    }
    __syncthreads();
    const uint32_t m2 = s.job;
    // merges and compaction, a block's width of clusters at a time: a
    // survivor moves to a position at or below its own, so what later passes
    // read is in place
    for (uint32_t pass = 0; pass < passes; ++pass) {
      const uint32_t i = pass * kSmallThreads + tid;
      if (pass * kSmallThreads + warp * 32u >= m) {
        __syncthreads();
        __syncthreads();
        continue;
      }
      const bool keep = (flags >> (2u * pass)) & 1u, create = (flags >> (2u * pass)) & 2u;
      const uint32_t bk = __ballot_sync(0xffffffffu, keep);
      const uint32_t pos = s.wsum[pass * kSmallWarps + warp] + __popc(bk & below);
      float2 a[3];
      uint32_t ref = 0, num = 0, sg = 0, spare = 0;
      Covering<W> C;
      auto covering = [&](uint32_t p, Covering<W>& c) {
#pragma unroll
        for (int k = 1; k <= W; ++k) {
          c.cost[k] = s.c.cost[k - 1][p];
          c.wide[k] = s.c.wide[k - 1][p];
        }
      };
      if (keep) {
#pragma unroll
        for (int k = 0; k < 3; ++k) a[k] = s.box[k][i];
        ref = s.ref[i];
        num = s.c.cnt[i];
        sg = s.seg[i];
        spare = s.c.spare[i];
        covering(i, C);
      }
      if (create) {
        const uint32_t j = i + s.c.nn[i] - kPlocRadius, node = b0 + s.c.spare[j];
        Covering<W> cr, cn;
        NodeMeta M;
        covering(j, cr);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float2 b = s.box[k][j];
          a[k] = make_float2(fminf(a[k].x, b.x), fmaxf(a[k].y, b.y));
        }
        num += s.c.cnt[j];
        collapse_step<W>(C, cr, half_area2(a), num, leaf_size, cn, M);
        tr.node[node].lo = make_float4(a[0].x, a[1].x, a[2].x, __uint_as_float(ref));
        tr.node[node].hi = make_float4(a[0].y, a[1].y, a[2].y, __uint_as_float(s.ref[j]));
        tr.meta[node] = M;
        ref = node;
        C = cn;
      }
      __syncthreads();
      if (keep && (create || pos != i)) {
#pragma unroll
        for (int k = 0; k < 3; ++k) s.box[k][pos] = a[k];
        s.ref[pos] = ref;
        s.c.cnt[pos] = (uint8_t)num;
        s.seg[pos] = (uint16_t)sg;
        s.c.spare[pos] = (uint16_t)spare;
#pragma unroll
        for (int k = 1; k <= W; ++k) {
          s.c.cost[k - 1][pos] = C.cost[k];
          s.c.wide[k - 1][pos] = (uint8_t)C.wide[k];
        }
      }
      __syncthreads();
    }
    if (m2 >= m) {  // no pair merges (areas past the largest float)
      if (tid == 0) atomicOr(tr.error, 2u);
      break;
    }
    m = m2;
  }
  return m;
}

// (The covering carries the wide nodes too: k_collapse_place then writes every
// wide node where it stays, without the two passes over the levels that
// counted and numbered them and the permutation: with the top nodes' coverings
// made below instead of in a pass per level, and the bounding box's last step
// by a block, builds of 82k and 2M triangles with their first frame went from
// 1230 to 992 and from 3729 to 3322 us.)

// A small task's subtree is complete: the covering of every top node whose
// two children are. The second of a node's two to arrive makes it and goes on
// upwards (the nodes above were made by earlier launches, the coverings by
// blocks of this one, on any SM).
template <int W>
__device__ void climb(const Tree& tr, const BinNode* __restrict__ tbox, uint32_t n, uint32_t leaf_size) {
  auto covering = [&](uint32_t r, Covering<W>& c) {
    if (r & 0x80000000u) {
      const BinNode b = tbox[r & 0x7fffffffu];
      c.triangle(half_area(b.lo, b.hi));
    } else {
#pragma unroll
      for (int i = 1; i <= W; ++i) {
        c.cost[i] = __ldcg(tr.cost + (size_t)r * W + i - 1);
        c.wide[i] = __ldcg(tr.wide + (size_t)r * W + i - 1);
      }
    }
  };
  while (n != kNoParent) {
    __threadfence();
    if (atomicAdd(tr.done + n, 1u) == 0u) return;
    __threadfence();
    const float4 lo = __ldcg(&tr.node[n].lo), hi = __ldcg(&tr.node[n].hi);
    Covering<W> l, r, c;
    NodeMeta M;
    covering(left_ref(lo), l);
    covering(right_ref(hi), r);
    collapse_step<W>(l, r, half_area(lo, hi), tr.meta[n].count, leaf_size, c, M);
#pragma unroll
    for (int i = 1; i <= W; ++i) {
      tr.cost[(size_t)n * W + i - 1] = c.cost[i];
      tr.wide[(size_t)n * W + i - 1] = c.wide[i];
    }
    tr.meta[n] = M;
    n = tr.up[n];
  }
}

// tasks that still wait for SAH levels at level `base + k`
__device__ __forceinline__ uint32_t top_tasks_left(const BuildCtl* c, uint32_t k) {
  const uint32_t level = c->top_base + k;
  return c->top[min(level, kMaxTopLevels)].tasks;
}

template <int W>
__global__ void __launch_bounds__(kSmallThreads, W == 8 ? J3DG_SMALL_BLOCKS - 1 : J3DG_SMALL_BLOCKS)
    k_small_tasks(const uint32_t* __restrict__ ord_a, const uint32_t* __restrict__ ord_b,
                  const BinNode* __restrict__ tbox, const TopTask* __restrict__ tasks, const TopRange* __restrict__ ranges,
                  BuildCtl* __restrict__ c, uint32_t level_k, uint32_t leaf_size, uint32_t nt,
                  uint32_t cap_small, uint2* __restrict__ rec, const Tree tr, uint32_t* status) {
  extern __shared__ __align__(16) uint8_t small_raw[];
  SmallMem<W>& s = *reinterpret_cast<SmallMem<W>*>(small_raw);
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (top_tasks_left(c, level_k)) return;  // more SAH levels come first
  const uint32_t n_tasks = min(c->n_small, cap_small), n_jobs = n_tasks + min(c->n_ranges, nt);
  for (;;) {
    if (tid == 0) s.job = atomicAdd(&c->next_job, 1u);
    __syncthreads();
    const uint32_t job = s.job;
    if (job >= n_jobs) return;
    TopTask T;
    if (job < n_tasks) {
      T = tasks[job];
    } else {
      const TopRange R = ranges[job - n_tasks];
      T.begin = R.begin;
      T.end = R.end;
      T.parent = R.parent;
      T.side = R.side;
      T.clo = T.chi = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const uint32_t b0 = T.begin, n = T.end - T.begin;
    if (T.end > nt || T.begin >= T.end || n > (job < n_tasks ? kSmallTask : J3DG_SAH_TOP)) {  // block-uniform
      if (tid == 0) {
        atomicOr(status, J3DG_DEV_BAD_INDEX);
        atomicOr(tr.error, 1u);
      }
      __syncthreads();
      continue;
    }
    const uint32_t* ord = (T.side >> 1) & 1u ? ord_b : ord_a;  // the levels alternate: where the last one put the task
    if (tid == 0) {
      s.task[0][0] = T;
      s.n_task[0] = 1;
      s.n_seg = s.n_rec = s.bad = 0;
    }
    for (uint32_t p = tid; p < n; p += kSmallThreads) {
      const uint32_t t = ord[b0 + p];
      const float4 lo = tbox[t].lo, hi = tbox[t].hi;
      s.ref[p] = t;
      s.box[0][p] = make_float2(lo.x, hi.x);
      s.box[1][p] = make_float2(lo.y, hi.y);
      s.box[2][p] = make_float2(lo.z, hi.z);
      s.t.ord[0][p] = (uint16_t)p;
      s.t.tk[0][p] = 0;
      s.seg[p] = 0;
    }
    __syncthreads();
    if (n > J3DG_SAH_TOP) {
      const int cur = small_levels<W>(s, b0, n, rec, tr, status);
      if (s.bad) {
        __syncthreads();
        continue;
      }
      // boxes and triangles into the final order, one array at a time
      uint32_t idx[kSmallPer];
#pragma unroll
      for (int k = 0; k < kSmallPer; ++k) {
        const uint32_t p = tid + k * kSmallThreads;
        idx[k] = p < n ? s.t.ord[cur][p] : 0u;
      }
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        float2 v[kSmallPer];
#pragma unroll
        for (int k = 0; k < kSmallPer; ++k) v[k] = s.box[a][idx[k]];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kSmallPer; ++k)
          if (tid + k * kSmallThreads < n) s.box[a][tid + k * kSmallThreads] = v[k];
      }
      uint32_t r[kSmallPer];
#pragma unroll
      for (int k = 0; k < kSmallPer; ++k) r[k] = s.ref[idx[k]];
      __syncthreads();
#pragma unroll
      for (int k = 0; k < kSmallPer; ++k)
        if (tid + k * kSmallThreads < n) s.ref[tid + k * kSmallThreads] = r[k];
    } else if (tid == 0) {
      s.par[0] = 0xffffu;  // one segment: its root is the task's
      s.n_seg = 1;
    }
    __syncthreads();
    for (uint32_t p = tid; p < n; p += kSmallThreads) {
      s.ref[p] |= 0x80000000u;
      s.c.cnt[p] = 1;
      s.c.spare[p] = (uint16_t)p;
      const float2 a[3] = {s.box[0][p], s.box[1][p], s.box[2][p]};
      const float v = half_area2(a) * J3DG_SAH_CTRI;
#pragma unroll
      for (int k = 0; k < W; ++k) {
        s.c.cost[k][p] = v;
        s.c.wide[k][p] = 0;
      }
    }
    __syncthreads();
    const uint32_t m = small_cluster<W>(s, b0, n, s.n_seg, leaf_size, tr);
    if (m != s.n_seg) {  // an error was raised: nothing is linked
      __syncthreads();
      continue;
    }
    // every cluster is a segment's root, its number left over the segment's
    // first position: the root goes under its parent, its costs are found there
    for (uint32_t c = tid; c < m; c += kSmallThreads) {
      const uint32_t first = s.c.spare[c], par = s.par[first];
      if (par == 0xffffu)
        link_child(tr, T.parent, T.side, s.ref[c]);
      else
        link_child(tr, b0 + (par >> 1), par & 1u, s.ref[c]);
      s.par[first] = (uint16_t)c;
#pragma unroll
      for (int k = 0; k < W; ++k) s.wide16[k][c] = s.c.wide[k][c];
    }
    __syncthreads();
    // the levels' nodes, deepest first: a subtree's costs are kept at its
    // first position's cluster
    if (warp == 0) {
      uint32_t at = s.n_rec;
      while (at > 0) {
        const bool have = lane < at;
        const uint2 x = have ? rec[b0 + at - 1u - lane] : make_uint2(0u, 0u);
        const uint32_t lv = __shfl_sync(0xffffffffu, x.y >> 16, 0);
        const uint32_t same = __ballot_sync(0xffffffffu, have && (x.y >> 16) == lv);
        const uint32_t take = same == 0xffffffffu ? 32u : (uint32_t)__ffs(~same) - 1u;  // one level's records
        if (lane < take) {
          const uint32_t mid = x.x >> 16, node = b0 + mid;
          const uint32_t cb = s.par[x.x & 0xffffu], cm = s.par[mid];
          Covering<W> l, r, c;
          NodeMeta M;
#pragma unroll
          for (int k = 1; k <= W; ++k) {
            l.cost[k] = s.c.cost[k - 1][cb];
            r.cost[k] = s.c.cost[k - 1][cm];
            l.wide[k] = s.wide16[k - 1][cb];
            r.wide[k] = s.wide16[k - 1][cm];
          }
          collapse_step<W>(l, r, half_area(tr.node[node].lo, tr.node[node].hi), (x.y & 0xffffu) - (x.x & 0xffffu), leaf_size,
                           c, M);
#pragma unroll
          for (int k = 1; k <= W; ++k) {
            s.c.cost[k - 1][cb] = c.cost[k];
            s.wide16[k - 1][cb] = (uint16_t)c.wide[k];
          }
          tr.meta[node] = M;
        }
        at -= take;
        __syncwarp();
      }
    }
    __syncthreads();
    // the task's root: its covering, for the top nodes above it
    if (tid < (uint32_t)W && n > 1u) {
      const uint32_t r = T.parent == kNoParent ? *tr.root
                         : T.side & 1u         ? right_ref(tr.node[T.parent].hi)
                                               : left_ref(tr.node[T.parent].lo);
      tr.cost[(size_t)r * W + tid] = s.c.cost[tid][s.par[0]];
      tr.wide[(size_t)r * W + tid] = s.wide16[tid][s.par[0]];
    }
    __syncthreads();
    if (tid == 0) climb<W>(tr, tbox, T.parent, leaf_size);
    __syncthreads();  // the block's memory is free for the next job
  }
}

// ------------------------------------------------------------- driver ----

#define J3DG_CK(x)                                             \
  do {                                                         \
    cudaError_t e_ = (x);                                      \
    if (e_ != cudaSuccess) {                                   \
      err = std::string(#x) + ": " + cudaGetErrorString(e_);   \
      rc = J3DG_ERR_CUDA;                                      \
      goto cleanup;                                            \
    }                                                          \
  } while (0)

// slot_of[id] = leaf position of triangle id (ids are a permutation of 0..nt)
__global__ void k_slot_of(const float4* __restrict__ tris, uint32_t nt, uint32_t* __restrict__ slot_of,
                          uint32_t* status) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nt) return;
  const uint32_t id = __float_as_uint(tris[3 * (size_t)i].w);
  if (id >= nt) {
    atomicOr(status, J3DG_DEV_BAD_INDEX);
    return;
  }
  slot_of[id] = i;
}

// ------------------------------------------------ device-driven build ----
//
// Kernels read their sizes from BuildCtl and stride over them with fixed grids,
// so the launches do not depend on the tree, and the host looks at it once, at
// the build's end (J3DG_BUILD_LBVH too); once before the placement as well where
// the nodes are made in an array of their number (kStagedNodes), and once more
// for every set of levels that a deep tree needs. The default builder's levels
// (SAH, placement) are launched a few more of than a balanced tree has; the
// tree that needs more gets them after the host has looked (j3dg_mesh_build),
// or from a conditional while node in a captured build (a batch rebuilds its
// meshes ahead of its frames; a body ends in a one-thread kernel that sets the
// loop's condition).
// A level past the last finds nothing and costs a launch (about 2 us), a round
// of a loop 13-26 us between its levels, and making the graph of a single
// build took longer than the radix sort that it ran beside. The LBVH's loops
// (the collapse and both depth-first sweeps) are while nodes always. Builds of
// 82k / 2M / 28.09M triangles with their first frame, as a graph of loops and
// launched: 992 -> 906, 3322 -> 3224, 26262 -> 24598 us (the large one also by
// its nodes' array, kStagedNodes, and the index array from the pool).

// the root task, by its size: split level by level, by one block, or a segment
__global__ void k_ctl_init(BuildCtl* __restrict__ c, TopTask* __restrict__ tasks, TopTask* __restrict__ small,
                           TopRange* __restrict__ ranges, uint32_t nt, uint32_t top, uint32_t chunk,
                           uint32_t small_max) {
  if (top) {
    const float* bb = c->bb;
    TopTask r0;
    r0.begin = 0;
    r0.end = nt;
    r0.parent = kNoParent;
    r0.side = 0;
    r0.clo = make_float4(bb[0], bb[1], bb[2], 0.f);  // the vertex bbox holds every centroid
    r0.chi = make_float4(bb[3], bb[4], bb[5], 0.f);
    if (nt > small_max) {
      tasks[0] = r0;
      c->top[0].tasks = 1;
      c->top[0].items = (nt + chunk - 1) / chunk;
    } else if (nt > J3DG_SAH_TOP) {
      small[0] = r0;
      c->n_small = 1;
    } else {
      ranges[0] = TopRange{0, nt, kNoParent, 0};
      c->n_ranges = 1;
    }
  }
  // LBVH: the collapse's root item
  c->n_wide = 1;
  c->n_in = 1;
  c->place_levels = 1;
  c->level_end[0] = 1;
}

// The SAH levels were launched up to `base + k`: if no task is left, the
// binary tree is complete and the placement starts at its root; else nothing
// happens here.
__global__ void k_tree_done(BuildCtl* __restrict__ c, uint32_t k, const NodeMeta* __restrict__ meta, uint32_t nt,
                            PlaceItem* __restrict__ qa) {
  c->n_wide = 0;
  c->top_left = top_tasks_left(c, k);
  if (c->error || c->top_left) return;
  const uint32_t root = c->root;
  if (root == 0u || root >= nt || meta[root].wide >= nt) {  // a malformed tree: nothing is placed
    c->error |= 2u;
    return;
  }
  c->n_wide = meta[root].wide;
  c->place[0] = 1;
  qa[0] = PlaceItem{root, 0u, 1u, 0u};
}

// a captured build: the loop after the levels that were launched one by one
// goes on from here while something is left
__global__ void k_top_more(BuildCtl* __restrict__ c, uint32_t done, cudaGraphConditionalHandle h) {
  c->top_base += done;
  const bool left = c->top[min(c->top_base, kMaxTopLevels)].tasks > 0 && !c->error;
  if (left && c->top_base >= kMaxTopLevels) c->error |= 1u;
  cudaGraphSetConditional(h, left && c->top_base < kMaxTopLevels ? 1u : 0u);
}
__global__ void k_place_more(BuildCtl* __restrict__ c, uint32_t done, cudaGraphConditionalHandle h) {
  c->place_base += done;
  const bool left = c->place[min(c->place_base, kMaxPlaceLevels)] > 0 && !c->error;
  if (left && c->place_base >= kMaxPlaceLevels) c->error |= 4u;
  cudaGraphSetConditional(h, left && c->place_base < kMaxPlaceLevels ? 1u : 0u);
}

// node range [lohi[0], lohi[1]) of wide level l (empty outside the tree)
__device__ __forceinline__ void level_range(BuildCtl* c, int32_t l) {
  const bool ok = l >= 0 && l < (int32_t)c->place_levels;
  c->lohi[0] = ok && l > 0 ? c->level_end[l - 1] : 0u;
  c->lohi[1] = ok ? c->level_end[l] : 0u;
}

__global__ void k_dfs_setup(BuildCtl* __restrict__ c, uint32_t* __restrict__ pos, uint32_t up) {
  if (!up) {  // subtree sizes, deepest level first
    c->dfs_level = (int32_t)c->place_levels - 1;
  } else {  // positions, root level first
    c->dfs_level = 0;
    pos[0] = 0;
  }
  level_range(c, c->dfs_level);
}

__global__ void k_dfs_step(BuildCtl* __restrict__ c, uint32_t up, cudaGraphConditionalHandle h, uint32_t set) {
  c->dfs_level += up ? 1 : -1;
  level_range(c, c->dfs_level);  // past the last level: an empty range
  if (set) cudaGraphSetConditional(h, (c->dfs_level >= 0 && c->dfs_level < (int32_t)c->place_levels) ? 1u : 0u);
}

// the LBVH's collapse starts at the root that k_lbvh left
__global__ void k_lbvh_root(BuildCtl* __restrict__ c, CollapseItem* __restrict__ qa) {
  qa[0] = CollapseItem{c->root, 0u, 1u};
}

// after an LBVH collapse level: k_collapse allocated its wide nodes itself
__global__ void k_lbvh_step(BuildCtl* __restrict__ c, uint32_t nt, cudaGraphConditionalHandle h, uint32_t set) {
  if (c->n_in) {  // the level ran
    if (c->n_wide > nt || c->n_out > nt || c->place_levels >= kMaxPlaceLevels) {
      c->error |= 4u;
      c->n_in = 0;
    } else {
      if (c->n_wide > c->level_end[c->place_levels - 1]) c->level_end[c->place_levels++] = c->n_wide;
      c->n_in = c->n_out;
    }
    c->n_out = 0;
  }
  if (set) cudaGraphSetConditional(h, c->n_in > 0 ? 1u : 0u);
}

// Appends a while node to the graph that `st` is capturing: its condition is
// initially 1, or what `before(handle)` enqueues on `st` sets;
// `body(side, handle)` enqueues the loop body on `side`, which captures it
// into the node's body graph.
template <class Before, class Body>
static cudaError_t capture_while(cudaStream_t st, cudaStream_t side, Before&& before, Body&& body) {
  cudaStreamCaptureStatus cs;
  unsigned long long id = 0;
  cudaGraph_t g = nullptr;
  const cudaGraphNode_t* deps = nullptr;
  size_t nd = 0;
  cudaError_t e = cudaStreamGetCaptureInfo(st, &cs, &id, &g, &deps, nullptr, &nd);
  if (e != cudaSuccess) return e;
  if (cs != cudaStreamCaptureStatusActive) return cudaErrorStreamCaptureUnsupported;
  cudaGraphConditionalHandle h;
  if ((e = cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault)) != cudaSuccess) return e;
  before(h);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if ((e = cudaStreamGetCaptureInfo(st, &cs, &id, &g, &deps, nullptr, &nd)) != cudaSuccess) return e;
  cudaGraphNodeParams p = {};
  p.type = cudaGraphNodeTypeConditional;
  p.conditional.handle = h;
  p.conditional.type = cudaGraphCondTypeWhile;
  p.conditional.size = 1;
  cudaGraphNode_t node;
  if ((e = cudaGraphAddNode(&node, g, deps, nullptr, nd, &p)) != cudaSuccess) return e;
  if ((e = cudaStreamBeginCaptureToGraph(side, p.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                         cudaStreamCaptureModeThreadLocal)) != cudaSuccess)
    return e;
  body(side, h);
  const cudaError_t eb = cudaGetLastError();
  cudaGraph_t captured = nullptr;
  e = cudaStreamEndCapture(side, &captured);
  if (eb != cudaSuccess) return eb;
  if (e != cudaSuccess) return e;
  return cudaStreamUpdateCaptureDependencies(st, &node, nullptr, 1, cudaStreamSetCaptureDependencies);
}
template <class Body>
static cudaError_t capture_while(cudaStream_t st, cudaStream_t side, Body&& body) {
  return capture_while(st, side, [](cudaGraphConditionalHandle) {}, body);
}

// Every buffer of one build, sized by the triangle count alone (upper bounds
// where the tree decides: the wide nodes, the queues).
struct BuildPlan {
  uint32_t nv = 0, nt = 0, W = 4, leaf = 2;
  bool top = false;   // the default builder (binned-SAH top levels, PLOC below them)
  bool lbvh = false;  // this build is an LBVH (J3DG_BUILD_LBVH)
  // the builders the scratch serves: PLOC (the default) and / or LBVH (a
  // batch's rebuild lane may serve both)
  bool need_ploc = true, need_lbvh = false;
  // what was allocated: the scratch's smaller arrays as one
  std::vector<void*> owned;
  // scratch
  float* part = nullptr;
  uint64_t *k0 = nullptr, *k1 = nullptr;
  uint32_t *v0 = nullptr, *v1 = nullptr, *sort = nullptr;  // sort: per pass a ticket, the totals, the rows
  uint32_t *ord_a = nullptr, *ord_b = nullptr, *top_up = nullptr, *top_done = nullptr, *bins_a = nullptr, *bins_b = nullptr,
           *icum = nullptr;
  BinNode* tbox = nullptr;
  uint16_t* codes = nullptr;
  TopItem *items_a = nullptr, *items_b = nullptr;
  TopTask *tasks_a = nullptr, *tasks_b = nullptr, *small = nullptr;
  TopSplit* splits = nullptr;
  TopRange* ranges = nullptr;
  uint2* child = nullptr;
  BinNode* box = nullptr;
  uint32_t* other = nullptr;  // LBVH: the sibling handshake of k_lbvh
  NodeMeta* meta = nullptr;
  float* dp_cost = nullptr;
  uint32_t* dp_wide = nullptr;
  float4* wide = nullptr;
  PlaceItem *pa = nullptr, *pb = nullptr;
  uint2* range = nullptr;  // LBVH: each binary node's leaf range
  CollapseItem *qa = nullptr, *qb = nullptr;
  uint32_t *dfs_size = nullptr, *dfs_pos = nullptr;
  BuildCtl* ctl = nullptr;
  // outputs (the mesh keeps them once `owned` does not)
  float4 *normals = nullptr, *soup = nullptr, *tris_out = nullptr, *nodes = nullptr;
  uint32_t* slot_of = nullptr;
  // tasks of one level are disjoint, each above small_task(); so are the small tasks, each above J3DG_SAH_TOP
  uint32_t small_task() const { return nt >= kSmallFewBelow ? kSmallTask : kSmallTaskFew; }
  uint32_t cap_tasks() const { return nt / small_task() + 1; }
  uint32_t cap_small() const { return nt / J3DG_SAH_TOP + 1; }
  // keys per thread of the sort: the tile is as large as registers and shared
  // memory carry well where there are tiles for every SM, else smaller
  uint32_t sort_items() const { return nt >= kSortLarge ? kSortItems : kSortFew; }
  uint32_t sort_tiles() const { return (nt + sort_items() * kSortThreads - 1) / (sort_items() * kSortThreads); }
  size_t sort_words() const { return kRadixPasses * (256 * ((size_t)sort_tiles() + 1) + 1); }
  // positions per item of the SAH levels: large ones keep the runs of the
  // binning long and the bins to merge few; below about two items an SM (304
  // on 152 SMs) smaller items fill the device instead
  uint32_t chunk() const { return nt >= 600000u ? 2048u : (nt >= 300000u ? 1024u : 512u); }
  uint32_t cap_items() const { return nt / chunk() + cap_tasks() + 1; }
  // levels launched without looking: SAH splits halve at best, a placement
  // level takes every subtree W ways at best; the trees of scans and of the
  // procedural surfaces need 1-3 levels more (82k / 2M / 28.09M triangles: SAH
  // 7, 12, 15 at best), even numbers for the loops behind them
  uint32_t top_levels() const {
    uint32_t l = 0;
    while ((uint64_t)small_task() << l < nt) ++l;
    return l ? (l + 4u) & ~1u : 0u;
  }
  uint32_t place_levels() const {
    uint32_t l = 1;
    for (uint64_t n = W * (uint64_t)kPlaceJob; n < nt; n *= W) ++l;
    return std::min((l + 4u) & ~1u, kMaxPlaceLevels);
  }
  // the placement's jobs have two triangles and more each; the coverings are done with by then
  PlaceItem* jobs() const { return reinterpret_cast<PlaceItem*>(dp_cost); }
  Tree tree() const { return Tree{box, meta, top_up, top_done, dp_cost, dp_wide, &ctl->root, &ctl->error}; }
};

static const int kBBoxBlocks = 1024;

// Up to this size the wide nodes are made in an array at their bound and then
// copied into one of the tree's size: a copy of up to about 20 us, the time
// that the host takes to look at the tree's size first. 28.09M triangles: 0.25
// ms of copy and 3.6 GB less.
static const size_t kStagedNodes = (size_t)256 << 20;

// outputs: the mesh's arrays too (else the mesh's own: a rebuild in place);
// node_bound: with them, a node array at the size bound (rebuildable meshes;
// other builds write the nodes into an array of the tree's size at the end)
static cudaError_t plan_alloc(BuildPlan& P, cudaStream_t st, bool outputs = true, bool node_bound = true) {
  const size_t nt = P.nt, F4 = J3DG_NODE_F4(P.W);
  cudaError_t e = cudaSuccess;
  auto own = [&](void** p, size_t bytes) {
    if (e == cudaSuccess) e = cudaMallocAsync(p, bytes, st);
    if (e == cudaSuccess) P.owned.push_back(*p);
  };
  // arrays of at most 16 MB share one allocation (an allocation and its
  // release take 1.6 us, and a small build has 35 arrays); a larger one has
  // its own, which the pool can place where a freed one was
  struct Part {
    void** p;
    size_t at;
  };
  std::vector<Part> parts;
  size_t shared = 0;
  auto A = [&](auto*& p, size_t bytes) {
    if (bytes > ((size_t)16 << 20)) return own((void**)&p, bytes);
    parts.push_back(Part{(void**)&p, shared});
    shared += (bytes + 255) & ~(size_t)255;
  };
  A(P.part, sizeof(float) * 6 * kBBoxBlocks);
  A(P.k0, sizeof(uint64_t) * nt);
  A(P.k1, sizeof(uint64_t) * nt);
  A(P.v0, sizeof(uint32_t) * nt);
  A(P.v1, sizeof(uint32_t) * nt);
  // (a lane's smaller meshes may have more tiles)
  A(P.sort, sizeof(uint32_t) *
                std::max(P.sort_words(), (size_t)kRadixPasses * (256 * (kSortLarge / (kSortFew * kSortThreads) + 3))));
  if (P.need_ploc) {
    A(P.ord_a, sizeof(uint32_t) * nt);
    A(P.ord_b, sizeof(uint32_t) * nt);
    A(P.tbox, sizeof(BinNode) * nt);
    // (a lane's smaller meshes may have more items, of smaller chunks)
    const uint32_t tasks = std::max(P.cap_tasks(), std::min(P.nt, kSmallFewBelow) / kSmallTaskFew + 1);
    const uint32_t items = std::max(P.cap_items(), std::min(P.nt, 600000u) / 512u + tasks + 1);
    A(P.codes, sizeof(uint16_t) * std::max((size_t)P.cap_items() * P.chunk(), (size_t)items * 512));
    A(P.top_up, sizeof(uint32_t) * nt);
    A(P.top_done, sizeof(uint32_t) * nt);
    A(P.bins_a, sizeof(uint32_t) * (size_t)tasks * kTopBinRow);
    A(P.bins_b, sizeof(uint32_t) * (size_t)tasks * kTopBinRow);
    A(P.icum, sizeof(uint32_t) * (size_t)items * 3 * kTopBins);
    A(P.items_a, sizeof(TopItem) * items);
    A(P.items_b, sizeof(TopItem) * items);
    A(P.tasks_a, sizeof(TopTask) * tasks);
    A(P.tasks_b, sizeof(TopTask) * tasks);
    A(P.small, sizeof(TopTask) * P.cap_small());
    A(P.splits, sizeof(TopSplit) * tasks);
    A(P.ranges, sizeof(TopRange) * nt);  // at most one range per triangle
  }
  A(P.box, sizeof(BinNode) * nt);
  if (P.need_ploc) {
    A(P.dp_cost, sizeof(float) * P.W * nt);
    A(P.dp_wide, sizeof(uint32_t) * P.W * nt);
    A(P.meta, sizeof(NodeMeta) * nt);
    A(P.pa, sizeof(PlaceItem) * nt);
    A(P.pb, sizeof(PlaceItem) * nt);
    A(P.soup, sizeof(float4) * 3 * nt);  // the LBVH gathers straight into the leaf order
  }
  if (P.need_lbvh) {
    A(P.child, sizeof(uint2) * nt);
    A(P.other, sizeof(uint32_t) * nt);
    A(P.dfs_size, sizeof(uint32_t) * nt);
    A(P.dfs_pos, sizeof(uint32_t) * nt);
    A(P.range, sizeof(uint2) * (nt - 1));
    A(P.qa, sizeof(CollapseItem) * nt);
    A(P.qb, sizeof(CollapseItem) * nt);
  }
  // the wide nodes at their bound. The default builder writes them straight
  // into the mesh's array where that is there before them (a rebuildable mesh)
  // or worth waiting for (run_tree_ploc)
  const size_t wide_bytes = sizeof(float4) * F4 * nt;
  if (P.need_lbvh || (outputs && !node_bound && wide_bytes <= kStagedNodes)) A(P.wide, wide_bytes);
  A(P.ctl, sizeof(BuildCtl));
  char* base = nullptr;
  own((void**)&base, shared);
  if (e == cudaSuccess)
    for (const Part& q : parts) *q.p = base + q.at;
  if (outputs) {  // else the mesh's own arrays (a rebuild in place)
    own((void**)&P.normals, sizeof(float4) * nt);
    own((void**)&P.tris_out, sizeof(float4) * 3 * nt);
    if (node_bound) own((void**)&P.nodes, sizeof(float4) * F4 * nt);  // the wide nodes are at most nt - 1
    own((void**)&P.slot_of, sizeof(uint32_t) * nt);
  }
  return e;
}

// an output that the caller takes over
template <class T>
static void* plan_take(BuildPlan& P, T*& p) {
  const auto it = std::find(P.owned.begin(), P.owned.end(), (void*)p);
  if (it != P.owned.end()) P.owned.erase(it);
  void* r = p;
  p = nullptr;
  return r;
}
// frees what is left
static void plan_free(BuildPlan& P, cudaStream_t st) {
  for (void* p : P.owned) cudaFreeAsync(p, st);
  P = BuildPlan{};
}

#define J3DG_EQ(x)                                \
  do {                                            \
    if (e == cudaSuccess) e = (x);                \
    if (e == cudaSuccess) e = cudaGetLastError(); \
  } while (0)

// a level's items, a block at a time: as many blocks as are resident or the
// level can have items
template <int K>
static void launch_top_bin_k(BuildPlan& P, cudaStream_t s, const uint32_t* oi, uint32_t* oo, const TopItem* items,
                             const TopTask* tasks, uint32_t* bins, const NextLevel& next, uint32_t k,
                             uint32_t* d_status) {
  const uint32_t blocks = std::min(wave_blocks128() / 16u * J3DG_LEVEL_BLOCKS, P.cap_items());
  cudaFuncSetAttribute(k_top_bin<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TopBinMem<K>));
  k_top_bin<K><<<blocks, kLevelThreads, sizeof(TopBinMem<K>), s>>>(oi, oo, P.tbox, items, tasks, P.ctl, k, bins,
                                                                   P.codes, P.icum, P.splits, next, P.tree(), d_status);
}
static void launch_top_bin(BuildPlan& P, cudaStream_t s, const uint32_t* oi, uint32_t* oo, const TopItem* items,
                           const TopTask* tasks, uint32_t* bins, const NextLevel& next, uint32_t k, uint32_t* d_status) {
  switch (P.chunk() / kLevelThreads) {
    case 8: return launch_top_bin_k<8>(P, s, oi, oo, items, tasks, bins, next, k, d_status);
    case 4: return launch_top_bin_k<4>(P, s, oi, oo, items, tasks, bins, next, k, d_status);
    default: return launch_top_bin_k<2>(P, s, oi, oo, items, tasks, bins, next, k, d_status);
  }
}

static void launch_top_scatter(BuildPlan& P, cudaStream_t s, const uint32_t* oi, uint32_t* oo, const TopItem* items,
                               const TopTask* tasks, uint32_t k, uint32_t* d_status) {
  const uint32_t blocks = std::min(wave_blocks128() / 2u, P.cap_items()), cap = P.cap_items();
  auto go = [&](auto kernel) {
    kernel<<<blocks, kLevelThreads, 0, s>>>(oi, oo, items, tasks, P.ctl, k, cap, P.codes, P.icum, P.splits, d_status);
  };
  switch (P.chunk() / kLevelThreads) {
    case 8: return go(k_top_scatter<8>);
    case 4: return go(k_top_scatter<4>);
    default: return go(k_top_scatter<2>);
  }
}

// SAH level `base + k`
static void launch_top_level(BuildPlan& P, cudaStream_t s, uint32_t k, uint32_t* d_status) {
  const bool odd = k & 1u;
  const uint32_t *oi = odd ? P.ord_b : P.ord_a;
  uint32_t* oo = odd ? P.ord_a : P.ord_b;
  const TopTask* tasks = odd ? P.tasks_b : P.tasks_a;
  const TopItem* items = odd ? P.items_b : P.items_a;
  const NextLevel next{odd ? P.tasks_a : P.tasks_b, odd ? P.items_a : P.items_b, odd ? P.bins_a : P.bins_b, P.small,
                       P.ranges, P.cap_tasks(), P.cap_small(), P.cap_items(), P.nt, P.small_task()};
  uint32_t* bins = odd ? P.bins_b : P.bins_a;
  launch_top_bin(P, s, oi, oo, items, tasks, bins, next, k, d_status);
  if (P.chunk() == 8 * kLevelThreads)  // !kSplitWhereBinned
    k_top_split<<<std::min(kStrideBlocks, P.cap_tasks() / 4u + 1u), 128, 0, s>>>(tasks, P.chunk(), bins, P.splits, P.ctl, k,
                                                                                 next, P.tree(), d_status);
  launch_top_scatter(P, s, oi, oo, items, tasks, k, d_status);
}

// section 5d over every small task and range: persistent blocks, as many as
// the device holds at the kernel's shared memory
template <int W>
static cudaError_t launch_small_tasks_w(BuildPlan& P, cudaStream_t st, uint32_t k, uint32_t* d_status) {
  const size_t smem = small_smem<W>();
  cudaError_t e = cudaFuncSetAttribute(k_small_tasks<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int dev = 0, sms = 0, per = 0;
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_small_tasks<W>, kSmallThreads, smem);
  if (e != cudaSuccess) return e;
  const uint32_t grid = std::min((uint32_t)std::max(1, sms * per), P.cap_small());
  k_small_tasks<W><<<grid, kSmallThreads, smem, st>>>(
      P.ord_a, P.ord_b, P.tbox, P.small, P.ranges, P.ctl, k, P.leaf, P.nt, P.cap_small(),
      reinterpret_cast<uint2*>(P.pb), P.tree(), d_status);
  return cudaGetLastError();
}

static cudaError_t launch_small_tasks(uint32_t W, BuildPlan& P, cudaStream_t st, uint32_t k, uint32_t* d_status) {
  if (W == 2) return launch_small_tasks_w<2>(P, st, k, d_status);
  if (W == 8) return launch_small_tasks_w<8>(P, st, k, d_status);
  return launch_small_tasks_w<4>(P, st, k, d_status);
}

// The default builder's binary tree and its wide nodes (in depth-first order):
// binned-SAH levels down to small tasks, each small task's subtree by one
// block (and the cost programme up to the root), the placement; the
// leaf-ordered triangles go to P.tris_out, their positions to P.slot_of.
static void enqueue_top_levels(BuildPlan& P, cudaStream_t st, uint32_t k0, uint32_t k1, uint32_t* d_status) {
  for (uint32_t k = k0; k < k1; ++k) launch_top_level(P, st, k, d_status);
}
template <int W>
static void enqueue_place_levels_w(BuildPlan& P, cudaStream_t st, uint32_t k0, uint32_t k1, uint32_t* d_status) {
  for (uint32_t k = k0; k < k1; ++k)
    k_collapse_place<W><<<wave_blocks128(), kPlaceThreads, 0, st>>>(
        P.box, P.meta, P.tbox, P.soup, k & 1u ? P.pb : P.pa, k & 1u ? P.pa : P.pb, P.jobs(), P.ctl, k,
        P.nodes ? P.nodes : P.wide, P.tris_out, P.slot_of, P.nt, d_status);
}
static void enqueue_place_levels(BuildPlan& P, cudaStream_t st, uint32_t k0, uint32_t k1, uint32_t* d_status) {
  if (P.W == 2)
    enqueue_place_levels_w<2>(P, st, k0, k1, d_status);
  else if (P.W == 8)
    enqueue_place_levels_w<8>(P, st, k0, k1, d_status);
  else
    enqueue_place_levels_w<4>(P, st, k0, k1, d_status);
}
static void enqueue_place_jobs(BuildPlan& P, cudaStream_t st, uint32_t k, uint32_t* d_status) {
  auto go = [&](auto kernel) {
    // more blocks than are resident: the jobs' sizes differ (28.09M triangles: 1.62 ms, in one wave 1.89)
    kernel<<<std::min(8u * wave_blocks128(), P.nt / 64u + 1u), kPlaceThreads, 0, st>>>(
        P.box, P.meta, P.tbox, P.soup, P.jobs(), P.ctl, k, P.nodes ? P.nodes : P.wide, P.tris_out, P.slot_of, P.nt, d_status);
  };
  if (P.W == 2)
    go(k_place_jobs<2>);
  else if (P.W == 8)
    go(k_place_jobs<8>);
  else
    go(k_place_jobs<4>);
}
static void enqueue_top_start(BuildPlan& P, cudaStream_t st) {
  k_top_boxes<<<(P.nt + 255) / 256, 256, 0, st>>>(P.soup, P.nt, P.tbox, P.ord_a);
  if (P.top_levels())
    k_top_items<<<std::min(kStrideBlocks, P.cap_items() / 256 + 1), 256, 0, st>>>(P.items_a, P.bins_a, P.nt, P.chunk());
}

// ... captured: loops after the levels
static cudaError_t capture_tree_ploc(BuildPlan& P, cudaStream_t st, cudaStream_t side, uint32_t* d_status) {
  BuildCtl* c = P.ctl;
  cudaError_t e = cudaSuccess;
  enqueue_top_start(P, st);
  const uint32_t levels = P.top_levels(), places = P.place_levels();
  if (levels) {
    enqueue_top_levels(P, st, 0, levels, d_status);
    J3DG_EQ(capture_while(
        st, side, [&](cudaGraphConditionalHandle h) { k_top_more<<<1, 1, 0, st>>>(c, levels, h); },
        [&](cudaStream_t s, cudaGraphConditionalHandle h) {
          enqueue_top_levels(P, s, 0, 2, d_status);
          k_top_more<<<1, 1, 0, s>>>(c, 2u, h);
        }));
  }
  J3DG_EQ(launch_small_tasks(P.W, P, st, 0, d_status));
  k_tree_done<<<1, 1, 0, st>>>(c, 0, P.meta, P.nt, P.pa);
  enqueue_place_levels(P, st, 0, places, d_status);
  J3DG_EQ(capture_while(
      st, side, [&](cudaGraphConditionalHandle h) { k_place_more<<<1, 1, 0, st>>>(c, places, h); },
      [&](cudaStream_t s, cudaGraphConditionalHandle h) {
        enqueue_place_levels(P, s, 0, 2, d_status);
        k_place_more<<<1, 1, 0, s>>>(c, 2u, h);
      }));
  enqueue_place_jobs(P, st, 0, d_status);
  J3DG_EQ(cudaSuccess);
  return e;
}

// ... on a stream, to its end: h is what the build left
static cudaError_t run_tree_ploc(BuildPlan& P, cudaStream_t st, uint32_t* d_status, BuildCtl& h) {
  cudaError_t e = cudaSuccess;
  enqueue_top_start(P, st);
  uint32_t levels = 0, places = 0, more_levels = P.top_levels(), more_places = P.place_levels();
  bool tree = false;
  for (;;) {
    if (!tree) {
      enqueue_top_levels(P, st, levels, levels + more_levels, d_status);
      levels += more_levels;
      J3DG_EQ(launch_small_tasks(P.W, P, st, levels, d_status));
      k_tree_done<<<1, 1, 0, st>>>(P.ctl, levels, P.meta, P.nt, P.pa);
      if (!P.nodes && !P.wide) {  // the nodes' array first
        J3DG_EQ(cudaMemcpyAsync(&h, P.ctl, kCtlHead, cudaMemcpyDeviceToHost, st));
        J3DG_EQ(cudaStreamSynchronize(st));
        if (e != cudaSuccess || h.error) return e;
        if (h.top_left == 0) {
          J3DG_EQ(cudaMallocAsync((void**)&P.nodes, sizeof(float4) * J3DG_NODE_F4(P.W) * (size_t)h.n_wide, st));
          if (e != cudaSuccess) return e;
          P.owned.push_back(P.nodes);
        }
      }
    }
    enqueue_place_levels(P, st, places, places + more_places, d_status);
    enqueue_place_jobs(P, st, places + more_places, d_status);
    J3DG_EQ(cudaMemcpyAsync(&h, P.ctl, kCtlHead, cudaMemcpyDeviceToHost, st));
    J3DG_EQ(cudaStreamSynchronize(st));
    if (e != cudaSuccess || h.error) return e;
    tree = h.top_left == 0;
    if (tree) {
      places += more_places;
      if (places >= kMaxPlaceLevels || h.place[places] == 0) {
        if (h.place[std::min(places, kMaxPlaceLevels)]) h.error |= 4u;
        return e;
      }
      more_places = std::min(4u, kMaxPlaceLevels - places);
    } else {
      if (levels >= kMaxTopLevels) {
        h.error |= 1u;
        return e;
      }
      more_levels = std::min(8u, kMaxTopLevels - levels);
    }
  }
}

// the LBVH (J3DG_BUILD_LBVH): Apetrei's one-pass binary tree over the sorted
// Morton codes, then the 4-wide collapse level by level; the triangles are
// already in leaf order (P.tris_out)
static cudaError_t enqueue_tree_lbvh(BuildPlan& P, const uint64_t* keys, cudaStream_t st, cudaStream_t side,
                                     uint32_t* d_status) {
  const uint32_t nt = P.nt;
  BuildCtl* c = P.ctl;
  cudaError_t e = cudaSuccess;
  J3DG_EQ(cudaMemsetAsync(P.other, 0xff, sizeof(uint32_t) * (nt - 1), st));
  k_lbvh<<<(nt + 255) / 256, 256, 0, st>>>(keys, P.tris_out, nt, P.child, P.box, P.range, P.other, &c->root);
  k_lbvh_root<<<1, 1, 0, st>>>(c, P.qa);
  J3DG_EQ(cudaSuccess);
  J3DG_EQ(capture_while(st, side, [&](cudaStream_t s, cudaGraphConditionalHandle h) {
    k_collapse<<<wave_blocks128(), 128, 0, s>>>(P.child, P.box, P.range, P.tris_out, P.qa, &c->n_in, P.qb, &c->n_out,
                                             &c->n_wide, P.wide, nt, P.leaf, &c->max_depth, d_status);
    k_lbvh_step<<<1, 1, 0, s>>>(c, nt, h, 0u);
    k_collapse<<<wave_blocks128(), 128, 0, s>>>(P.child, P.box, P.range, P.tris_out, P.qb, &c->n_in, P.qa, &c->n_out,
                                             &c->n_wide, P.wide, nt, P.leaf, &c->max_depth, d_status);
    k_lbvh_step<<<1, 1, 0, s>>>(c, nt, h, 1u);
  }));
  return e;
}

// the sorted Morton codes after the radix passes (they alternate k0 / k1)
static const uint64_t* sorted_keys(const BuildPlan& P) { return (kRadixPasses & 1) ? P.k1 : P.k0; }

template <int ITEMS>
static cudaError_t enqueue_radix_pass(BuildPlan& P, const uint64_t* ka, const uint32_t* va, uint64_t* kb, uint32_t* vb,
                                      int pass, cudaStream_t st, uint32_t* d_status) {
  const cudaError_t e =
      cudaFuncSetAttribute(k_radix_pass<ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SortMem<ITEMS>));
  if (e != cudaSuccess) return e;
  const uint32_t tiles = P.sort_tiles();
  uint32_t *tickets = P.sort, *totals = tickets + kRadixPasses, *rows = totals + kRadixPasses * 256;
  k_radix_pass<ITEMS><<<tiles, kSortThreads, sizeof(SortMem<ITEMS>), st>>>(
      ka, va, kb, vb, P.nt, 8 * pass, totals + 256 * pass, rows + (size_t)pass * tiles * 256, tickets + pass, d_status);
  return cudaGetLastError();
}

// keys P.k0 (the passes alternate k0 / k1) to the order of the triangles
static cudaError_t enqueue_sort(BuildPlan& P, cudaStream_t st, uint32_t* d_status) {
  cudaError_t e = cudaSuccess;
  J3DG_EQ(cudaMemsetAsync(P.sort, 0, sizeof(uint32_t) * P.sort_words(), st));
  k_radix_totals<<<std::min(kStrideBlocks / 4u, (P.nt + 2047u) / 2048u), 512, 0, st>>>(P.k0, P.nt, P.sort + kRadixPasses);
  J3DG_EQ(cudaSuccess);
  uint64_t *ka = P.k0, *kb = P.k1;
  uint32_t *va = P.v0, *vb = P.v1;
  for (int pass = 0; pass < kRadixPasses; ++pass) {
    const uint32_t* in = pass ? va : nullptr;
    uint64_t* out = pass + 1 < kRadixPasses || P.lbvh ? kb : nullptr;  // the LBVH reads the sorted codes
    J3DG_EQ(P.sort_items() == kSortItems ? enqueue_radix_pass<kSortItems>(P, ka, in, out, vb, pass, st, d_status)
                                              : enqueue_radix_pass<kSortFew>(P, ka, in, out, vb, pass, st, d_status));
    std::swap(ka, kb);
    std::swap(va, vb);
  }
  return e;
}

// A build's first part, whose launches do not depend on the tree: the loop
// state reset, the bounding box, normals and Morton codes, the radix sort
// and the gather into Morton order. No host synchronisation.
static cudaError_t enqueue_prefix(BuildPlan& P, const float* dV, const uint32_t* dT, cudaStream_t st,
                                  uint32_t* d_status) {
  const uint32_t nt = P.nt, nv = P.nv;
  BuildCtl* c = P.ctl;
  cudaError_t e = cudaSuccess;
  J3DG_EQ(cudaMemsetAsync(c, 0, sizeof(BuildCtl), st));
  k_bbox_partial<<<kBBoxBlocks, 256, 0, st>>>(dV, nv, P.part);
  k_bbox_final<<<1, 1024, 0, st>>>(P.part, kBBoxBlocks, c->bb);
  k_ctl_init<<<1, 1, 0, st>>>(c, P.tasks_a, P.small, P.ranges, nt, P.top ? 1u : 0u, P.chunk(), P.small_task());
  k_tri_prep<<<(nt + 255) / 256, 256, 0, st>>>(dV, nv, dT, nt, c->bb, P.normals, P.k0, d_status);
  J3DG_EQ(cudaSuccess);
  J3DG_EQ(enqueue_sort(P, st, d_status));
  k_soup<<<(nt + 255) / 256, 256, 0, st>>>(dV, dT, kRadixPasses & 1 ? P.v1 : P.v0, nt, nv, P.lbvh ? P.tris_out : P.soup,
                                           d_status);
  J3DG_EQ(cudaSuccess);
  return e;
}

// The rest, captured: the tree, its wide nodes in depth-first order and the
// triangles' slots. The nodes go to P.nodes where it is given, else to P.wide
// (LBVH: the permutation into depth-first order is then left to the caller).
static cudaError_t enqueue_tree(BuildPlan& P, cudaStream_t st, cudaStream_t side, uint32_t* d_status) {
  const uint32_t nt = P.nt;
  BuildCtl* c = P.ctl;
  cudaError_t e = cudaSuccess;
  if (!P.lbvh) return capture_tree_ploc(P, st, side, d_status);
  J3DG_EQ(enqueue_tree_lbvh(P, sorted_keys(P), st, side, d_status));
  // depth-first numbering: subtree sizes bottom-up, positions top-down, permute
  k_dfs_setup<<<1, 1, 0, st>>>(c, P.dfs_pos, 0u);
  J3DG_EQ(capture_while(st, side, [&](cudaStream_t s, cudaGraphConditionalHandle h) {
    k_dfs_size<4><<<kStrideBlocks, 256, 0, s>>>(P.wide, c->lohi, P.dfs_size);
    k_dfs_step<<<1, 1, 0, s>>>(c, 0u, h, 0u);
    k_dfs_size<4><<<kStrideBlocks, 256, 0, s>>>(P.wide, c->lohi, P.dfs_size);
    k_dfs_step<<<1, 1, 0, s>>>(c, 0u, h, 1u);
  }));
  k_dfs_setup<<<1, 1, 0, st>>>(c, P.dfs_pos, 1u);
  J3DG_EQ(capture_while(st, side, [&](cudaStream_t s, cudaGraphConditionalHandle h) {
    k_dfs_place<4><<<kStrideBlocks, 256, 0, s>>>(P.wide, c->lohi, P.dfs_size, P.dfs_pos);
    k_dfs_step<<<1, 1, 0, s>>>(c, 1u, h, 0u);
    k_dfs_place<4><<<kStrideBlocks, 256, 0, s>>>(P.wide, c->lohi, P.dfs_size, P.dfs_pos);
    k_dfs_step<<<1, 1, 0, s>>>(c, 1u, h, 1u);
  }));
  if (P.nodes) k_dfs_permute<4><<<(nt + 255) / 256, 256, 0, st>>>(P.wide, &c->n_wide, P.dfs_pos, P.nodes);
  k_slot_of<<<(nt + 255) / 256, 256, 0, st>>>(P.tris_out, nt, P.slot_of, d_status);
  J3DG_EQ(cudaSuccess);
  return e;
}

// all of a build's work on `st` (capturing)
static cudaError_t enqueue_build(BuildPlan& P, const float* dV, const uint32_t* dT, cudaStream_t st,
                                 cudaStream_t side, uint32_t* d_status) {
  cudaError_t e = cudaSuccess;
  J3DG_EQ(enqueue_prefix(P, dV, dT, st, d_status));
  J3DG_EQ(enqueue_tree(P, st, side, d_status));
  return e;
}

// One mesh's build: the prefix, then the tree on the same stream (LBVH: the
// GPU sorts while the host captures and instantiates the tree's part), then
// the tree's size from the device and a copy of the nodes of that size, unless
// they were made where they stay.
static int build_bvh_tree(j3dg_mesh* m, const float* dV, const uint32_t* dT, cudaStream_t st, uint32_t* d_status,
                          cudaEvent_t done, std::string& err) {
  BuildPlan P;
  P.nv = m->nv;
  P.nt = m->nt;
  P.W = m->width;
  P.leaf = m->leaf_size;
  P.lbvh = (m->build_flags & J3DG_BUILD_LBVH) != 0;
  P.need_ploc = !P.lbvh;
  P.need_lbvh = P.lbvh;
  P.top = !P.lbvh;
  cudaStream_t side = nullptr;
  cudaGraph_t g = nullptr;
  cudaGraphExec_t ex = nullptr;
  BuildCtl h;
  int rc = J3DG_OK;
  cudaError_t e = plan_alloc(P, st, true, (m->build_flags & J3DG_BUILD_REBUILDABLE) != 0);
  J3DG_EQ(enqueue_prefix(P, dV, dT, st, d_status));
  if (!P.lbvh) {
    J3DG_EQ(run_tree_ploc(P, st, d_status, h));
  } else {
    J3DG_EQ(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
    if (e == cudaSuccess) e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      const cudaError_t eq = enqueue_tree(P, st, side, d_status);
      e = cudaStreamEndCapture(st, &g);
      if (eq != cudaSuccess) e = eq;
    }
    J3DG_EQ(cudaGraphInstantiate(&ex, g, 0));
    J3DG_EQ(cudaGraphLaunch(ex, st));
    J3DG_EQ(cudaMemcpyAsync(&h, P.ctl, kCtlHead, cudaMemcpyDeviceToHost, st));
    J3DG_EQ(cudaStreamSynchronize(st));
  }
  if (e != cudaSuccess) {
    err = std::string("build: ") + cudaGetErrorString(e);
    rc = e == cudaErrorMemoryAllocation ? J3DG_ERR_OUT_OF_MEMORY : J3DG_ERR_CUDA;
  } else if (h.error) {
    err = (h.error & 1u) ? "SAH top levels overran their bounds"
                         : ((h.error & 2u) ? "PLOC clustering ended with a malformed tree"
                                           : "BVH collapse overran its node bound");
    rc = J3DG_ERR_CUDA;
  }
  if (rc == J3DG_OK) {
    m->scale = 0.f;
    for (int k = 0; k < 3; ++k) {
      m->min_bb[k] = h.bb[k];
      m->max_bb[k] = h.bb[3 + k];
    }
    for (int k = 0; k < 6; ++k) m->scale = std::max(m->scale, std::fabs(h.bb[k]));
    m->n_nodes = h.n_wide;
    m->max_depth = h.max_depth;
    m->root_ref = 0;
    // the nodes into an array of the tree's size, unless they are where they
    // stay (a rebuildable mesh keeps an array at the size bound)
    if (P.nodes) {
      m->d_nodes = plan_take(P, P.nodes);
    } else {
      const size_t node = sizeof(float4) * J3DG_NODE_F4(P.W);
      e = cudaMallocAsync(&m->d_nodes, node * std::max(1u, m->n_nodes), st);
      if (e == cudaSuccess && m->n_nodes) {
        if (P.lbvh)
          k_dfs_permute<4><<<(m->n_nodes + 255) / 256, 256, 0, st>>>(P.wide, &P.ctl->n_wide, P.dfs_pos,
                                                                     (float4*)m->d_nodes);
        else
          e = cudaMemcpyAsync(m->d_nodes, P.wide, node * m->n_nodes, cudaMemcpyDeviceToDevice, st);
        J3DG_EQ(cudaSuccess);
      }
    }
    if (e == cudaSuccess && done) e = cudaEventRecord(done, st);  // the BVH is ready; the rest is clean-up
    if (e == cudaSuccess) {
      m->d_normals = plan_take(P, P.normals);
      m->d_tris = plan_take(P, P.tris_out);
      m->d_slot_of = plan_take(P, P.slot_of);
    } else {
      err = std::string("build: ") + cudaGetErrorString(e);
      rc = e == cudaErrorMemoryAllocation ? J3DG_ERR_OUT_OF_MEMORY : J3DG_ERR_CUDA;
    }
  }
  plan_free(P, st);
  if (ex) cudaGraphExecDestroy(ex);
  if (g) cudaGraphDestroy(g);
  if (side) cudaStreamDestroy(side);
  {
    const cudaError_t es = cudaStreamSynchronize(st);
    if (rc == J3DG_OK && es != cudaSuccess) {
      err = std::string("build: ") + cudaGetErrorString(es);
      rc = J3DG_ERR_CUDA;
    }
  }
  if (rc != J3DG_OK) return rc;
  const uint32_t W = m->width;
  if (m->max_depth > J3DG_MAX_DEPTH_W(W)) {
    err = "BVH depth " + std::to_string(m->max_depth) + " exceeds the traversal stack at width " + std::to_string(W);
    return J3DG_ERR_UNSUPPORTED;
  }
  m->device_bytes = sizeof(float4) * J3DG_NODE_F4(W) *
                        (uint64_t)((m->build_flags & J3DG_BUILD_REBUILDABLE) ? m->nt : (m->n_nodes ? m->n_nodes : 1)) +
                    sizeof(float4) * 4 * (uint64_t)m->nt + sizeof(uint32_t) * 4 * (uint64_t)m->nt;
  return J3DG_OK;
}

// ---------------------------------------------------- batch rebuilds ----
//
// A batch's graph rebuilds its meshes in place: each lane (a forked capture
// stream) owns one build's scratch, sized for its largest mesh, and builds
// its meshes one after another into their own arrays.

struct RebuildLane {
  BuildPlan P;  // scratch only; nt = the lane's largest mesh
};

int rebuild_lane_alloc(uint32_t nt_max, uint32_t nv_max, uint32_t W, bool ploc, bool lbvh, cudaStream_t st,
                       RebuildLane** out, std::string& err) {
  RebuildLane* L = new (std::nothrow) RebuildLane();
  if (!L) return J3DG_ERR_OUT_OF_MEMORY;
  L->P.nt = nt_max;
  L->P.nv = nv_max;
  L->P.W = W;
  L->P.need_ploc = ploc;
  L->P.need_lbvh = lbvh;
  L->P.top = ploc;
  const cudaError_t e = plan_alloc(L->P, st, false);
  if (e != cudaSuccess) {
    plan_free(L->P, st);
    delete L;
    err = std::string("batch rebuild scratch: ") + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? J3DG_ERR_OUT_OF_MEMORY : J3DG_ERR_CUDA;
  }
  *out = L;
  return J3DG_OK;
}

void rebuild_lane_free(RebuildLane* L, cudaStream_t st) {
  if (!L) return;
  plan_free(L->P, st);
  delete L;
}

// enqueues (under a capture) the rebuild of mesh m into its own arrays
cudaError_t rebuild_enqueue(RebuildLane* L, const j3dg_mesh* m, cudaStream_t st, cudaStream_t side, uint32_t* d_status) {
  if (m->nt <= m->leaf_size) return cudaSuccess;  // one leaf: nothing to rebuild
  BuildPlan Pm = L->P;  // the lane's scratch, this mesh's sizes and arrays
  Pm.nt = m->nt;
  Pm.nv = m->nv;
  Pm.leaf = m->leaf_size;
  Pm.lbvh = (m->build_flags & J3DG_BUILD_LBVH) != 0;
  Pm.top = !Pm.lbvh;
  if (Pm.lbvh ? !Pm.need_lbvh : !Pm.need_ploc) return cudaErrorInvalidValue;  // the lane has no scratch for it
  Pm.normals = (float4*)m->d_normals;
  Pm.tris_out = (float4*)m->d_tris;
  Pm.nodes = (float4*)m->d_nodes;
  Pm.slot_of = (uint32_t*)m->d_slot_of;
  return enqueue_build(Pm, (const float*)m->d_verts, (const uint32_t*)m->d_index, st, side, d_status);
}

// Builds the device BVH. dV and dT are device arrays. On success fills the
// mesh fields (bbox, scale, nodes, leaf-ordered triangles, normals); `done`
// (may be null) is recorded on st once the BVH is ready, before the host's
// clean-up (the build time is taken up to it). Both builders go through
// build_bvh_tree; a mesh of at most one leaf is built here.
int build_bvh(j3dg_mesh* m, const float* dV, const uint32_t* dT, cudaStream_t st, uint32_t* d_status,
              cudaEvent_t done, std::string& err) {
  if (m->nt > m->leaf_size) return build_bvh_tree(m, dV, dT, st, d_status, done, err);
  int rc = J3DG_OK;
  const uint32_t nv = m->nv, nt = m->nt;
  float* d_part = nullptr;
  float* d_bb = nullptr;
  uint64_t* k0 = nullptr;
  const int bbox_blocks = 1024;
  float hbb[6];
  const uint32_t W = m->width;
  const size_t F4 = J3DG_NODE_F4(W);

  J3DG_CK(cudaMallocAsync((void**)&d_part, sizeof(float) * 6 * bbox_blocks, st));
  J3DG_CK(cudaMallocAsync((void**)&d_bb, sizeof(float) * 6, st));
  k_bbox_partial<<<bbox_blocks, 256, 0, st>>>(dV, nv, d_part);
  k_bbox_final<<<1, 1024, 0, st>>>(d_part, bbox_blocks, d_bb);
  J3DG_CK(cudaGetLastError());
  J3DG_CK(cudaMemcpyAsync(hbb, d_bb, sizeof(hbb), cudaMemcpyDeviceToHost, st));
  J3DG_CK(cudaStreamSynchronize(st));
  m->scale = 0.f;
  for (int k = 0; k < 3; ++k) {
    m->min_bb[k] = hbb[k];
    m->max_bb[k] = hbb[3 + k];
  }
  for (int k = 0; k < 6; ++k) m->scale = std::max(m->scale, std::fabs(hbb[k]));

  // the triangles in input order (a single leaf), their normals; the root
  // is the leaf and the node array one empty node
  J3DG_CK(cudaMallocAsync(&m->d_normals, sizeof(float4) * (size_t)nt, st));
  J3DG_CK(cudaMallocAsync(&m->d_tris, sizeof(float4) * 3 * (size_t)nt, st));
  J3DG_CK(cudaMallocAsync((void**)&k0, sizeof(uint64_t) * nt, st));
  k_tri_prep<<<1, 256, 0, st>>>(dV, nv, dT, nt, d_bb, (float4*)m->d_normals, k0, d_status);
  k_soup<<<1, 256, 0, st>>>(dV, dT, nullptr, nt, nv, (float4*)m->d_tris, d_status);
  J3DG_CK(cudaGetLastError());
  m->root_ref = J3DG_LEAF_BIT | (nt - 1u);
  m->n_nodes = 0;
  m->max_depth = 0;
  J3DG_CK(cudaMallocAsync(&m->d_nodes, sizeof(float4) * F4, st));
  J3DG_CK(cudaMemsetAsync(m->d_nodes, 0, sizeof(float4) * F4, st));
  J3DG_CK(cudaMallocAsync(&m->d_slot_of, sizeof(uint32_t) * (size_t)nt, st));
  k_slot_of<<<1, 256, 0, st>>>((const float4*)m->d_tris, nt, (uint32_t*)m->d_slot_of, d_status);
  J3DG_CK(cudaGetLastError());
  if (done) J3DG_CK(cudaEventRecord(done, st));

cleanup:
  if (d_part) cudaFreeAsync(d_part, st);
  if (d_bb) cudaFreeAsync(d_bb, st);
  if (k0) cudaFreeAsync(k0, st);
  {
    cudaError_t e = cudaStreamSynchronize(st);
    if (rc == J3DG_OK && e != cudaSuccess) {
      err = std::string("build: ") + cudaGetErrorString(e);
      rc = J3DG_ERR_CUDA;
    }
  }
  if (rc != J3DG_OK) return rc;
  m->device_bytes = sizeof(float4) * F4 + sizeof(float4) * 4 * (uint64_t)nt + sizeof(uint32_t) * 4 * (uint64_t)nt;
  return J3DG_OK;
}

#undef J3DG_EQ
}  // namespace j3dg
