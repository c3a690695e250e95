// GPU PLOC build (Meister and Bittner, "Parallel Locally-Ordered
// Clustering for Bounding Volume Hierarchy Construction", TVCG 2018), in the
// exact form of the reference's PLOCAggregate::Build
// (core/aggregate/ploc_aggregate.cpp:252-327):
//   1. 30-bit Morton codes of the triangle-box centres in the scene box
//      (ploc_aggregate.cpp:37-82, 513-541);
//   2. a stable LSD radix sort over three 10-bit digits
//      (ploc_aggregate.cpp:84-132) -- optionally reproducing the reference's
//      stale digit-0 offset, so that the tree is the reference's own;
//   3. leaves in sorted order, then Cluster iterations until one node is left
//      (ploc_aggregate.cpp:400-511): nearest neighbour by joined-box area
//      within +-r (first minimum in index order), mutual pairs merge, an
//      inclusive scan places parents and children.
// The result is bit-identical to the reference's node array; it is then
// re-laid out for traversal (two child boxes per interior node, leaf slots
// holding the triangles in Morton order).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "scan.cuh"
#include "scene.cuh"

namespace ajg {
namespace {

constexpr int kBuckets = 1024;
constexpr int kRadixThreads = 256;
constexpr int kRadixWarps = kRadixThreads / 32;
// Keys a warp ranks in order, 32 at a time: 512 amortise the digit tables of
// a large sort; up to kSmallSort keys 64 spread the sort over eight times the
// blocks (10,214 keys: 16 -> 5 us a pass).
constexpr int kKeysPerWarp = 512, kKeysPerWarpSmall = 64;
constexpr uint64_t kSmallSort = 1ull << 18;
constexpr int kClusterThreads = 256;

struct PNode {  // reference Node: bound, primitive_count, first_child
  float4 a;     // lo.xyz, first (int bits)
  float4 b;     // hi.xyz, count (int bits)
};

__device__ __forceinline__ bool is_point(const F3& lo, const F3& hi) {
  return lo.x == hi.x && lo.y == hi.y && lo.z == hi.z;
}
// math/bounds.h:108-113
__device__ __forceinline__ void join(F3 alo, F3 ahi, F3 blo, F3 bhi, F3& lo,
                                     F3& hi) {
  if (is_point(alo, ahi)) {
    lo = blo;
    hi = bhi;
  } else if (is_point(blo, bhi)) {
    lo = alo;
    hi = ahi;
  } else {
    lo = vmin3(alo, blo);
    hi = vmax3(ahi, bhi);
  }
}
// math/bounds.h:98-101
__device__ __forceinline__ float area(F3 lo, F3 hi) {
  F3 d = hi - lo;
  return 2.f * (d.x * d.y + d.x * d.z + d.y * d.z);
}
// ploc_aggregate.cpp:168-182
__device__ __forceinline__ void tri_box(const float* t, F3& lo, F3& hi) {
  lo = mk3(FLT_MAX, FLT_MAX, FLT_MAX);
  hi = mk3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    F3 v = mk3(t[3 * k], t[3 * k + 1], t[3 * k + 2]);
    lo = vmin3(lo, v);
    hi = vmax3(hi, v);
  }
}

__device__ __forceinline__ uint32_t morton_split(uint32_t x) {
  x &= 0x3ffu;
  x = (x | (x << 16)) & 0x030000FFu;
  x = (x | (x << 8)) & 0x0300F00Fu;
  x = (x | (x << 4)) & 0x030C30C3u;
  x = (x | (x << 2)) & 0x09249249u;
  return x;
}
__device__ __forceinline__ uint32_t grid_coord(float f) {
  float g = ref_max(f, 0.f);
  if (g != g) return 0u;  // flat axis: NaN converts to 0
  uint32_t m = __float2uint_rz(g);
  return m < 1023u ? m : 1023u;
}

__global__ void k_morton(const float* __restrict__ tris, uint64_t n, F3 w2g,
                         F3 off, uint32_t* __restrict__ codes,
                         int32_t* __restrict__ vals) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    F3 lo, hi;
    tri_box(tris + 9 * i, lo, hi);
    F3 c = (hi + lo) / 2.f;
    F3 g = c * w2g + off;
    codes[i] = morton_split(grid_coord(g.x)) |
               (morton_split(grid_coord(g.y)) << 1) |
               (morton_split(grid_coord(g.z)) << 2);
    vals[i] = (int32_t)i;
  }
}

template <int KPW>
__global__ void k_radix_hist(const uint32_t* __restrict__ keys, uint64_t n,
                             int bit, uint32_t* __restrict__ hist,
                             uint32_t nb) {
  constexpr int kRadixTile = kRadixWarps * KPW;
  __shared__ uint32_t h[kBuckets];
  for (int d = threadIdx.x; d < kBuckets; d += blockDim.x) h[d] = 0;
  __syncthreads();
  const uint64_t t0 = (uint64_t)blockIdx.x * kRadixTile;
  for (int k = threadIdx.x; k < kRadixTile; k += blockDim.x) {
    uint64_t i = t0 + k;
    if (i < n) atomicAdd(&h[(keys[i] >> bit) & (kBuckets - 1)], 1u);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < kBuckets; d += blockDim.x)
    hist[(uint64_t)d * nb + blockIdx.x] = h[d];
}

// Stable scatter: warp w owns keys [t0 + w*KPW, t0 + (w+1)*KPW) and walks
// them in order, 32 at a time; lanes with equal digits rank by lane.
template <int KPW>
__global__ void __launch_bounds__(kRadixThreads)
    k_radix_scatter(const uint32_t* __restrict__ keys_in,
                    const int32_t* __restrict__ vals_in,
                    uint32_t* __restrict__ keys_out,
                    int32_t* __restrict__ vals_out, uint64_t n, int bit,
                    const uint32_t* __restrict__ offsets, uint32_t nb,
                    int compat, const uint32_t* __restrict__ compat_base,
                    int32_t* __restrict__ owner, uint32_t* __restrict__ pos_of,
                    uint32_t* __restrict__ err) {
  constexpr int kKeysPerWarp = KPW, kRadixTile = kRadixWarps * KPW;
  __shared__ uint32_t wh[kRadixWarps][kBuckets];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int k = threadIdx.x; k < kRadixWarps * kBuckets; k += blockDim.x)
    (&wh[0][0])[k] = 0;
  __syncthreads();
  const uint64_t wbase = (uint64_t)blockIdx.x * kRadixTile +
                         (uint64_t)w * kKeysPerWarp;
  for (int s = 0; s < kKeysPerWarp; s += 32) {
    uint64_t i = wbase + s + lane;
    if (i < n) atomicAdd(&wh[w][(keys_in[i] >> bit) & (kBuckets - 1)], 1u);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < kBuckets; d += blockDim.x) {
    uint32_t run = offsets[(uint64_t)d * nb + blockIdx.x];
#pragma unroll
    for (int q = 0; q < kRadixWarps; ++q) {
      uint32_t c = wh[q][d];
      wh[q][d] = run;
      run += c;
    }
  }
  __syncthreads();
  const uint32_t base0 = compat ? *compat_base : 0u;
  const unsigned lt = (1u << lane) - 1u;
  for (int s = 0; s < kKeysPerWarp; s += 32) {
    uint64_t i = wbase + s + lane;
    const bool valid = i < n;
    uint32_t key = valid ? keys_in[i] : 0u;
    uint32_t d = valid ? ((key >> bit) & (kBuckets - 1)) : 0xffffffffu;
    unsigned peers = __match_any_sync(0xffffffffu, d);
    uint32_t pos = 0;
    if (valid) pos = wh[w][d] + __popc(peers & lt);
    __syncwarp();
    if (valid && lane == __ffs(peers) - 1) wh[w][d] += __popc(peers);
    __syncwarp();
    if (!valid) continue;
    if (!compat) {
      keys_out[pos] = key;
      vals_out[pos] = vals_in[i];
    } else {
      uint64_t p = pos;
      if (d == 0) p += base0;
      if (p >= n) {
        raise_device_error(err, kDevSortOutOfBounds);
        pos_of[i] = 0xffffffffu;
      } else {
        atomicMax(&owner[p], (int32_t)i);
        pos_of[i] = (uint32_t)p;
      }
    }
  }
}

// Reference-compatible pass: the later key (in input order) wins a slot,
// unwritten slots keep the stale contents of the destination.
__global__ void k_radix_compat_write(const uint32_t* __restrict__ keys_in,
                                     const int32_t* __restrict__ vals_in,
                                     uint32_t* __restrict__ keys_out,
                                     int32_t* __restrict__ vals_out,
                                     uint64_t n,
                                     const int32_t* __restrict__ owner,
                                     const uint32_t* __restrict__ pos_of) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t p = pos_of[i];
    if (p != 0xffffffffu && owner[p] == (int32_t)i) {
      keys_out[p] = keys_in[i];
      vals_out[p] = vals_in[i];
    }
  }
}

// After pass p's offset scan: base = sum of digit-0 counts of passes < p.
__global__ void k_compat_base(const uint32_t* __restrict__ offsets,
                              uint32_t nb, uint32_t* acc) {
  const uint32_t count0 = offsets[(uint64_t)1 * nb + 0];
  acc[0] = acc[1];
  acc[1] += count0;
}

__global__ void k_leaf_init(const float* __restrict__ tris,
                            const int32_t* __restrict__ perm,
                            PNode* __restrict__ nodes, uint64_t n) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    F3 lo, hi;
    tri_box(tris + 9 * (uint64_t)perm[i], lo, hi);
    nodes[i].a = make_float4(lo.x, lo.y, lo.z, __int_as_float((int)i));
    nodes[i].b = make_float4(hi.x, hi.y, hi.z, __int_as_float(1));
  }
}

// SAH-optimal collapse into 4-wide nodes (the dynamic program of Ylitie,
// Karras, Laine, "Efficient incoherent ray traversal on GPUs through
// compressed wide BVHs", HPG 2017, with one triangle per leaf): cost[n].i
// (i = 1..4 slots) is the least sum of wide-node surface areas with which
// the subtree of binary node n fills at most i children of a wide node --
// one slot holding n itself (a leaf, or a wide node of its own: its area
// plus its children's best use of 4 slots), or its two children sharing
// the slots.  Leaves cost 0 in every slot count (a leaf's triangle test is
// the same whatever the tree).  choice[n] packs the decisions: byte 0 the
// left child's share of a wide node's 4 slots, byte i-1 (i = 2..4) for i
// slots 0 (n itself) or (left share << 4 | slots used).  A node's entry is
// computed when the clustering places it (its children were placed before).
#ifndef AJG_SAH_COLLAPSE
#define AJG_SAH_COLLAPSE 1
#endif
struct SahTable {
  float4* cost;      // [2n-1], null: not wanted
  uint32_t* choice;  // [2n-1]
};
__device__ __forceinline__ void sah_node(const SahTable& t, uint32_t at,
                                         const PNode& x) {
  if (!t.cost) return;
  if (__float_as_int(x.b.w) != 0) {  // leaf
    t.cost[at] = make_float4(0.f, 0.f, 0.f, 0.f);
    t.choice[at] = 0u;
    return;
  }
  const uint32_t f = (uint32_t)__float_as_int(x.a.w);
  const float4 L = t.cost[f], R = t.cost[f + 1];
  const float l[5] = {0.f, L.x, L.y, L.z, L.w};
  const float r[5] = {0.f, R.x, R.y, R.z, R.w};
  float dist[5];
  uint32_t dk[5];
#pragma unroll
  for (int j = 2; j <= 4; ++j) {
    dist[j] = __int_as_float(0x7f800000);
    dk[j] = 1;
#pragma unroll
    for (int k = 1; k < j; ++k) {
      const float v = l[k] + r[j - k];
      if (v < dist[j]) {
        dist[j] = v;
        dk[j] = (uint32_t)k;
      }
    }
  }
  float c[5];
  uint32_t kind[5] = {0u, 0u, 0u, 0u, 0u};
  c[1] = area(xyz(x.a), xyz(x.b)) + dist[4];
#pragma unroll
  for (int i = 2; i <= 4; ++i) {
    if (dist[i] < c[i - 1]) {
      c[i] = dist[i];
      kind[i] = (dk[i] << 4) | (uint32_t)i;
    } else {
      c[i] = c[i - 1];
      kind[i] = kind[i - 1];
    }
  }
  t.cost[at] = make_float4(c[1], c[2], c[3], c[4]);
  t.choice[at] = dk[4] | (kind[2] << 8) | (kind[3] << 16) | (kind[4] << 24);
}

// Cluster (ploc_aggregate.cpp:400-511), driven by device state: an iteration
// over `cnt` clusters finds neighbours (k_neighbors), pairs them
// (k_pairs: the merges per tile, and the last block to finish scans the
// tiles and writes the next iteration's state) and writes the next clusters
// and the pairs' nodes (k_cluster).  The active clusters are compact (two
// alternating arrays); a node goes to its place in the final array once,
// when it becomes a child: at `end` - 2 x merges, as the reference fills its
// array from the back.  The host enqueues a guess of iterations and reads
// the state once; kernels past the end of the work do nothing.  Once at most
// kTail clusters are left, one block runs all the iterations that remain
// (k_cluster_tail): they are short and most of the iterations.  kTail: one
// SM's neighbour search over 2,048 clusters of 32 candidates takes as long as
// the three launches it replaces (7 us), over 1,024 half of that.  Launch
// and synchronisation bound before: five launches, a copy and a wait per
// iteration (10,214 triangles, load to first picks: 3.00 -> 1.06 ms;
// 1,310,722 triangles, load to a 640x360 first image: 12.08 -> 7.27 ms).
struct PlocState {
  uint32_t cnt;    // clusters
  uint32_t end;    // final nodes at and above `end` are placed
  uint32_t iters;  // iterations done
  uint32_t buf;    // the cluster array in use
  uint32_t stuck;  // an iteration merged no pair
};
constexpr uint32_t kTail = 1024;
constexpr uint32_t kMaxIterations = 100000;
constexpr int kLevels = 64;  // levels of the wide collapse enqueued at most
constexpr int kTailThreads = 1024;
constexpr int kPairItems = 4;
constexpr uint32_t kPairTile = kClusterThreads * kPairItems;

__global__ void k_ploc_start(PlocState* s, uint32_t n, uint32_t* ticket) {
  s[0] = PlocState{n, 2 * n - 1, 0, 0, 0};
  *ticket = 0;
}
__device__ __forceinline__ bool ploc_idle(const PlocState& s) {
  return s.cnt <= kTail || s.stuck;
}

// A cluster's box in shared memory: lo.xy, (lo.z, hi.x), hi.yz.  Neighbouring
// lanes' boxes are 6 words apart, so a half warp's 8-byte loads hit different
// banks, and a candidate is three loads at constant offsets.  (A plane per
// coordinate is six loads with an address each: 100,000 clusters of 33
// candidates 12 -> 10.6 us, of 2,049 470 -> 405.)
struct Box6 {
  float2 a, b, c;
  __device__ __forceinline__ F3 lo() const { return mk3(a.x, a.y, b.x); }
  __device__ __forceinline__ F3 hi() const { return mk3(b.y, c.x, c.y); }
};
__device__ __forceinline__ Box6 box6(const PNode& n) {
  return Box6{make_float2(n.a.x, n.a.y), make_float2(n.a.z, n.b.x),
              make_float2(n.b.y, n.b.z)};
}

// Nearest neighbour of box k within [s0, s1) of `box`
// (ploc_aggregate.cpp:408-459): in ascending order with a strict comparison.
// 0xffffffff: none.
__device__ __forceinline__ uint32_t nearest(const Box6* box, uint32_t k,
                                            uint32_t s0, uint32_t s1) {
  const F3 ilo = box[k].lo(), ihi = box[k].hi();
  float best = FLT_MAX;
  uint32_t bj = 0xffffffffu;
  for (uint32_t j = s0; j < s1; ++j) {
    if (j == k) continue;
    const Box6 o = box[j];
    F3 lo, hi;
    join(ilo, ihi, o.lo(), o.hi(), lo, hi);
    const float d = area(lo, hi);
    if (d < best) {
      best = d;
      bj = j;
    }
  }
  return bj;
}

__global__ void __launch_bounds__(kClusterThreads)
    k_neighbors(const PlocState* __restrict__ st, const PNode* __restrict__ a,
                const PNode* __restrict__ b, int r, uint32_t* __restrict__ nb) {
  extern __shared__ Box6 sb[];
  const PlocState s = *st;
  if (ploc_idle(s)) return;
  const PNode* __restrict__ in = s.buf ? b : a;
  for (uint32_t i0 = blockIdx.x * kClusterThreads; i0 < s.cnt;
       i0 += gridDim.x * kClusterThreads) {
    const uint32_t lo_idx = i0 > (uint32_t)r ? i0 - r : 0u;
    const uint32_t hi_idx = min(i0 + kClusterThreads + (uint32_t)r, s.cnt);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < hi_idx - lo_idx; k += blockDim.x)
      sb[k] = box6(in[lo_idx + k]);
    __syncthreads();
    const uint32_t i = i0 + threadIdx.x;
    if (i >= s.cnt) continue;
    const uint32_t s0 = i > (uint32_t)r ? i - r : 0u;
    const uint32_t s1 = min(i + (uint32_t)r + 1, s.cnt);
    const uint32_t j = nearest(sb, i - lo_idx, s0 - lo_idx, s1 - lo_idx);
    nb[i] = j == 0xffffffffu ? j : j + lo_idx;
  }
}

// mate[i]: the cluster i merges with, or i itself; rank[i]: the merges of i's
// tile up to and with i (a merge counts at its first cluster).
__global__ void __launch_bounds__(kClusterThreads)
    k_pairs(PlocState* st, int cur, const uint32_t* __restrict__ nb,
            uint32_t* __restrict__ mate, uint16_t* __restrict__ rank,
            uint32_t* tile_sum, uint32_t* ticket) {
  __shared__ uint32_t s_count[kPairItems][kClusterThreads / 32];
  __shared__ uint32_t s_warp[kClusterThreads / 32];
  __shared__ uint32_t s_run;
  const PlocState s = st[cur];
  if (ploc_idle(s)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) st[cur ^ 1] = s;
    return;
  }
  const uint32_t tiles = (s.cnt + kPairTile - 1) / kPairTile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned le = 0xffffffffu >> (31 - lane);
  for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    uint32_t in_warp[kPairItems];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPairItems; ++k) {
      const uint32_t i = t * kPairTile + k * kClusterThreads + threadIdx.x;
      bool merges = false;
      if (i < s.cnt) {
        const uint32_t j = nb[i];
        const bool mutual = j != 0xffffffffu && nb[j] == i;
        mate[i] = mutual ? j : i;
        merges = mutual && i < j;
      }
      const unsigned bal = __ballot_sync(0xffffffffu, merges);
      in_warp[k] = __popc(bal & le);
      if (lane == 0) s_count[k][warp] = __popc(bal);
    }
    __syncthreads();
    uint32_t run = 0;
#pragma unroll
    for (int k = 0; k < kPairItems; ++k) {
      const uint32_t i = t * kPairTile + k * kClusterThreads + threadIdx.x;
      uint32_t before = run;
      for (int w = 0; w < kClusterThreads / 32; ++w) {
        if (w < warp) before += s_count[k][w];
        run += s_count[k][w];
      }
      if (i < s.cnt) rank[i] = (uint16_t)(before + in_warp[k]);
    }
    if (threadIdx.x == 0) tile_sum[t] = run;
  }
  // the last block scans the tiles' merges in place (exclusive)
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_run = atomicAdd(ticket, 1u);
  __syncthreads();
  if (s_run != gridDim.x - 1) return;
  __threadfence();
  uint32_t run = 0;
  for (uint32_t t0 = 0; t0 < tiles; t0 += kClusterThreads) {
    const uint32_t t = t0 + threadIdx.x;
    const uint32_t own = t < tiles ? __ldcg(&tile_sum[t]) : 0u;
    uint32_t x = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    uint32_t before = run, all = 0;
    for (int w = 0; w < kClusterThreads / 32; ++w) {
      if (w < warp) before += s_warp[w];
      all += s_warp[w];
    }
    if (t < tiles) tile_sum[t] = before + x - own;
    run += all;
  }
  if (threadIdx.x == 0) {
    PlocState next = s;
    next.stuck = run == 0;
    next.iters = s.iters + 1;
    next.cnt = s.cnt - run;
    next.end = s.end - 2 * run;
    next.buf = s.buf ^ 1;
    st[cur ^ 1] = next;
    *ticket = 0;
  }
}

// The parent of clusters i < j whose nodes go to fc and fc + 1
// (ploc_aggregate.cpp:481-501).
__device__ __forceinline__ PNode merged_node(const PNode& ni, const PNode& nj,
                                             uint32_t fc) {
  F3 lo, hi;
  join(xyz(nj.a), xyz(nj.b), xyz(ni.a), xyz(ni.b), lo, hi);
  PNode p;
  p.a = make_float4(lo.x, lo.y, lo.z, __int_as_float((int)fc));
  p.b = make_float4(hi.x, hi.y, hi.z, __int_as_float(0));
  return p;
}

// (A cluster's rank is read, not counted over the clusters up to its mate, which
// is up to the search radius away.  100,000 clusters, counted: 78 us an
// iteration at a radius of 1,024 and 15 at 16; read: 6 at both.)
__global__ void __launch_bounds__(kClusterThreads)
    k_cluster(const PlocState* __restrict__ st, int cur, PNode* a, PNode* b,
              const uint32_t* __restrict__ mate,
              const uint16_t* __restrict__ rank,
              const uint32_t* __restrict__ tile_sum, PNode* __restrict__ nodes,
              SahTable sah) {
  const PlocState s = st[cur];
  if (ploc_idle(s)) return;
  const uint32_t first = st[cur ^ 1].end;  // this iteration's nodes start here
  if (st[cur ^ 1].stuck) return;
  const PNode* in = s.buf ? b : a;
  PNode* out = s.buf ? a : b;
  // merges up to and with cluster i
  auto merges = [&](uint32_t i) { return tile_sum[i / kPairTile] + rank[i]; };
  for (uint32_t i = blockIdx.x * kClusterThreads + threadIdx.x; i < s.cnt;
       i += gridDim.x * kClusterThreads) {
    const uint32_t j = mate[i];
    if (j < i) continue;
    const uint32_t mi = merges(i);
    if (j == i) {
      out[i - mi] = in[i];
    } else {
      const uint32_t fc = first + (mi - 1) * 2;
      const PNode ni = in[i], nj = in[j];
      out[j - merges(j)] = merged_node(ni, nj, fc);
      nodes[fc] = ni;
      nodes[fc + 1] = nj;
      sah_node(sah, fc, ni);
      sah_node(sah, fc + 1, nj);
    }
  }
}

// The iterations over at most kTail clusters, in one block: clusters in
// shared memory, a barrier where the other kernels end.  Runs no more
// iterations than there are clusters (each merges a pair or stops).
struct TailMem {
  Box6 box[kTail];
  int first[kTail], count[kTail];
  uint32_t nb[kTail], mi[kTail];
  uint32_t warp[kTailThreads / 32];
};
__global__ void __launch_bounds__(kTailThreads)
    k_cluster_tail(PlocState* st, int cur, const PNode* a, const PNode* b,
                   int r, PNode* nodes, SahTable sah) {
  extern __shared__ char tail_smem[];
  TailMem& m = *reinterpret_cast<TailMem*>(tail_smem);
  PlocState s = st[cur];
  if (s.cnt > kTail || s.stuck) return;
  const PNode* in = s.buf ? b : a;
  constexpr int kPer = kTail / kTailThreads;
  const uint32_t tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  auto put = [&](uint32_t k, const PNode& x) {
    m.box[k] = box6(x);
    m.first[k] = __float_as_int(x.a.w);
    m.count[k] = __float_as_int(x.b.w);
  };
  auto get = [&](uint32_t k) {
    const F3 lo = m.box[k].lo(), hi = m.box[k].hi();
    PNode x;
    x.a = make_float4(lo.x, lo.y, lo.z, __int_as_float(m.first[k]));
    x.b = make_float4(hi.x, hi.y, hi.z, __int_as_float(m.count[k]));
    return x;
  };
  for (uint32_t k = tid; k < s.cnt; k += kTailThreads) put(k, in[k]);
  __syncthreads();
  while (s.cnt > 1) {
    for (uint32_t i = tid; i < s.cnt; i += kTailThreads) {
      const uint32_t s0 = i > (uint32_t)r ? i - r : 0u;
      m.nb[i] = nearest(m.box, i, s0, min(i + (uint32_t)r + 1, s.cnt));
    }
    __syncthreads();
    // merges up to and with each cluster (a thread holds kPer in a row)
    uint32_t mate[kPer], sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const uint32_t i = tid * kPer + k;
      mate[k] = i;
      if (i < s.cnt) {
        const uint32_t j = m.nb[i];
        if (j != 0xffffffffu && m.nb[j] == i) mate[k] = j;
      }
      sum += mate[k] > i;
    }
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) m.warp[warp] = x;
    __syncthreads();
    uint32_t before = 0, merged = 0;
    {
      const uint32_t w = m.warp[lane];
      before = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u);
      merged = __reduce_add_sync(0xffffffffu, w);
    }
    uint32_t run = before + x - sum;
    PNode own[kPer], other[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const uint32_t i = tid * kPer + k;
      if (i >= s.cnt) continue;
      run += mate[k] > i;
      m.mi[i] = run;
      own[k] = get(i);
      if (mate[k] > i) other[k] = get(mate[k]);
    }
    __syncthreads();
    if (merged == 0) {
      s.stuck = 1;
      break;
    }
    s.end -= 2 * merged;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const uint32_t i = tid * kPer + k;
      if (i >= s.cnt) continue;
      const uint32_t mi = m.mi[i], j = mate[k];
      if (j == i) {
        put(i - mi, own[k]);
      } else if (j > i) {
        const uint32_t fc = s.end + (mi - 1) * 2;
        nodes[fc] = own[k];
        nodes[fc + 1] = other[k];
        sah_node(sah, fc, own[k]);
        sah_node(sah, fc + 1, other[k]);
        put(j - m.mi[j], merged_node(own[k], other[k], fc));
      }
    }
    s.cnt -= merged;
    ++s.iters;
    __syncthreads();
  }
  if (tid == 0) {
    if (s.cnt == 1) {
      const PNode root = get(0);
      nodes[0] = root;
      sah_node(sah, 0, root);
    }
    st[cur] = s;
  }
}


__global__ void k_inner_flags(const PNode* __restrict__ nodes, uint64_t m,
                              uint32_t* __restrict__ flags) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
       i += (uint64_t)gridDim.x * blockDim.x)
    flags[i] = __float_as_int(nodes[i].b.w) == 0 ? 1u : 0u;
}

__device__ __forceinline__ int child_ref(const PNode* nodes,
                                         const uint32_t* compact, uint32_t c) {
  const PNode x = nodes[c];
  if (__float_as_int(x.b.w) != 0) return ~__float_as_int(x.a.w);
  return (int)compact[c];
}

__global__ void k_bvh2(const PNode* __restrict__ nodes, uint64_t m,
                       const uint32_t* __restrict__ compact,
                       float4* __restrict__ bvh) {
  for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < m;
       k += (uint64_t)gridDim.x * blockDim.x) {
    const PNode x = nodes[k];
    if (__float_as_int(x.b.w) != 0) continue;
    const uint32_t c0 = (uint32_t)__float_as_int(x.a.w);
    const PNode a = nodes[c0], b = nodes[c0 + 1];
    float4* o = bvh + 4 * (uint64_t)compact[k];
    o[0] = make_float4(a.a.x, a.a.y, a.b.x, a.b.y);
    o[1] = make_float4(b.a.x, b.a.y, b.b.x, b.b.y);
    o[2] = make_float4(a.a.z, a.b.z, b.a.z, b.b.z);
    o[3] = make_float4(__int_as_float(child_ref(nodes, compact, c0)),
                       __int_as_float(child_ref(nodes, compact, c0 + 1)), 0.f,
                       0.f);
  }
}

// A single triangle: one node whose two children are the same leaf.
__global__ void k_bvh2_single(const PNode* __restrict__ nodes,
                              float4* __restrict__ bvh) {
  const PNode a = nodes[0];
  bvh[0] = make_float4(a.a.x, a.a.y, a.b.x, a.b.y);
  bvh[1] = bvh[0];
  bvh[2] = make_float4(a.a.z, a.b.z, a.a.z, a.b.z);
  bvh[3] = make_float4(__int_as_float(~0), __int_as_float(~0), 0.f, 0.f);
}

// Collapse of the binary tree into W-wide nodes, top down, one level of
// wide nodes per launch: a wide node takes its binary node and expands the
// interior child with the largest surface area until it has W children (or
// only leaves); its interior children become the wide nodes of the next
// level, allocated contiguously.  A level's length is a counter of its own
// (n_in, n_out), so levels are enqueued without the host reading them.  Node
// layout (2W float4, 32W bytes) for W = 8: the children's lo.x, hi.x, lo.y,
// hi.y, lo.z, hi.z in groups of four, then the references (>= 0 wide node,
// ~slot leaf, kWideEmpty unused), then padding; for W = 4: wide4_node.
constexpr int kWideEmpty = (int)0x80000000;

// A 4-wide node (8 float4) from its children's planes (lo.x, hi.x, lo.y, hi.y,
// lo.z, hi.z) and references: per child (lo.x, lo.y, hi.x, hi.y), then the
// children's (lo.z, hi.z), the references, padding.
__device__ __forceinline__ void wide4_node(float4* o, const float pl[6][4],
                                           const int rf[4]) {
  for (int c = 0; c < 4; ++c)
    o[c] = make_float4(pl[0][c], pl[2][c], pl[1][c], pl[3][c]);
  o[4] = make_float4(pl[4][0], pl[5][0], pl[4][1], pl[5][1]);
  o[5] = make_float4(pl[4][2], pl[5][2], pl[4][3], pl[5][3]);
  o[6] = make_float4(__int_as_float(rf[0]), __int_as_float(rf[1]),
                     __int_as_float(rf[2]), __int_as_float(rf[3]));
  o[7] = make_float4(0.f, 0.f, 0.f, 0.f);
}

template <int W>
__global__ void k_collapse(const PNode* __restrict__ nodes,
                           const uint2* __restrict__ fin,
                           const uint32_t* __restrict__ n_in_,
                           uint2* __restrict__ fout, uint32_t* n_out,
                           uint32_t* __restrict__ counters,
                           float4* __restrict__ wide) {
  constexpr int G = W / 4;
  const uint32_t n_in = *n_in_;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_in;
       i += gridDim.x * blockDim.x) {
    const uint2 e = fin[i];  // (binary node, wide slot)
    uint32_t ch[W];
    int nc = 1;
    ch[0] = e.x;
    while (nc < W) {
      int best = -1;
      float ba = 0.f;
      for (int c = 0; c < nc; ++c) {
        const PNode x = nodes[ch[c]];
        if (__float_as_int(x.b.w) != 0) continue;  // leaf
        const float a = area(xyz(x.a), xyz(x.b));
        if (best < 0 || a > ba) {
          best = c;
          ba = a;
        }
      }
      if (best < 0) break;
      const uint32_t f = (uint32_t)__float_as_int(nodes[ch[best]].a.w);
      ch[best] = f;
      ch[nc++] = f + 1;
    }
    int ni = 0;
    for (int c = 0; c < nc; ++c)
      ni += __float_as_int(nodes[ch[c]].b.w) == 0 ? 1 : 0;
    uint32_t base = 0, fo = 0;
    if (ni) {
      base = atomicAdd(&counters[0], (uint32_t)ni);
      fo = atomicAdd(n_out, (uint32_t)ni);
    }
    float pl[6][W];
    int rf[W];
    int j = 0;
    for (int c = 0; c < W; ++c) {
      if (c < nc) {
        const PNode x = nodes[ch[c]];
        pl[0][c] = x.a.x;
        pl[1][c] = x.b.x;
        pl[2][c] = x.a.y;
        pl[3][c] = x.b.y;
        pl[4][c] = x.a.z;
        pl[5][c] = x.b.z;
        if (__float_as_int(x.b.w) != 0) {
          rf[c] = ~__float_as_int(x.a.w);
        } else {
          rf[c] = (int)(base + j);
          fout[fo + j] = make_uint2(ch[c], base + j);
          ++j;
        }
      } else {
        for (int k = 0; k < 6; ++k) pl[k][c] = 0.f;
        rf[c] = kWideEmpty;
      }
    }
    float4* o = wide + (uint64_t)e.y * (2 * W);
    if constexpr (W == 4) {
      wide4_node(o, pl, rf);
    } else {
      for (int g = 0; g < G; ++g) {
        for (int k = 0; k < 6; ++k)
          o[k * G + g] = make_float4(pl[k][4 * g], pl[k][4 * g + 1],
                                     pl[k][4 * g + 2], pl[k][4 * g + 3]);
        o[6 * G + g] = make_float4(
            __int_as_float(rf[4 * g]), __int_as_float(rf[4 * g + 1]),
            __int_as_float(rf[4 * g + 2]), __int_as_float(rf[4 * g + 3]));
        o[7 * G + g] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  }
}

// k_collapse with the children of each wide node taken from the dynamic
// program above instead of by expanding the largest-area child.
//
// The order of a node's children is the order any-hit rays take them in (the
// first, then from the last to the second).  Sorted by area, the smallest
// first, they find occluders sooner than in the program's left-to-right order:
// any hits of a 256x256x64 box 1.71 -> 1.45 ms, of 1024x1024x32 paths over
// 1.3 M triangles 25.3 -> 23.2 ms and their packets 7.7 -> 6.4, of 16 batched
// jobs 18.6 -> 17.5; point pairs over 327,682 triangles unchanged, 1 M of them
// in the box 75 -> 67 us and in the emitter box 86 -> 74.  The material box is an
// exception, 85 -> 107.  The largest first, or the most expensive subtree: 1.86
// ms, 25.1, 7.2, 18.6; by subtree cost per area the same as by area.
__global__ void k_collapse_sah(const PNode* __restrict__ nodes,
                               const uint32_t* __restrict__ choice,
                               const uint2* __restrict__ fin,
                               const uint32_t* __restrict__ n_in_,
                               uint2* __restrict__ fout, uint32_t* n_out,
                               uint32_t* __restrict__ counters,
                               float4* __restrict__ wide) {
  constexpr int W = 4;
  const uint32_t n_in = *n_in_;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_in;
       i += gridDim.x * blockDim.x) {
    const uint2 e = fin[i];  // (binary node, wide slot)
    uint32_t ch[W];
    int nc = 0;
    const PNode root = nodes[e.x];
    if (__float_as_int(root.b.w) != 0) {
      ch[nc++] = e.x;  // a one-triangle tree
    } else {
      // (node, slots) still to resolve; each entry holds >= 1 of the 4 slots
      uint32_t sn[W], sj[W];
      int sp = 0;
      const uint32_t f = (uint32_t)__float_as_int(root.a.w);
      const uint32_t k = choice[e.x] & 0xffu;
      sn[sp] = f + 1;
      sj[sp++] = W - k;
      sn[sp] = f;
      sj[sp++] = k;
      while (sp > 0) {
        --sp;
        const uint32_t c = sn[sp], j = sj[sp];
        const uint32_t kd = j < 2 ? 0u : (choice[c] >> (8 * (j - 1))) & 0xffu;
        if (kd == 0u || nc + sp + 2 > W) {  // (the second never holds)
          ch[nc++] = c;
        } else {
          const uint32_t fc = (uint32_t)__float_as_int(nodes[c].a.w);
          const uint32_t k2 = kd >> 4, used = kd & 15u;
          sn[sp] = fc + 1;
          sj[sp++] = used - k2;
          sn[sp] = fc;
          sj[sp++] = k2;
        }
      }
    }
    // interior children by surface area, the smallest first, then the leaves,
    // then the unused slots
    constexpr float kLeaf = 3.402823466e38f;
    float key[W];
    int ni = 0;
#pragma unroll
    for (int c = 0; c < W; ++c) {
      key[c] = __int_as_float(0x7f800000);
      if (c < nc) {
        const PNode x = nodes[ch[c]];
        const bool leaf = __float_as_int(x.b.w) != 0;
        key[c] = leaf ? kLeaf : fminf(area(xyz(x.a), xyz(x.b)), 1e38f);
        ni += leaf ? 0 : 1;
      } else {
        ch[c] = 0;
      }
    }
    auto order = [&](int p, int q) {
      if (key[q] < key[p]) {
        const float tk = key[p];
        key[p] = key[q];
        key[q] = tk;
        const uint32_t tc = ch[p];
        ch[p] = ch[q];
        ch[q] = tc;
      }
    };
    order(0, 1);
    order(2, 3);
    order(0, 2);
    order(1, 3);
    order(1, 2);
    uint32_t base = 0, fo = 0;
    if (ni) {
      base = atomicAdd(&counters[0], (uint32_t)ni);
      fo = atomicAdd(n_out, (uint32_t)ni);
    }
    float pl[6][W];
    int rf[W];
    int jn = 0;
    for (int c = 0; c < W; ++c) {
      if (c < nc) {
        const PNode x = nodes[ch[c]];
        pl[0][c] = x.a.x;
        pl[1][c] = x.b.x;
        pl[2][c] = x.a.y;
        pl[3][c] = x.b.y;
        pl[4][c] = x.a.z;
        pl[5][c] = x.b.z;
        if (__float_as_int(x.b.w) != 0) {
          rf[c] = ~__float_as_int(x.a.w);
        } else {
          rf[c] = (int)(base + jn);
          fout[fo + jn] = make_uint2(ch[c], base + jn);
          ++jn;
        }
      } else {
        for (int k = 0; k < 6; ++k) pl[k][c] = 0.f;
        rf[c] = kWideEmpty;
      }
    }
    float4* o = wide + (uint64_t)e.y * (2 * W);
    wide4_node(o, pl, rf);
  }
}

// The same collapse into compressed nodes (layout in scene.cuh), moving the
// leaf triangles of every node next to each other in `tris_new`.
template <int W>
__global__ void k_collapse_c(const PNode* __restrict__ nodes,
                             const float4* __restrict__ tris_old,
                             const uint2* __restrict__ fin,
                             const uint32_t* __restrict__ n_in_,
                             uint2* __restrict__ fout, uint32_t* n_out,
                             uint32_t* __restrict__ counters,
                             float4* __restrict__ wide,
                             float4* __restrict__ tris_new) {
  constexpr int NF = CwLayout<W>::kFloat4;
  const uint32_t n_in = *n_in_;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_in;
       i += gridDim.x * blockDim.x) {
    const uint2 e = fin[i];
    uint32_t ch[W];
    int nc = 1;
    ch[0] = e.x;
    while (nc < W) {
      int best = -1;
      float ba = 0.f;
      for (int c = 0; c < nc; ++c) {
        const PNode x = nodes[ch[c]];
        if (__float_as_int(x.b.w) != 0) continue;
        const float a = area(xyz(x.a), xyz(x.b));
        if (best < 0 || a > ba) {
          best = c;
          ba = a;
        }
      }
      if (best < 0) break;
      const uint32_t f = (uint32_t)__float_as_int(nodes[ch[best]].a.w);
      ch[best] = f;
      ch[nc++] = f + 1;
    }
    // quantisation grid: origin = lo of the union, 255 steps of 2^e cover
    // the union's extent per axis
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX};
    float hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (int c = 0; c < nc; ++c) {
      const PNode x = nodes[ch[c]];
      lo[0] = fminf(lo[0], x.a.x);
      lo[1] = fminf(lo[1], x.a.y);
      lo[2] = fminf(lo[2], x.a.z);
      hi[0] = fmaxf(hi[0], x.b.x);
      hi[1] = fmaxf(hi[1], x.b.y);
      hi[2] = fmaxf(hi[2], x.b.z);
    }
    uint32_t eb[3];
    float sc[3];
    double step[3];
    for (int a = 0; a < 3; ++a) {
      const double ext = (double)hi[a] - (double)lo[a];
      int ex = -126;
      if (ext > 0.0) {
        int k = 0;
        frexp(ext / 255.0, &k);  // ext / 255 < 2^k
        ex = k;
      }
      ex = ex < -126 ? -126 : (ex > 127 ? 127 : ex);
      eb[a] = (uint32_t)(ex + 127);
      sc[a] = cw_scale(eb[a]);
      step[a] = ldexp(1.0, ex);
    }
    uint32_t vmask = 0, imask = 0;
    uint8_t q[6][W];
    for (int c = 0; c < W; ++c) {
      if (c >= nc) {
        for (int k = 0; k < 6; ++k) q[k][c] = 0;
        continue;
      }
      const PNode x = nodes[ch[c]];
      vmask |= 1u << c;
      if (__float_as_int(x.b.w) == 0) imask |= 1u << c;
      const float cl[3] = {x.a.x, x.a.y, x.a.z};
      const float chh[3] = {x.b.x, x.b.y, x.b.z};
      for (int a = 0; a < 3; ++a) {
        double fl = floor(((double)cl[a] - (double)lo[a]) / step[a]);
        double fh = ceil(((double)chh[a] - (double)lo[a]) / step[a]);
        uint32_t ql = fl < 0.0 ? 0u : (fl > 255.0 ? 255u : (uint32_t)fl);
        uint32_t qh = fh < 0.0 ? 0u : (fh > 255.0 ? 255u : (uint32_t)fh);
        // the decoded planes must enclose the child's box
        while (ql > 0 &&
               cw_decode(lo[a], cw_qfloat(0x4B000000u | ql), sc[a]) > cl[a])
          --ql;
        while (qh < 255 &&
               cw_decode(lo[a], cw_qfloat(0x4B000000u | qh), sc[a]) < chh[a])
          ++qh;
        q[2 * a][c] = (uint8_t)ql;
        q[2 * a + 1][c] = (uint8_t)qh;
      }
    }
    const int ni = __popc(imask), nl = __popc(vmask & ~imask);
    uint32_t base = 0, fo = 0, tb = 0;
    if (ni) {
      base = atomicAdd(&counters[0], (uint32_t)ni);
      fo = atomicAdd(n_out, (uint32_t)ni);
    }
    if (nl) tb = atomicAdd(&counters[1], (uint32_t)nl);
    int ji = 0, jl = 0;
    for (int c = 0; c < nc; ++c) {
      const PNode x = nodes[ch[c]];
      if ((imask >> c) & 1u) {
        fout[fo + ji] = make_uint2(ch[c], base + ji);
        ++ji;
      } else {
        const uint32_t slot = (uint32_t)__float_as_int(x.a.w);
        for (int k = 0; k < 3; ++k)
          tris_new[3 * (uint64_t)(tb + jl) + k] = tris_old[3 * (uint64_t)slot + k];
        ++jl;
      }
    }
    float4* o = wide + (uint64_t)e.y * NF;
    o[0] = make_float4(lo[0], lo[1], lo[2],
                       __uint_as_float(eb[0] | (eb[1] << 8) | (eb[2] << 16) |
                                       (imask << 24)));
    o[1] = make_float4(__uint_as_float(base), __uint_as_float(tb),
                       __uint_as_float(vmask), 0.f);
    uint32_t words[4 * (NF - 2)];
    for (int k = 0; k < 4 * (NF - 2); ++k) words[k] = 0;
    for (int k = 0; k < 6; ++k)
      for (int c = 0; c < W; ++c) {
        const int byte = k * W + c;
        words[byte >> 2] |= (uint32_t)q[k][c] << (8 * (byte & 3));
      }
    for (int f = 0; f < NF - 2; ++f)
      o[2 + f] = make_float4(
          __uint_as_float(words[4 * f]), __uint_as_float(words[4 * f + 1]),
          __uint_as_float(words[4 * f + 2]), __uint_as_float(words[4 * f + 3]));
  }
}

__global__ void k_slot_tris(const float* __restrict__ tris,
                            const int32_t* __restrict__ perm, uint64_t n,
                            float4* __restrict__ out) {
  for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s < n;
       s += (uint64_t)gridDim.x * blockDim.x) {
    const int32_t p = perm[s];
    const float* t = tris + 9 * (uint64_t)p;
    out[3 * s + 0] = make_float4(t[0], t[1], t[2], __int_as_float(p));
    out[3 * s + 1] = make_float4(t[3], t[4], t[5], 0.f);
    out[3 * s + 2] = make_float4(t[6], t[7], t[8], 0.f);
  }
}

// Geometric normal of each primitive as its PostIntersect leaves it:
// normalize(cross(b-a, c-a)) (Triangle::Intersect, quad.cpp, mesh.cpp) or
// from the tuple order (c, b, a) for cubes (cube.cpp:96-108).
__global__ void k_shade_data(const float* __restrict__ tris,
                             const int32_t* __restrict__ mat,
                             const int32_t* __restrict__ flags, uint64_t n,
                             float4* __restrict__ out) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const float* t = tris + 9 * i;
    F3 a = ld3(t), b = ld3(t + 3), c = ld3(t + 6);
    const int fl = flags[i];
    F3 ng = (fl & AJG_MESH_NG_REVERSED) ? normalize3(cross3(b - c, a - c))
                                        : normalize3(cross3(b - a, c - a));
    const uint32_t w = ((uint32_t)mat[i] & 0xffffffu) | ((uint32_t)fl << 24);
    out[i] = make_float4(ng.x, ng.y, ng.z, __uint_as_float(w));
  }
}

// The build's temporaries: the context's kept scratch, or past kScratchKeep
// an allocation of its own.
struct BuildMem {
  Scratch scratch;
  void* own = nullptr;
  char* p = nullptr;
  bool take(ajg_ctx* ctx, uint64_t bytes, cudaStream_t st) {
    if (bytes <= kScratchKeep) {
      if (scratch.take(ctx, bytes, st) != cudaSuccess) return false;
      p = scratch.p;
      return true;
    }
    if (!device_malloc(ctx, &own, bytes)) return false;
    p = static_cast<char*>(own);
    return true;
  }
  ~BuildMem() {
    if (own) cudaFree(own);
  }
};

// The arrays only shading reads, copied in on the trace stream while the
// tree is built (1,310,722 triangles: 58 of 105 MB, 330 us); done before the
// build returns, whichever way it does.  Two of them lie in the kept scratch,
// which the renders enqueued before may still be using on the context's
// stream (ajg_render_device returns with its film there): the trace stream
// waits for that stream as it was when the scratch was taken.
struct ShadingCopy {
  ajg_ctx* ctx;
  bool started = false;
  explicit ShadingCopy(ajg_ctx* c) : ctx(c) {
    cudaEventRecord(ctx->ev_queue, ctx->stream);
    cudaStreamWaitEvent(ctx->trace_stream, ctx->ev_queue, 0);
  }
  void start(int32_t* d_mat, const int32_t* mat, int32_t* d_flags,
             const int32_t* flags, float* d_corner, const float* corner,
             uint64_t n) {
    started = true;
    cudaStream_t ts = ctx->trace_stream;
    cudaMemcpyAsync(d_mat, mat, n * sizeof(int32_t), cudaMemcpyHostToDevice, ts);
    cudaMemcpyAsync(d_flags, flags, n * sizeof(int32_t), cudaMemcpyHostToDevice, ts);
    if (d_corner)
      cudaMemcpyAsync(d_corner, corner, n * 9 * sizeof(float),
                      cudaMemcpyHostToDevice, ts);
    cudaEventRecord(ctx->ev_queue, ts);
  }
  ~ShadingCopy() {
    if (started) cudaStreamSynchronize(ctx->trace_stream);
  }
};

// The GPU time of a build: the spans between begin and end, which leave out the
// copies in and the host's share (from pageable memory the copies of the
// shading arrays hold the host, and the stream waits for both).
struct BuildTimer {
  ajg_ctx* ctx;
  int n = 0;  // events recorded
  explicit BuildTimer(ajg_ctx* c) : ctx(c) {
    for (cudaEvent_t& e : ctx->ev_build)
      if (!e) cudaEventCreate(&e);
  }
  void mark() { cudaEventRecord(ctx->ev_build[n++], ctx->stream); }
  float ms() const {
    float sum = 0.f;
    for (int k = 0; k + 1 < n; k += 2) {
      float t = 0.f;
      cudaEventElapsedTime(&t, ctx->ev_build[k], ctx->ev_build[k + 1]);
      sum += t;
    }
    return sum;
  }
};

int set_err(ajg_ctx* ctx, int code, const std::string& msg) {
  ctx->last_error = msg;
  return code;
}

// The scene's typical triangle size: the median longest edge over up to
// 4,096 evenly spaced triangles.
float median_edge(const float* t, uint64_t n) {
  const uint64_t k = std::min<uint64_t>(n, 4096);
  std::vector<float> e(k);
  for (uint64_t i = 0; i < k; ++i) {
    const float* p = t + 9 * (i * n / k);
    float m = 0.f;
    for (int a = 0; a < 3; ++a) {
      const float* u = p + 3 * a;
      const float* v = p + 3 * ((a + 1) % 3);
      const float dx = u[0] - v[0], dy = u[1] - v[1], dz = u[2] - v[2];
      m = std::max(m, dx * dx + dy * dy + dz * dz);
    }
    e[i] = std::sqrt(m);
  }
  std::nth_element(e.begin(), e.begin() + k / 2, e.end());
  return e[k / 2];
}

}  // namespace

int build_scene(ajg_ctx* ctx, ajg_scene* s, const float* h_tris,
                const float* h_corner, const int32_t* h_mat,
                const int32_t* h_flags, uint64_t n, const float* world,
                const ajg_scene_opts& opts) {
  cudaStream_t st = ctx->stream;
  if (n == 0 || n > (1ull << 30))
    return set_err(ctx, AJG_ERR_INVALID, "triangle count must be in [1, 2^30]");
  const int r = (int)opts.search_radius;
  if (r < 1 || r > 1024)
    return set_err(ctx, AJG_ERR_INVALID, "search_radius must be in [1, 1024]");
  const uint64_t m = 2 * n - 1;
  bool any_normals = false;
  for (uint64_t i = 0; i < n && h_corner; ++i)
    if (h_flags[i] & AJG_MESH_HAS_NORMALS) {
      any_normals = true;
      break;
    }

  const uint64_t inner = n > 1 ? n - 1 : 1;
  // default: the 4-wide tree (the fastest measured on GB300 for the
  // workloads here; 8-wide nodes cost occupancy)
  const int width = opts.bvh_width ? (int)opts.bvh_width : 4;
  const bool compressed = (width & kBvhCompressed) != 0;
  const int wn = width & 0xff;  // children per node
  if (!(width == 2 || wn == 4 || wn == 8) || (width & ~0x1ff))
    return set_err(ctx, AJG_ERR_INVALID,
                   "bvh_width must be 0, 2, 4 or 8 (4 and 8 optionally "
                   "| AJG_BVH_COMPRESSED)");
  // the binary layout: the tree itself (width 2), or beside a plain 4-wide
  // tree for the closest-hit traversal (closest_width)
  const bool hybrid = closest_width(width) != width;
  const bool wide = width != 2;
  const bool sah = AJG_SAH_COLLAPSE && wn == 4 && !compressed;
  const uint64_t node_f4 =
      compressed ? (wn == 8 ? CwLayout<8>::kFloat4 : CwLayout<4>::kFloat4)
                 : 2 * (uint64_t)wn;

  // persistent scene buffers: one allocation (the wide tree, whose size the
  // collapse finds, is the other)
  float4 *bvh = nullptr, *bvh_bin = nullptr, *slot_tris, *shade, *ploc_nodes;
  float* corner = nullptr;
  int32_t* perm_keep;
  uint64_t kept = 0;  // bytes in use
  auto layout = [&](char* cur) {
    kept = 0;
    auto get = [&](auto* type, uint64_t count) {
      using T = std::remove_pointer_t<decltype(type)>;
      kept += count * sizeof(T);
      return carve<T>(cur, count);
    };
    if (!wide) bvh = get((float4*)nullptr, inner * 4);
    if (hybrid) bvh_bin = get((float4*)nullptr, inner * 4);
    slot_tris = get((float4*)nullptr, n * 3);
    shade = get((float4*)nullptr, n);
    if (any_normals) corner = get((float*)nullptr, n * 9);
    ploc_nodes = get((float4*)nullptr, 2 * m);
    perm_keep = get((int32_t*)nullptr, n);
    return cur;
  };
  void* block = nullptr;
  if (!device_malloc(ctx, &block, (uint64_t)(uintptr_t)layout(nullptr)))
    return set_err(ctx, AJG_ERR_OOM, "device allocation failed (scene)");
  s->allocations.push_back(block);
  layout(static_cast<char*>(block));
  s->info.device_bytes += kept;

  float* d_tris;
  int32_t *d_mat, *d_flags, *va, *vb, *owner = nullptr;
  uint16_t* rank;
  uint32_t *ka, *kb, *hist, *scratch, *pos_of = nullptr, *acc, *nbr, *mate, *tile_sum,
      *flags = nullptr, *mi = nullptr, *choice = nullptr, *wc = nullptr;
  PNode *na, *nbuf;
  PlocState* state;
  float4 *cost = nullptr, *wtmp = nullptr, *tri_tmp = nullptr;
  uint2 *fa = nullptr, *fb = nullptr;
  const bool small_sort = n <= kSmallSort;
  const uint64_t radix_tile =
      (uint64_t)kRadixWarps * (small_sort ? kKeysPerWarpSmall : kKeysPerWarp);
  const uint32_t nbt = (uint32_t)((n + radix_tile - 1) / radix_tile);
  const uint64_t hist_n = (uint64_t)kBuckets * nbt;
  auto temporaries = [&](char* cur) {
    d_tris = carve<float>(cur, n * 9);
    d_mat = carve<int32_t>(cur, n);
    d_flags = carve<int32_t>(cur, n);
    ka = carve<uint32_t>(cur, n);
    kb = carve<uint32_t>(cur, n);
    va = carve<int32_t>(cur, n);
    vb = carve<int32_t>(cur, n);
    hist = carve<uint32_t>(cur, hist_n);
    scratch = carve<uint32_t>(cur, scan_scratch_words(hist_n > m ? hist_n : m));
    if (opts.radix_compat) {
      owner = carve<int32_t>(cur, n);
      pos_of = carve<uint32_t>(cur, n);
    }
    acc = carve<uint32_t>(cur, 2);  // the sort's, then the clustering's ticket
    na = carve<PNode>(cur, n);
    nbuf = carve<PNode>(cur, n);
    nbr = carve<uint32_t>(cur, n);
    mate = carve<uint32_t>(cur, n);
    rank = carve<uint16_t>(cur, n);
    tile_sum = carve<uint32_t>(cur, (n + kPairTile - 1) / kPairTile);
    state = carve<PlocState>(cur, 2);
    if (!wide || hybrid) {
      flags = carve<uint32_t>(cur, m);
      mi = carve<uint32_t>(cur, m);
    }
    if (sah) {
      cost = carve<float4>(cur, m);
      choice = carve<uint32_t>(cur, m);
    }
    if (wide) {
      wtmp = carve<float4>(cur, inner * node_f4);
      if (compressed) tri_tmp = carve<float4>(cur, 3 * n);
      fa = carve<uint2>(cur, inner);
      fb = carve<uint2>(cur, inner);
      wc = carve<uint32_t>(cur, 2 + kLevels + 1);
    }
    return cur;
  };
  BuildMem tmp;
  if (!tmp.take(ctx, (uint64_t)(uintptr_t)temporaries(nullptr), st))
    return set_err(ctx, AJG_ERR_OOM, "device allocation failed (PLOC build)");
  temporaries(tmp.p);
  ShadingCopy shading(ctx);

  BuildTimer timer(ctx);
  cudaMemcpyAsync(d_tris, h_tris, n * 9 * sizeof(float),
                  cudaMemcpyHostToDevice, st);
  cudaMemsetAsync(ctx->d_error, 0, sizeof(uint32_t), st);
  timer.mark();

  // MortonEncoder (ploc_aggregate.cpp:61-66): grid = 1024 / size, offset =
  // -min * grid, all in float
  const F3 wlo = mk3(world[0], world[1], world[2]);
  const F3 whi = mk3(world[3], world[4], world[5]);
  const F3 size = whi - wlo;
  const F3 inv = mk3(1.f / size.x, 1.f / size.y, 1.f / size.z);
  const F3 w2g = inv * 1024.f;
  const F3 off = (-wlo) * w2g;
  const int gb = grid_for(n, 256);
  k_morton<<<gb, 256, 0, st>>>(d_tris, n, w2g, off, ka, va);

  // three 10-bit passes; compat passes scatter into buffers whose stale
  // contents match the reference's (zeroed copies, then originals, ...)
  if (opts.radix_compat) {
    cudaMemsetAsync(kb, 0, n * sizeof(uint32_t), st);
    cudaMemsetAsync(vb, 0, n * sizeof(int32_t), st);
    cudaMemsetAsync(acc, 0, 2 * sizeof(uint32_t), st);
  }
  uint32_t* kin = ka;
  uint32_t* kout = kb;
  int32_t* vin = va;
  int32_t* vout = vb;
  for (int bit = 0; bit < 30; bit += 10) {
    if (small_sort)
      k_radix_hist<kKeysPerWarpSmall><<<nbt, kRadixThreads, 0, st>>>(kin, n, bit, hist, nbt);
    else
      k_radix_hist<kKeysPerWarp><<<nbt, kRadixThreads, 0, st>>>(kin, n, bit, hist, nbt);
    device_scan(hist, hist, hist_n, true, scratch, st);
    if (opts.radix_compat) {
      k_compat_base<<<1, 1, 0, st>>>(hist, nbt, acc);
      cudaMemsetAsync(owner, 0xff, n * sizeof(int32_t), st);
    }
    auto* scatter = small_sort ? k_radix_scatter<kKeysPerWarpSmall>
                               : k_radix_scatter<kKeysPerWarp>;
    scatter<<<nbt, kRadixThreads, 0, st>>>(
        kin, vin, kout, vout, n, bit, hist, nbt, opts.radix_compat ? 1 : 0,
        acc, owner, pos_of, ctx->d_error);
    if (opts.radix_compat)
      k_radix_compat_write<<<gb, 256, 0, st>>>(kin, vin, kout, vout, n, owner,
                                               pos_of);
    std::swap(kin, kout);
    std::swap(vin, vout);
  }
  const int32_t* perm = vin;  // sorted values after three passes

  // leaves, then cluster until one node remains: a batch of iterations is
  // enqueued, then the one-block tail, and the state read once.  An iteration
  // leaves about four of five clusters (1,310,722 triangles: 62 iterations in
  // all), so the first batch rarely needs a second; iterations past the end
  // cost three empty launches.
  PNode* nodes = reinterpret_cast<PNode*>(ploc_nodes);
  const SahTable table{cost, choice};
  k_leaf_init<<<gb, 256, 0, st>>>(d_tris, perm, na, n);
  k_ploc_start<<<1, 1, 0, st>>>(state, (uint32_t)n, acc);
  const size_t smem = (size_t)(kClusterThreads + 2 * r) * sizeof(Box6);
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(k_neighbors,
                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem);
  cudaFuncSetAttribute(k_cluster_tail, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)sizeof(TailMem));
  const int g_nb = grid_for(n, kClusterThreads, kSMs * 8);
  const int g_pair = grid_for(n, kPairTile, kSMs * 8);
  PlocState h{};
  int batch = n > kTail ? (int)std::ceil(std::log((double)n / kTail) / std::log(1.25)) + 1
                        : 0;
  uint64_t it = 0;
  for (;;) {
    for (int k = 0; k < batch; ++k, ++it) {
      const int cur = (int)(it & 1);
      k_neighbors<<<g_nb, kClusterThreads, smem, st>>>(state + cur, na, nbuf, r, nbr);
      k_pairs<<<g_pair, kClusterThreads, 0, st>>>(state, cur, nbr, mate, rank,
                                                  tile_sum, acc);
      k_cluster<<<g_nb, kClusterThreads, 0, st>>>(state, cur, na, nbuf, mate, rank,
                                                  tile_sum, nodes, table);
    }
    k_cluster_tail<<<1, kTailThreads, sizeof(TailMem), st>>>(
        state, (int)(it & 1), na, nbuf, r, nodes, table);
    if (!shading.started) {  // beside the clustering
      timer.mark();
      shading.start(d_mat, h_mat, d_flags, h_flags, corner, h_corner, n);
    }
    cudaError_t e = cudaMemcpyAsync(&h, state + (it & 1), sizeof(h),
                                    cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess)
      return set_err(ctx, AJG_ERR_CUDA,
                     std::string("PLOC build: ") + cudaGetErrorString(e));
    if (timer.n == 2) timer.mark();
    if (h.iters > kMaxIterations)  // ended or not: the last batch and the
                                   // tail do not stop at the limit
      return set_err(ctx, AJG_ERR_DEVICE, "PLOC did not converge");
    if (h.stuck)
      return set_err(ctx, AJG_ERR_DEVICE, "PLOC iteration merged no pair");
    if (h.cnt == 1) break;
    batch = 8;
  }
  const uint32_t iters = h.iters;

  // traversal layout
  cudaMemcpyAsync(perm_keep, perm, n * sizeof(int32_t),
                  cudaMemcpyDeviceToDevice, st);
  uint32_t num_nodes = (uint32_t)inner;
  if (width == 2) {
    if (n > 1) {
      k_inner_flags<<<grid_for(m, 256), 256, 0, st>>>(nodes, m, flags);
      device_scan(flags, mi, m, true, scratch, st);
      k_bvh2<<<grid_for(m, 256), 256, 0, st>>>(nodes, m, mi, bvh);
    } else {
      k_bvh2_single<<<1, 1, 0, st>>>(nodes, bvh);
    }
  } else {
    if (hybrid && n > 1) {
      k_inner_flags<<<grid_for(m, 256), 256, 0, st>>>(nodes, m, flags);
      device_scan(flags, mi, m, true, scratch, st);
      k_bvh2<<<grid_for(m, 256), 256, 0, st>>>(nodes, m, mi, bvh_bin);
    } else if (hybrid) {
      k_bvh2_single<<<1, 1, 0, st>>>(nodes, bvh_bin);
    }
    // wide layout: collapse level by level into a worst-case buffer, then
    // keep the nodes made; the triangles move into node order for compressed
    // nodes.  wc: wide nodes, triangles moved, then the levels' lengths.
    k_slot_tris<<<gb, 256, 0, st>>>(d_tris, perm, n, slot_tris);
    uint32_t init[3] = {1u, 0u, 1u};
    const uint2 root = make_uint2(0u, 0u);
    cudaMemcpyAsync(fa, &root, sizeof(root), cudaMemcpyHostToDevice, st);
    const int g = grid_for(inner, 128, kSMs * 16);
    int levels = std::min(kLevels, 6 + (int)(0.6 * std::log2((double)n)));
    uint64_t done = 0;
    for (;;) {
      cudaMemsetAsync(wc + 3, 0, kLevels * sizeof(uint32_t), st);
      cudaMemcpyAsync(wc, init, sizeof(init), cudaMemcpyHostToDevice, st);
      for (int l = 0; l < levels; ++l) {
        const uint32_t* ni = wc + 2 + l;
        uint32_t* no = wc + 3 + l;
        if (compressed && wn == 4)
          k_collapse_c<4><<<g, 128, 0, st>>>(nodes, slot_tris, fa, ni, fb, no, wc,
                                             wtmp, tri_tmp);
        else if (compressed)
          k_collapse_c<8><<<g, 128, 0, st>>>(nodes, slot_tris, fa, ni, fb, no, wc,
                                             wtmp, tri_tmp);
        else if (sah)
          k_collapse_sah<<<g, 128, 0, st>>>(nodes, choice, fa, ni, fb, no, wc, wtmp);
        else if (wn == 4)
          k_collapse<4><<<g, 128, 0, st>>>(nodes, fa, ni, fb, no, wc, wtmp);
        else
          k_collapse<8><<<g, 128, 0, st>>>(nodes, fa, ni, fb, no, wc, wtmp);
        std::swap(fa, fb);
      }
      uint32_t hw[2 + kLevels + 1];
      if (cudaMemcpyAsync(hw, wc, sizeof(hw), cudaMemcpyDeviceToHost, st) !=
              cudaSuccess ||
          cudaStreamSynchronize(st) != cudaSuccess)
        return set_err(ctx, AJG_ERR_CUDA, "wide BVH collapse failed");
      num_nodes = hw[0];
      if (hw[2 + levels] == 0) break;
      done += levels;
      if (done > inner + 1)
        return set_err(ctx, AJG_ERR_DEVICE, "wide BVH collapse did not end");
      init[0] = hw[0];
      init[1] = hw[1];
      init[2] = hw[2 + levels];
      levels = kLevels;
    }
    // (not device_malloc: the temporaries are in the kept scratch)
    const uint64_t bytes = (uint64_t)num_nodes * node_f4 * sizeof(float4);
    if (cudaMalloc((void**)&bvh, bytes) != cudaSuccess) {
      cudaGetLastError();
      return set_err(ctx, AJG_ERR_OOM, "device allocation failed (wide BVH)");
    }
    s->allocations.push_back(bvh);
    s->info.device_bytes += bytes;
    cudaMemcpyAsync(bvh, wtmp, bytes, cudaMemcpyDeviceToDevice, st);
    if (compressed)
      cudaMemcpyAsync(slot_tris, tri_tmp, 3 * n * sizeof(float4),
                      cudaMemcpyDeviceToDevice, st);
  }
  if (width == 2) k_slot_tris<<<gb, 256, 0, st>>>(d_tris, perm, n, slot_tris);
  timer.mark();
  cudaStreamWaitEvent(st, ctx->ev_queue, 0);
  timer.mark();
  k_shade_data<<<gb, 256, 0, st>>>(d_tris, d_mat, d_flags, n, shade);
  timer.mark();
  cudaError_t ce = cudaStreamSynchronize(st);
  uint32_t derr = 0;
  if (ce == cudaSuccess)
    ce = cudaMemcpy(&derr, ctx->d_error, sizeof(uint32_t),
                    cudaMemcpyDeviceToHost);
  const float ms = timer.ms();
  if (ce != cudaSuccess)
    return set_err(ctx, AJG_ERR_CUDA,
                   std::string("PLOC build: ") + cudaGetErrorString(ce));
  if (derr == kDevSortOutOfBounds)
    return set_err(ctx, AJG_ERR_INVALID,
                   "radix_compat: the reference's sort would write out of "
                   "bounds on this input");
  if (derr)
    return set_err(ctx, AJG_ERR_DEVICE, "device guard tripped in PLOC build");

  s->d.bvh = bvh;
  s->d.bvh_closest = bvh_bin;
  s->d.num_inner_closest = hybrid ? (uint32_t)inner : 0u;
  s->info.closest_node_bytes = 0;  // set with bvh_node_bytes below
  s->d.tris = slot_tris;
  s->d.shade = shade;
  s->d.corner = corner;
  s->d.n = n;
  s->d.num_inner = num_nodes;
  s->d.width = width;
  s->d.tri_test = (int32_t)opts.tri_test;
  s->ploc_nodes = ploc_nodes;
  s->perm = perm_keep;
  s->info.num_triangles = n;
  s->info.num_nodes = m;
  s->info.ploc_iterations = iters;
  s->info.build_ms = ms;
  s->info.bvh_width = (uint32_t)width;
  s->info.bvh_node_bytes =
      width == 2 ? 64u
                 : (compressed ? 16u * (wn == 8 ? CwLayout<8>::kFloat4
                                                : CwLayout<4>::kFloat4)
                               : 32u * (uint32_t)wn);
  s->info.bvh_nodes = num_nodes;
  s->info.closest_node_bytes = hybrid ? 64u : s->info.bvh_node_bytes;
  for (int k = 0; k < 6; ++k) s->world[k] = world[k];
  // lights are fitted to the world bounds (default_scene.cpp:41-48)
  const F3 center = (whi + wlo) / 2.f;
  const F3 half = whi - center;
  float d = 0.f;
  d += half.x * half.x;
  d += half.y * half.y;
  d += half.z * half.z;
  s->d.radius = sqrtf(d);
  s->d.packet_spread = kPacketSpread * median_edge(h_tris, n);
  return AJG_OK;
}

}  // namespace ajg
