// Stochastic progressive photon mapping: SPPMRenderer::Render
// (core/renderer/sppm.cpp:180-296) on the GPU.
//
// The camera pass (TracerVP) runs once through the path-tracing wave
// (sppm_camera_pass): the reference reseeds every pixel each iteration, so
// every iteration finds the same visible points and the same direct light.
// Per iteration:
//   the visible-point grid -- the reference's VisiblePointSearcher
//     (photon_mapping.h:69-148): 40960 hash entries, each visible point
//     filed under the cells [lo, hi) of its radius box -- built as count,
//     scan and fill over the entries instead of linked lists;
//   the photon pass (TracerPhoton, sppm.cpp:103-143) as a wavefront, of one
//     iteration or several (photons do not depend on the visible points): emit
//     from a light chosen by the scene's uniform selector, then per depth a
//     closest-hit traversal and a shading kernel that records the photon's
//     deposit and samples the BSDF; roulette draws as the reference draws
//     them;
//   the deposits (AddPhoton: EvalAll at each visible point of the photon's
//     entry within its radius) of all depths of an iteration at once, or of
//     the depths a record buffer holds (photon_plan.cuh): the records sorted
//     by hash entry and joined entry by entry with the grid's visible points
//     (k_deposit);
//   the radius reduction and UpdatePixel (sppm.cpp:145-169).
// Photon i of iteration k draws from path_key(photon_seed(seed), i, k).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "photon_plan.cuh"
#include "shade.cuh"
#include "trace.cuh"

namespace ajg {
namespace {

constexpr uint32_t kEntries = 40960;   // VisiblePointSearcher(..., 40960)
constexpr int kMaxCellsPerAxis = 4;    // a radius box spans <= 3 cells
constexpr int kThreads = 128;
constexpr unsigned kFull = 0xffffffffu;

int fail(ajg_ctx* ctx, int code, const std::string& m) {
  ctx->last_error = m;
  return code;
}

// photon streams (the oracle's ajg_photon_seed)
__host__ __device__ __forceinline__ uint64_t photon_seed(uint64_t seed) {
  return mix64(seed ^ 0x50484F544F4E5321ull);
}

// Per-render constants.
struct SppmArgs {
  DeviceScene s;
  F3 lo;              // world bounds grown by the initial radius
  F3 center;          // world centre (the lights' emission disks)
  float init_radius;
  uint64_t pseed;     // photon stream seed
  uint32_t npix;
  // a photon wave: photons [i0, i0 + m) of each iteration from it0 on
  uint32_t it0, i0, m;
  int pmin, pmax;
  float cont;
  // DefaultScene's light selector (default_scene.cpp:48-53, 77-86)
  float cdf[16];
  float lpdf;
  uint32_t nl;
};

// Per-pixel state (sppm::Pixel, photon_mapping.h:54-67).
struct SppmPixels {
  const VisPointD* vp;
  const float4* direct;
  float* radius;
  float* N;
  uint32_t* M;
  float4* phi;
  float4* tau;
};

struct Grid {
  uint32_t* counts;   // [kEntries]
  uint32_t* offsets;  // [kEntries + 1]
  uint32_t* cursor;   // [kEntries]
  uint32_t* items;    // pixel indices, entry by entry
  float4* spheres;    // per item: the visible point and radius^2, so the
                      // distance test of a deposit reads one 16-byte record
  uint32_t cap;
  const float* maxr;  // this iteration's max radius (the cell side / 1.05)
};

// VisiblePointSearcher::ToGrid and ToEntry (photon_mapping.h:123-139).
__device__ __forceinline__ void to_grid(F3 pos, F3 lo, float side, int c[3]) {
  const F3 hd = pos - lo;
  c[0] = (int)((hd.x < 0.f ? 0.f : hd.x) / side);
  c[1] = (int)((hd.y < 0.f ? 0.f : hd.y) / side);
  c[2] = (int)((hd.z < 0.f ? 0.f : hd.z) / side);
}
__device__ __forceinline__ uint64_t hash_combine(uint64_t a, uint64_t b) {
  return a ^ (b + 0x9e3779b97f4a7c15ull + (a << 6) + (a >> 2));
}
__device__ __forceinline__ uint32_t to_entry(int x, int y, int z) {
  const uint64_t low3 = (uint64_t)(((x & 1) << 0) | ((y & 1) << 1) | (z & 2));
  uint64_t h = (uint64_t)(int64_t)x;  // std::hash<int>
  h = hash_combine(h, (uint64_t)(int64_t)y);
  h = hash_combine(h, (uint64_t)(int64_t)z);
  return (uint32_t)(((h << 3) % kEntries) | low3);
}

__device__ __forceinline__ bool has_vp(const VisPointD& v) {
  return __float_as_uint(v.pos.w) != kNoVisPoint;
}

// AddVp's cell range of pixel i (photon_mapping.h:80-96); false when the
// box spans more cells than a radius below the cell side allows.
__device__ __forceinline__ bool vp_cells(const SppmArgs& a,
                                         const SppmPixels& px, const Grid& g,
                                         uint32_t i, int lo[3], int hi[3]) {
  const float side = 1.05f * *g.maxr;
  const F3 pos = xyz(px.vp[i].pos);
  const float r = px.radius[i];
  to_grid(pos - mk3(r, r, r), a.lo, side, lo);
  to_grid(pos + mk3(r, r, r), a.lo, side, hi);
  for (int k = 0; k < 3; ++k)
    if (hi[k] - lo[k] > kMaxCellsPerAxis) return false;
  return true;
}

__global__ void k_grid_count(SppmArgs a, SppmPixels px, Grid g,
                             uint32_t* err) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.npix;
       i += gridDim.x * blockDim.x) {
    if (!has_vp(px.vp[i])) continue;
    int lo[3], hi[3];
    if (!vp_cells(a, px, g, i, lo, hi)) {
      raise_device_error(err, kDevIterationBound);
      continue;
    }
    for (int z = lo[2]; z < hi[2]; ++z)
      for (int y = lo[1]; y < hi[1]; ++y)
        for (int x = lo[0]; x < hi[0]; ++x)
          atomicAdd(&g.counts[to_entry(x, y, z)], 1u);
  }
}

// The deposits of one iteration's photons of a wave.  A record is three
// float4: position and power, incoming direction, and -- filled in once the
// iteration's grid stands (k_deposit_enter) -- hash entry and rank among the
// entry's deposits.  `hist` counts an entry's deposits, `offsets` and `units`
// are their exclusive scans (k_entry_scan), `sorted` the records' indices
// entry by entry.
struct Deposits {
  float4* rec;                // [cap][3]; a wave's iterations one after the other
  uint32_t* count;            // one per iteration of the wave
  uint32_t* hist;             // [kEntries]
  uint32_t* offsets;          // [kEntries + 1]
  unsigned long long* units;  // [kEntries + 1]
  uint32_t* sorted;           // [cap]
  uint32_t cap;
};

// Exclusive scans over the hash entries: a block per 1,024 entries sums its
// own (k_entry_totals), then scans them from the blocks before it
// (k_entry_scan).  Two short launches: one block over all 40,960 entries
// took 65 us an iteration, most of it its own serial reads and writes.
constexpr int kEntryThreads = 1024;
constexpr int kEntryBlocks = kEntries / kEntryThreads;
static_assert(kEntries % kEntryThreads == 0 && kEntryBlocks <= 64, "entry blocks");
struct EntryVal {
  uint32_t n;            // items, or deposits
  unsigned long long u;  // units of k_deposit
};
// The work of k_deposit is cut into units of 32 visible points x 32 deposits
// of one entry.
template <bool DEP>
__device__ __forceinline__ EntryVal entry_val(const Grid& g, const Deposits& d,
                                              uint32_t e) {
  EntryVal v;
  if constexpr (DEP) {
    v.n = d.hist[e];
    const uint32_t i0 = min(g.offsets[e], g.cap), i1 = min(g.offsets[e + 1], g.cap);
    v.u = (unsigned long long)((i1 - i0 + 31) / 32) * ((v.n + 31) / 32);
  } else {
    v.n = g.counts[e];
    v.u = 0;
  }
  return v;
}
template <bool DEP>
__global__ void __launch_bounds__(kEntryThreads)
    k_entry_totals(Grid g, Deposits d, EntryVal* totals) {
  __shared__ EntryVal s_w[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  EntryVal v = entry_val<DEP>(g, d, blockIdx.x * kEntryThreads + threadIdx.x);
  for (int o = 16; o > 0; o >>= 1) {
    v.n += __shfl_xor_sync(kFull, v.n, o);
    if constexpr (DEP) v.u += __shfl_xor_sync(kFull, v.u, o);
  }
  if (lane == 0) s_w[warp] = v;
  __syncthreads();
  if (warp == 0) {
    v = s_w[lane];
    for (int o = 16; o > 0; o >>= 1) {
      v.n += __shfl_xor_sync(kFull, v.n, o);
      if constexpr (DEP) v.u += __shfl_xor_sync(kFull, v.u, o);
    }
    if (lane == 0) totals[blockIdx.x] = v;
  }
}
template <bool DEP>
__global__ void __launch_bounds__(kEntryThreads)
    k_entry_scan(Grid g, Deposits d, const EntryVal* totals) {
  __shared__ EntryVal s_w[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t e = blockIdx.x * kEntryThreads + threadIdx.x;
  const EntryVal own = entry_val<DEP>(g, d, e);
  EntryVal x = own;  // inclusive within the warp
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t n = __shfl_up_sync(kFull, x.n, o);
    const unsigned long long u = DEP ? __shfl_up_sync(kFull, x.u, o) : 0ull;
    if (lane >= o) {
      x.n += n;
      x.u += u;
    }
  }
  if (lane == 31) s_w[warp] = x;
  __syncthreads();
  if (warp == 0) {
    // the warps' exclusive prefix, from the totals of the blocks before
    EntryVal w = s_w[lane];
    const EntryVal last = w;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t n = __shfl_up_sync(kFull, w.n, o);
      const unsigned long long u = DEP ? __shfl_up_sync(kFull, w.u, o) : 0ull;
      if (lane >= o) {
        w.n += n;
        w.u += u;
      }
    }
    EntryVal b{0u, 0ull};
    for (int k = lane; k < (int)blockIdx.x; k += 32) {
      b.n += totals[k].n;
      b.u += totals[k].u;
    }
    for (int o = 16; o > 0; o >>= 1) {
      b.n += __shfl_xor_sync(kFull, b.n, o);
      if constexpr (DEP) b.u += __shfl_xor_sync(kFull, b.u, o);
    }
    s_w[lane] = EntryVal{w.n - last.n + b.n, w.u - last.u + b.u};
  }
  __syncthreads();
  const uint32_t n0 = s_w[warp].n + x.n - own.n;
  const unsigned long long u0 = s_w[warp].u + x.u - own.u;
  if constexpr (DEP) {
    d.offsets[e] = n0;
    d.units[e] = u0;
    if (e == kEntries - 1) {
      d.offsets[kEntries] = n0 + own.n;
      d.units[kEntries] = u0 + own.u;
    }
  } else {
    g.offsets[e] = n0;
    g.cursor[e] = 0;
    if (e == kEntries - 1) g.offsets[kEntries] = n0 + own.n;
  }
}

__global__ void k_grid_fill(SppmArgs a, SppmPixels px, Grid g,
                            uint32_t* err) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.npix;
       i += gridDim.x * blockDim.x) {
    if (!has_vp(px.vp[i])) continue;
    int lo[3], hi[3];
    if (!vp_cells(a, px, g, i, lo, hi)) continue;
    for (int z = lo[2]; z < hi[2]; ++z)
      for (int y = lo[1]; y < hi[1]; ++y)
        for (int x = lo[0]; x < hi[0]; ++x) {
          const uint32_t e = to_entry(x, y, z);
          const uint32_t slot = g.offsets[e] + atomicAdd(&g.cursor[e], 1u);
          if (slot >= g.cap) {
            raise_device_error(err, kDevQueueOverflow);
            continue;
          }
          const float4 p4 = px.vp[i].pos;
          const float r = px.radius[i];
          g.items[slot] = i;
          g.spheres[slot] = make_float4(p4.x, p4.y, p4.z, r * r);
        }
  }
}

// The photon queue (double buffered): ro.w = photon index bits, rd.w = the
// photon's next sampler dimension, coef = its power.
struct PhotonQ {
  float4* ro[2];
  float4* rd[2];
  float4* coef[2];
  ajg_hit* hits;
  uint32_t* counts;  // per depth: [2 d] its queue's length, [2 d + 1] fetch
  uint32_t cap;
};

// Into the queue of `depth` (buffer depth & 1).
__device__ __forceinline__ void push_photon(const PhotonQ& q, int depth, F3 o,
                                            F3 d, F3 c, uint32_t pid,
                                            uint32_t dim, bool pred,
                                            uint32_t* err) {
  const int qi = depth & 1;
  const uint32_t k = warp_append(&q.counts[2 * depth], pred);
  if (!pred) return;
  if (k >= q.cap) {
    raise_device_error(err, kDevQueueOverflow);
    return;
  }
  q.ro[qi][k] = make_float4(o.x, o.y, o.z, __uint_as_float(pid));
  q.rd[qi][k] = make_float4(d.x, d.y, d.z, __uint_as_float(dim));
  q.coef[qi][k] = make_float4(c.x, c.y, c.z, 0.f);
}

struct Emission {
  F3 pos, dir, normal, radiance;
  float pdf_pos = 0.f, pdf_dir = 0.f;
};

// Light::SampleEmit: directional_light.cpp:60-79, env_light.cpp:105-150,
// area_light.cpp:59-70.
__device__ Emission sample_emit(const SppmArgs& a, const float* L,
                                uint64_t key, uint32_t& dim) {
  Emission e;
  const int type = (int)L[0];
  if (type == kLightArea) {
    const float x = key_float(key, dim), y = key_float(key, dim + 1),
                z = key_float(key, dim + 2);
    dim += 3;
    const AreaSample g = area_sample(L, a.s.emit_pts, x, y, z);
    float pdf_dir;
    const F3 lwi =
        cosine_hemisphere(key_float(key, dim), key_float(key, dim + 1), &pdf_dir);
    dim += 2;
    e.pos = g.pos;
    e.dir = Frame(g.ng).to_world(lwi);
    e.normal = g.ng;
    e.radiance = mk3(L[1], L[2], L[3]);
    e.pdf_pos = g.pdf;
    e.pdf_dir = pdf_dir;
  } else if (type == AJG_LIGHT_DIRECTIONAL) {
    const float u0 = key_float(key, dim), u1 = key_float(key, dim + 1);
    dim += 2;
    const F3 r2l =
        Frame(mk3(L[8], L[9], L[10]), L[11]).to_world(uniform_cone(u0, u1, L[7]));
    const float pdf_dir = uniform_cone_pdf(L[7]);
    const float radius = a.s.radius;
    float dx, dy;
    concentric(key_float(key, dim), key_float(key, dim + 1), dx, dy);
    dim += 2;
    const Frame dc(r2l);
    e.pos = a.center + (dx * dc.dx + dy * dc.dy + r2l) * radius;
    e.dir = -r2l;
    e.normal = normalize3(-r2l);
    e.radiance = mk3(L[1], L[2], L[3]);
    e.pdf_pos = 1.f / (kPi * radius * radius);
    e.pdf_dir = pdf_dir;
  } else {
    // g++ evaluates SampleContinuous's two Next1D() arguments right to
    // left: the first draw is v
    const float v = key_float(key, dim);
    float u = key_float(key, dim + 1);
    dim += 2;
    if (L[10] == 0.f) return Emission{};  // the 1x1 distribution has no mass
    float pdf = 1.f;
    constexpr float two_pi = 2.f * kPi;
    u -= L[4];
    if (u > 1.f) u -= 1.f;
    if (u < 0.f) u += 1.f;
    const float phi = u * two_pi;
    const float theta = v * kPi;
    const float st = sinf(theta);
    pdf = st != 0.f ? pdf / (2.f * kPi * kPi * st) : 0.f;
    F3 dir = mk3(-sinf(theta) * cosf(phi), cosf(theta), -sinf(theta) * sinf(phi));
    dir = -dir;
    const float radius = a.s.radius;
    float dx, dy;
    concentric(key_float(key, dim), key_float(key, dim + 1), dx, dy);
    dim += 2;
    const Frame dc(-dir);
    e.pos = a.center + (dx * dc.dx + dy * dc.dy - dir) * radius;
    e.dir = dir;
    e.normal = normalize3(dir);
    e.radiance = mk3(L[1], L[2], L[3]);  // the texel, without the scaler
    e.pdf_pos = 1.f / (kPi * radius * radius);
    e.pdf_dir = pdf;
  }
  return e;
}

// Photon i of iteration k draws from path_key(photon_seed(seed), i, k).
__device__ __forceinline__ uint64_t photon_key(const SppmArgs& a, uint32_t pid) {
  return path_key(a.pseed, a.i0 + pid % a.m, a.it0 + pid / a.m);
}

// TracerPhoton's start (sppm.cpp:105-121) and depth 1's roulette.
__global__ void __launch_bounds__(kThreads)
    k_photon_emit(SppmArgs a, PhotonQ q, uint32_t n, uint32_t* err) {
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t wb = blockIdx.x * blockDim.x + (threadIdx.x - lane); wb < n;
       wb += gridDim.x * blockDim.x) {
    const uint32_t t = wb + lane;
    bool live = false;
    F3 o = mk3(0, 0, 0), d = mk3(0, 0, 1), coef = mk3(0, 0, 0);
    const uint32_t pid = t;  // the photon's number in the wave
    uint32_t dim = 0;
    if (t < n && a.nl > 0) {
      const uint64_t key = photon_key(a, pid);
      const float u = key_float(key, dim++);
      // upper_bound with <=: the first j with u <= cdf[j]
      uint32_t j = 0;
      while (j <= a.nl && !(u <= a.cdf[j])) ++j;
      const int idx = min(max((int)j - 1, 0), (int)a.nl - 1);
      const Emission e = sample_emit(a, a.s.lights + 12 * idx, key, dim);
      if (!(black3(e.radiance) || e.pdf_dir == 0.f || e.pdf_pos == 0.f)) {
        coef = e.radiance * fabsf(dot3(e.normal, e.dir)) /
               (a.lpdf * e.pdf_pos * e.pdf_dir);
        make_ray(e.pos, e.dir, o, d);
        live = 1 <= a.pmax;
        if (live && 1 > a.pmin) {
          if (key_float(key, dim++) > a.cont)
            live = false;
          else
            coef = coef / a.cont;
        }
      }
    }
    push_photon(q, 1, o, d, coef, pid, dim, live, err);
  }
}

template <int TEST, int W>
__global__ void __launch_bounds__(128, trace_min_blocks<W>())
    k_photon_extend(DeviceScene s, const float4* __restrict__ ro,
                    const float4* __restrict__ rd,
                    const uint32_t* __restrict__ count, uint32_t* fetch_next,
                    ajg_hit* __restrict__ hits, TraceCounters* ctr,
                    uint32_t* err) {
  const uint32_t n = *count;
  uint32_t nn = 0, nt = 0, nr = 0;
  auto fetch = [&](uint32_t k, TraceScene&) {
    return make_query(xyz(ro[k]), xyz(rd[k]), kRayEps,
                      __int_as_float(0x7f800000));
  };
  auto finish = [&](uint32_t k, const Hit& h, bool) {
    ajg_hit o;
    o.t = h.t;
    o.u = h.u;
    o.v = h.v;
    o.prim = h.prim;
    hits[k] = o;
  };
  trace_persistent<TEST, false, W>(trace_scene(s), n, fetch_next, fetch,
                                   finish, nr, nn, nt, err);
  flush_counters(ctr, nr, nn, nt);
}

// Records a photon's deposit for k_deposit, among those of its iteration
// (`seg` of the wave).  Every lane of the warp calls it.
__device__ __forceinline__ void record_deposit(const Deposits& dp, uint32_t seg,
                                               bool pred, F3 pos, F3 phi, F3 wr,
                                               uint32_t* err) {
  const int lane = threadIdx.x & 31;
  const unsigned peers = __match_any_sync(kFull, pred ? seg : 0xffffffffu);
  const int leader = __ffs(peers) - 1;
  uint32_t k = 0;
  if (pred && lane == leader) k = atomicAdd(&dp.count[seg], (uint32_t)__popc(peers));
  k = __shfl_sync(kFull, k, leader) + __popc(peers & ((1u << lane) - 1u));
  if (!pred) return;
  if (k >= dp.cap) {
    raise_device_error(err, kDevQueueOverflow);
    return;
  }
  float4* r = dp.rec + 3 * ((uint64_t)seg * dp.cap + k);
  r[0] = make_float4(pos.x, pos.y, pos.z, phi.x);
  r[1] = make_float4(phi.y, phi.z, wr.x, wr.y);
  r[2] = make_float4(wr.z, 0.f, 0.f, 0.f);
}

// The entry a deposit falls into (VisiblePointSearcher::AddPhoton,
// photon_mapping.h:101-120) and its rank there; entries without visible
// points drop theirs (kEntries).
__global__ void k_deposit_enter(SppmArgs a, Grid g, Deposits dp) {
  const uint32_t n = min(*dp.count, dp.cap);
  const float side = 1.05f * *g.maxr;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += gridDim.x * blockDim.x) {
    float4* r = dp.rec + 3 * (uint64_t)k;
    int c[3];
    to_grid(xyz(r[0]), a.lo, side, c);
    uint32_t e = to_entry(c[0], c[1], c[2]), rank = 0;
    if (g.offsets[e] < min(g.offsets[e + 1], g.cap))
      rank = atomicAdd(&dp.hist[e], 1u);
    else
      e = kEntries;
    reinterpret_cast<uint32_t*>(r + 2)[1] = e;
    reinterpret_cast<uint32_t*>(r + 2)[2] = rank;
  }
}

__global__ void k_deposit_sort(Deposits dp) {
  const uint32_t n = min(*dp.count, dp.cap);
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += gridDim.x * blockDim.x) {
    const float4 r = dp.rec[3 * (uint64_t)k + 2];
    const uint32_t e = __float_as_uint(r.y);
    if (e < kEntries) dp.sorted[dp.offsets[e] + __float_as_uint(r.z)] = k;
  }
}

// The deposits: every (visible point, photon) pair of an entry, a warp per
// unit of 32 points x 32 photons.  A lane holds one visible point and its
// sums; the 32 photons sit in shared memory, read by all lanes at once for
// the distance test; the photons a lane accepts are then evaluated one a
// round, so that lanes with different photons share the rounds.  A group of
// points keeps its sums over a run of photons: one atomic add per point and
// run instead of one per pair.
// Bound by instruction issue (the distance tests and BSDF evaluations).  A
// photon walking its entry's list by itself (the form before this) left
// 2.8 of 32 threads active and added every pair atomically: 925 us a depth
// on average against 585 us for all depths of an iteration (192x192 film of
// the emitter box, radius 0.1, 100,000 photons: 118.6 -> 14.3 ms for 12
// iterations; 512x512, radius 0.01, 2 M photons over 327,682 triangles:
// 14.1 -> 10.8 ms for 4), 372 us with the points' BSDF terms prepared once.
//
// A unit costs from 32 distance tests a lane to 32 evaluations more, and dense
// entries lie together, so a warp takes kRuns short runs spread over all units
// rather than one share (which left half the warps of the box above waiting
// for the rest: 4.6 ms, 4 runs 3.1, runs of one unit -- 8 and more -- 2.8; the
// sphere, with few pairs a unit and more units, loses 10 to 20 us of 210).
//
// 8 blocks of 128 an SM (64 registers, 200 bytes of spills beside the BSDF's
// prepared terms in local memory): 4.5 ms on the box above with one share
// a warp, 6 blocks 5.6, 5 6.1, 4 without spills 7.0.  Only the Lambertian lobe
// prepared: 7.6.
constexpr uint32_t kRuns = 8;
__global__ void __launch_bounds__(kThreads, 8)
    k_deposit(SppmArgs a, SppmPixels px, Grid g, Deposits dp) {
  __shared__ float4 s_rec[kThreads / 32][32 * 3];
  const int lane = threadIdx.x & 31;
  float4* const tile = s_rec[threadIdx.x >> 5];
  const uint64_t n_warps = (uint64_t)gridDim.x * (kThreads / 32);
  const uint64_t wid = (uint64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  const unsigned long long total = dp.units[kEntries];
  // the warps' runs of `run` units, dealt out in turn
  const unsigned long long share = (total + n_warps - 1) / n_warps;
  const unsigned long long run = (share + kRuns - 1) / kRuns;
  for (unsigned long long u0 = wid * run; u0 < total; u0 += n_warps * run) {
    unsigned long long u = u0;
    const unsigned long long end = min(u0 + run, total);
    // the entry of unit u: the last with units[e] <= u, 32 pivots a round
    uint32_t e = 0;
    for (uint32_t hi = kEntries; hi - e > 1;) {
      const uint32_t step = (hi - e + 31) / 32;
      const uint32_t c = e + step * ((uint32_t)lane + 1);
      const unsigned past = __ballot_sync(kFull, c < hi && dp.units[c] <= u);
      e += step * __popc(past);
      hi = min(hi, e + step);
    }
    while (u < end) {
      // skip entries whose units end at or before u
      for (;;) {
        const uint32_t c = e + 1 + (uint32_t)lane;
        const unsigned past =
            __ballot_sync(kFull, c < kEntries && dp.units[c] <= u);
        e += __popc(past);
        if (past != kFull) break;
      }
      const uint32_t i0 = g.offsets[e], i1 = min(g.offsets[e + 1], g.cap);
      const uint32_t p0 = dp.offsets[e], p1 = dp.offsets[e + 1];
      const uint32_t tiles = (p1 - p0 + 31) / 32;
      const unsigned long long local = u - dp.units[e];
      const uint32_t group = (uint32_t)(local / tiles);
      const uint32_t t0 = (uint32_t)(local % tiles);
      const uint32_t t1 = (uint32_t)min((unsigned long long)tiles, t0 + (end - u));
      const uint32_t item = i0 + group * 32 + (uint32_t)lane;
      const bool on = item < i1;
      const float4 sp = on ? __ldg(&g.spheres[item]) : make_float4(0, 0, 0, 0);
      Bsdf f;
      F3 sum = mk3(0, 0, 0);
      uint32_t pix = 0, m_sum = 0;
      bool loaded = false;
      for (uint32_t t = t0; t < t1; ++t) {
        const uint32_t first = p0 + 32 * t;
        const int cnt = (int)min(32u, p1 - first);
        if (lane < cnt) {
          const float4* r = dp.rec + 3 * (uint64_t)dp.sorted[first + lane];
          tile[3 * lane] = r[0];
          tile[3 * lane + 1] = r[1];
          tile[3 * lane + 2] = r[2];
        }
        __syncwarp();
        unsigned near = 0;
#pragma unroll 4
        for (int j = 0; j < cnt; ++j) {
          const F3 d = xyz(sp) - xyz(tile[3 * j]);
          if (!(dot3(d, d) > sp.w)) near |= 1u << j;
        }
        if (!on) near = 0;
        if (near && !loaded) {
          pix = g.items[item];
          const VisPointD v = px.vp[pix];
          const uint32_t mat = __float_as_uint(v.pos.w);
          f.prepare(a.s.materials + 16 * mat, __ldg(&a.s.mat_lum[mat].x), xyz(v.ng),
                    xyz(v.ns), xyz(v.wr));
          loaded = true;
        }
        while (__any_sync(kFull, near != 0)) {
          if (near) {
            const int j = __ffs(near) - 1;
            near &= near - 1;
            const float px_ = tile[3 * j].w;
            const float4 q = tile[3 * j + 1];
            const float wz = tile[3 * j + 2].x;
            const F3 c = mk3(px_, q.x, q.y) * f.eval(mk3(q.z, q.w, wz));
            if (isfinite(c.x) && isfinite(c.y) && isfinite(c.z)) {
              sum = sum + c;
              ++m_sum;
            }
          }
        }
        __syncwarp();
      }
      if (m_sum) {
        atomicAdd(&px.phi[pix].x, sum.x);
        atomicAdd(&px.phi[pix].y, sum.y);
        atomicAdd(&px.phi[pix].z, sum.z);
        atomicAdd(&px.M[pix], m_sum);
      }
      u += t1 - t0;
    }
  }
}

// One depth of TracerPhoton (sppm.cpp:122-142) over the queue: the deposit
// (from depth 2 on), the BSDF sample, and the next depth's roulette.
__global__ void __launch_bounds__(kThreads)
    k_photon_shade(SppmArgs a, PhotonQ q, Deposits dp, int depth,
                   uint32_t* err) {
  const int cur = depth & 1;
  const uint32_t n = min(q.counts[2 * depth], q.cap);
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t wb = blockIdx.x * blockDim.x + (threadIdx.x - lane); wb < n;
       wb += gridDim.x * blockDim.x) {
    const uint32_t k = wb + lane;
    bool live = false, hit = false;
    F3 no = mk3(0, 0, 0), nd = mk3(0, 0, 1), coef = mk3(0, 0, 0);
    F3 pos = mk3(0, 0, 0), power = mk3(0, 0, 0), wr = mk3(0, 0, 0);
    uint32_t pid = 0, dim = 0;
    if (k < n) {
      const ajg_hit h = q.hits[k];
      const float4 o4 = q.ro[cur][k], d4 = q.rd[cur][k];
      pid = __float_as_uint(o4.w);
      dim = __float_as_uint(d4.w);
      coef = xyz(q.coef[cur][k]);
      if (h.prim >= 0) {
        const uint64_t key = photon_key(a, pid);
        const HitInfo hi =
            complete_hit(a.s, xyz(o4), xyz(d4), h.t, h.u, h.v, h.prim);
        hit = true;
        pos = hi.pos;
        power = coef;
        wr = hi.wr;
        const float* m = a.s.materials + 16 * hi.mat;
        const F3 sam = mk3(key_float(key, dim), key_float(key, dim + 1),
                           key_float(key, dim + 2));
        dim += 3;
        const BsdfSample bs = bsdf_sample(
            (int)m[0], m, __ldg(&a.s.mat_lum[hi.mat].x), hi.ng, hi.ns, hi.wr, sam);
        if (!(black3(bs.f) || bs.pdf < 0.f)) {
          coef = coef * (bs.f / bs.pdf * fabsf(dot3(hi.ng, bs.dir)));
          make_ray(eps_offset(hi, bs.dir), bs.dir, no, nd);
          live = depth + 1 <= a.pmax;
          if (live && depth + 1 > a.pmin) {
            if (key_float(key, dim++) > a.cont)
              live = false;
            else
              coef = coef / a.cont;
          }
        }
      }
    }
    if (depth > 1) record_deposit(dp, pid / a.m, hit, pos, power, wr, err);
    push_photon(q, depth + 1, no, nd, coef, pid, dim, live, err);
  }
}

// The largest radius of a pixel with a visible point (before the update).
__global__ void k_max_radius(SppmArgs a, SppmPixels px, uint32_t* bits) {
  uint32_t m = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.npix;
       i += gridDim.x * blockDim.x)
    if (has_vp(px.vp[i])) m = max(m, __float_as_uint(px.radius[i]));
  m = __reduce_max_sync(kFull, m);
  if ((threadIdx.x & 31) == 0 && m) atomicMax(bits, m);
}

// UpdatePixel (sppm.cpp:145-169) and the next iteration's cell size.
__global__ void k_update(SppmArgs a, SppmPixels px, float alpha,
                         const uint32_t* bits, float* maxr) {
  const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x;
  if (i0 == 0) {
    const float m = __uint_as_float(*bits);
    *maxr = m == 0.f ? a.init_radius : m;
  }
  for (uint32_t i = i0; i < a.npix; i += gridDim.x * blockDim.x) {
    if (!has_vp(px.vp[i])) continue;
    const uint32_t M = px.M[i];
    if (M > 0) {
      const float N = px.N[i], r = px.radius[i];
      const float new_N = N + alpha * (float)M;
      const float new_R = r * sqrtf(new_N / (N + (float)M));
      const float4 p4 = px.phi[i];
      const F3 phi = mk3(p4.x, p4.y, p4.z);
      const F3 thr = xyz(px.vp[i].thr);
      const F3 tau = (xyz(px.tau[i]) + thr * phi) * (new_R * new_R) / (r * r);
      px.tau[i] = make_float4(tau.x, tau.y, tau.z, 0.f);
      px.N[i] = new_N;
      px.radius[i] = new_R;
      px.M[i] = 0;
      px.phi[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// ComputePixelRadiance (sppm.cpp:171-180): the direct light summed over the
// iterations as the reference's per-pixel accumulator sums it, divided by
// their count, plus the photon estimate; written as one film sample.
__global__ void k_final(SppmArgs a, SppmPixels px, uint32_t iters,
                        uint64_t photon_n, float4* fsum, float4* fcomp,
                        float* rad) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.npix;
       i += gridDim.x * blockDim.x) {
    const F3 d1 = xyz(px.direct[i]);
    F3 acc = mk3(0.f, 0.f, 0.f);
    for (uint32_t k = 0; k < iters; ++k) acc = acc + d1;
    const F3 direct = acc / (float)iters;
    const float r = px.radius[i];
    const float dem = (float)photon_n * kPi * r * r;
    const F3 L = direct + xyz(px.tau[i]) / dem;
    fsum[i] = make_float4(L.x, L.y, L.z, 1.f);
    fcomp[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (rad) {
      rad[3 * (uint64_t)i] = L.x;
      rad[3 * (uint64_t)i + 1] = L.y;
      rad[3 * (uint64_t)i + 2] = L.z;
    }
  }
}

__global__ void k_fill_f(float* p, uint64_t n, float v) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    p[i] = v;
}

}  // namespace

int sppm_render(ajg_scene* sc, const ajg_camera& cam, const ajg_sppm_params& p,
                bool want_film, bool want_rad, Scratch& scratch,
                float4** out_film, float** out_rad, cudaStream_t st) {
  ajg_ctx* ctx = sc->ctx;
  const DeviceScene& s = sc->d;
  const uint64_t npix = (uint64_t)cam.width * cam.height;
  if (npix == 0 || npix > (1ull << 30))
    return fail(ctx, AJG_ERR_INVALID, "empty or too large film");
  if (p.iterations == 0) return fail(ctx, AJG_ERR_INVALID, "no iterations");
  if (p.forward_max_depth < 1 || p.forward_max_depth > 1024 ||
      p.photon_max_depth < 0 || p.photon_max_depth > 1024)
    return fail(ctx, AJG_ERR_INVALID, "depths must be in [1, 1024]");
  if (!(p.init_radius != 0.f) || !std::isfinite(p.init_radius))
    return fail(ctx, AJG_ERR_INVALID, "init_radius must be nonzero and finite");

  // the world grown by the initial radius (sppm.cpp:184-194)
  const F3 wlo = mk3(sc->world[0], sc->world[1], sc->world[2]);
  const F3 whi = mk3(sc->world[3], sc->world[4], sc->world[5]);
  float init_radius = p.init_radius;
  if (init_radius < 0) {
    const F3 d = whi - wlo;
    float q = 0.f;
    q += d.x * d.x;
    q += d.y * d.y;
    q += d.z * d.z;
    init_radius = std::sqrt(q) / 1000.f;
  }
  SppmArgs a{};
  a.s = s;
  a.lo = wlo - mk3(init_radius, init_radius, init_radius);
  a.center = (whi + wlo) / 2.f;
  a.init_radius = init_radius;
  a.pseed = photon_seed(p.seed);
  a.npix = (uint32_t)npix;
  a.pmin = p.photon_min_depth;
  a.pmax = p.photon_max_depth;
  a.cont = p.photon_cont_prob;
  // DefaultScene's selector over its lights: pdf 1/n each, the cdf as
  // Distribution::SetFunction builds it (distribution.h:37-56)
  a.nl = s.num_lights;
  if (a.nl) {
    std::vector<float> table(a.nl, 1.f);
    float sum = 0.f;
    for (float t : table) sum += t;
    const float ratio = 1.f / sum;
    for (float& t : table) t *= ratio;
    const float inv = 1.f / float(a.nl);
    a.cdf[0] = 0.f;
    for (uint32_t i = 1; i <= a.nl; ++i) a.cdf[i] = a.cdf[i - 1] + table[i - 1] * inv;
    const float fi = a.cdf[a.nl];
    for (uint32_t i = 0; i <= a.nl; ++i)
      a.cdf[i] = fi > 0.f ? a.cdf[i] / fi : float(i) / float(a.nl);
    a.lpdf = table[0];
  }

  // Photon waves (photon_plan).  As photons do not depend on the iterations
  // before, a wave holds those of several, so that small ones still fill the
  // GPU (12 iterations x 100,000 photons of the emitter box, radius 0.1: 240
  // launches of rays and shading, 4.7 ms, became 20, 1.5 ms; 10.9 -> 7.5 ms a
  // render).
  const uint64_t dep_depths = p.photon_max_depth > 1 ? p.photon_max_depth - 1 : 0;
  const uint64_t n_depths = 2 * ((uint64_t)p.photon_max_depth + 2);
  PhotonPlan plan{};
  uint64_t wave = 0, n_counts = 0;
  const uint32_t cap = (uint32_t)std::min<uint64_t>(8 * npix, 0xffffffffull);

  // the camera pass's wave arena first, then everything else
  int rc = sppm_reserve(sc, cam, p.forward_max_depth);
  if (rc) return rc;
  VisPointD* vp = nullptr;
  float4 *direct, *phi, *tau, *film, *spheres, *qro, *qrd, *qcoef, *drec;
  float4* d_out = nullptr;
  float* d_rad = nullptr;
  float *radius, *N, *maxr;
  uint32_t *M, *counts, *offsets, *cursor, *items, *bits, *qcounts, *dhist, *doff, *dsorted;
  unsigned long long* dunits;
  ajg_hit* qhits;
  EntryVal* totals;
  auto layout = [&](char* cur) {
    vp = carve<VisPointD>(cur, npix);
    direct = carve<float4>(cur, npix);
    phi = carve<float4>(cur, npix);
    tau = carve<float4>(cur, npix);
    film = carve<float4>(cur, 2 * npix);
    radius = carve<float>(cur, npix);
    N = carve<float>(cur, npix);
    maxr = carve<float>(cur, 1);
    M = carve<uint32_t>(cur, npix);
    counts = carve<uint32_t>(cur, kEntries);
    offsets = carve<uint32_t>(cur, kEntries + 1);
    cursor = carve<uint32_t>(cur, kEntries);
    items = carve<uint32_t>(cur, cap);
    spheres = carve<float4>(cur, cap);
    bits = carve<uint32_t>(cur, 1);
    qro = carve<float4>(cur, 2 * wave);
    qrd = carve<float4>(cur, 2 * wave);
    qcoef = carve<float4>(cur, 2 * wave);
    qhits = carve<ajg_hit>(cur, wave);
    qcounts = carve<uint32_t>(cur, n_counts);
    dhist = carve<uint32_t>(cur, kEntries);
    drec = carve<float4>(cur, 3 * plan.records * plan.group);
    doff = carve<uint32_t>(cur, kEntries + 1);
    dunits = carve<unsigned long long>(cur, kEntries + 1);
    dsorted = carve<uint32_t>(cur, plan.records);
    totals = carve<EntryVal>(cur, kEntryBlocks);
    if (want_film) d_out = carve<float4>(cur, npix);
    if (want_rad) d_rad = carve<float>(cur, 3 * npix);
    return cur;
  };
  for (int tries = 0;; ++tries) {
    plan = photon_plan(p.photons_per_iteration, p.iterations, p.photon_max_depth,
                       ctx->wave_paths, tries);
    wave = plan.chunk * plan.group;  // photons
    // zeroed per wave: the depths' queue counters and the iterations' deposit
    // counts
    n_counts = n_depths + plan.group;
    if (scratch.take(ctx, (uint64_t)(uintptr_t)layout(nullptr), st) == cudaSuccess)
      break;
    if (tries > 0 && plan.chunk == 1)
      return fail(ctx, AJG_ERR_OOM, "device allocation failed (SPPM buffers)");
  }
  const uint64_t chunk = plan.chunk, group = plan.group;
  layout(scratch.p);
  *out_film = d_out;
  *out_rad = d_rad;

  rc = sppm_camera_pass(sc, cam, p.forward_max_depth, p.seed, vp, direct, st);
  if (rc) return rc;

  const int gs = kSMs * 8;
  cudaMemsetAsync(phi, 0, npix * sizeof(float4), st);
  cudaMemsetAsync(tau, 0, npix * sizeof(float4), st);
  cudaMemsetAsync(N, 0, npix * sizeof(float), st);
  cudaMemsetAsync(M, 0, npix * sizeof(uint32_t), st);
  k_fill_f<<<grid_for(npix, 256, gs), 256, 0, st>>>(radius, npix, init_radius);
  k_fill_f<<<1, 32, 0, st>>>(maxr, 1, init_radius);
  const SppmPixels px{vp, direct, radius, N, M, phi, tau};
  const Grid g{counts, offsets, cursor, items, spheres, cap, maxr};
  PhotonQ q{};
  q.ro[0] = qro;
  q.ro[1] = qro + wave;
  q.rd[0] = qrd;
  q.rd[1] = qrd + wave;
  q.coef[0] = qcoef;
  q.coef[1] = qcoef + wave;
  q.hits = qhits;
  q.counts = qcounts;
  q.cap = (uint32_t)wave;
  Deposits dp{};
  dp.rec = drec;
  dp.count = qcounts + n_depths;
  dp.hist = dhist;
  dp.offsets = doff;
  dp.units = dunits;
  dp.sorted = dsorted;
  dp.cap = (uint32_t)plan.records;
  const int gd = resident_grid((const void*)k_deposit, kThreads);
  // Joins the recorded deposits of an iteration with its grid.
  auto join = [&](const Deposits& d) {
    const int gr = grid_for(plan.records, 256, gs);
    cudaMemsetAsync(d.hist, 0, kEntries * sizeof(uint32_t), st);
    k_deposit_enter<<<gr, 256, 0, st>>>(a, g, d);
    k_entry_totals<true><<<kEntryBlocks, kEntryThreads, 0, st>>>(g, d, totals);
    k_entry_scan<true><<<kEntryBlocks, kEntryThreads, 0, st>>>(g, d, totals);
    k_deposit_sort<<<gr, 256, 0, st>>>(d);
    k_deposit<<<gd, kThreads, 0, st>>>(a, px, g, d);
  };
  // Traces photons [i0, i0 + m) of `iters` iterations from it0 on.
  auto trace = [&](uint32_t it0, uint32_t iters, uint64_t i0) {
    a.it0 = it0;
    a.i0 = (uint32_t)i0;
    a.m = (uint32_t)std::min<uint64_t>(chunk, p.photons_per_iteration - i0);
    const uint32_t n = a.m * iters;
    cudaMemsetAsync(q.counts, 0, n_counts * sizeof(uint32_t), st);
    k_photon_emit<<<grid_for(n, kThreads, gs), kThreads, 0, st>>>(a, q, n,
                                                                  ctx->d_error);
    for (int depth = 1; depth <= p.photon_max_depth; ++depth) {
      const int cur = depth & 1;
      // photon rays keep the wide tree: over the binary layout the
      // photon pass measured 8% slower (long rays from the lights)
      dispatch_trace(s.tri_test, s.width, [&](auto T, auto Wd) {
        constexpr int TT = decltype(T)::value, WW = decltype(Wd)::value;
        const int gr = trace_grid((const void*)k_photon_extend<TT, WW>, 128);
        k_photon_extend<TT, WW><<<gr, 128, 0, st>>>(
            s, q.ro[cur], q.rd[cur], &q.counts[2 * depth],
            &q.counts[2 * depth + 1], q.hits, &ctx->d_counters[0], ctx->d_error);
      });
      k_photon_shade<<<grid_for(n, kThreads, gs), kThreads, 0, st>>>(
          a, q, dp, depth, ctx->d_error);
      // the record buffer may be full, and photons of a depth to come live
      if (depth > 1 && depth < p.photon_max_depth && (depth - 1) % plan.depths == 0) {
        join(dp);
        cudaMemsetAsync(dp.count, 0, sizeof(uint32_t), st);
      }
    }
    ctx->paths_total += n;
  };
  for (uint32_t it = 0; it < p.iterations; ++it) {
    cudaMemsetAsync(counts, 0, kEntries * sizeof(uint32_t), st);
    k_grid_count<<<grid_for(npix, 256, gs), 256, 0, st>>>(a, px, g, ctx->d_error);
    k_entry_totals<false><<<kEntryBlocks, kEntryThreads, 0, st>>>(g, dp, totals);
    k_entry_scan<false><<<kEntryBlocks, kEntryThreads, 0, st>>>(g, dp, totals);
    k_grid_fill<<<grid_for(npix, 256, gs), 256, 0, st>>>(a, px, g, ctx->d_error);
    const uint32_t j = it % (uint32_t)group;  // of its wave
    for (uint64_t i0 = 0; i0 < p.photons_per_iteration; i0 += chunk) {
      if (j == 0)
        trace(it, std::min<uint32_t>((uint32_t)group, p.iterations - it), i0);
      if (!dep_depths) continue;
      Deposits own = dp;
      own.rec += 3 * plan.records * j;
      own.count += j;
      join(own);
    }
    cudaMemsetAsync(bits, 0, sizeof(uint32_t), st);
    k_max_radius<<<grid_for(npix, 256, gs), 256, 0, st>>>(a, px, bits);
    k_update<<<grid_for(npix, 256, gs), 256, 0, st>>>(a, px, p.update_alpha,
                                                      bits, maxr);
  }
  const uint64_t photon_n =
      (uint64_t)p.iterations * (uint64_t)p.photons_per_iteration;
  k_final<<<grid_for(npix, 256, gs), 256, 0, st>>>(
      a, px, p.iterations, photon_n, film, film + npix, d_rad);
  if (d_out)
    enqueue_resolve(film, film + npix, nullptr, cam.width, cam.height,
                    true, true, d_out, st);
  const cudaError_t le = cudaGetLastError();
  if (le != cudaSuccess) return fail(ctx, AJG_ERR_CUDA, cudaGetErrorString(le));
  return AJG_OK;
}

}  // namespace ajg
