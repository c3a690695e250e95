// Wavefront PT-MIS integrator: PathTracing::TraceMIS / Trace
// (core/renderer/pt.cpp:98-311) split into per-bounce kernels over SoA
// queues, driven by TiledIntegrator::Render's sample loop (pt.cpp:40-73).
//
// A single-job wave holds S samples of a range of pixels (path p -> pixel
// pix0 + p / S, sample s0 + p % S).  A multi-job wave holds chunks of many
// jobs (each its own scene, camera, film and parameters; see Chunk); every
// kernel exists in both forms (template flag MJ), and the multi-job form
// reads the per-path job, scene and sampler key from the wave's tables.
// Per bounce:
//   trace_closest(queue) -> shade (NEE candidates, MIS-BSDF escape ray,
//   continuation, Russian roulette for the next bounce) -> trace_any(shadow
//   queue) -> accumulate (the direct-lighting sum in the reference's order)
// Queues are compacted with warp-ballot appends; every kernel is a
// grid-stride loop that reads its queue length from device memory, so a wave
// needs no host synchronisation and a multi-job wave is one captured graph.
// After the last bounce each pixel adds its S samples to a Kahan-compensated
// float32 film (or a float64 one), and a resolve pass applies the
// reference's 2x2 box footprint.
//
// Sampler dimensions per path (the reference's draw order, pt.cpp:58-61,
// 107-108, 203-216, helper.h, directional_light.cpp:46, env_light.cpp:71):
//   0,1 pixel jitter; 2,3 lens; then per bounce b:
//   [Russian roulette if b > min_bounces]
//   2 per light in scene order (directional: cone u, v; env: v then u --
//     g++ evaluates SampleContinuous's two Next1D() arguments right to left),
//   3 for the MIS BSDF sample, 3 for the continuation sample.
#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

#include "shade.cuh"
#include "trace.cuh"

namespace ajg {
namespace {

#ifndef AJG_SHADE_THREADS
#define AJG_SHADE_THREADS 256
#endif
constexpr int kShadeThreads = AJG_SHADE_THREADS;
constexpr int kClassifyThreads = 256;
// Queue appends of the shading kernels: a block at a time (block_append,
// block-uniform loops), or with AJG_BLOCK_APPEND=0 a warp at a time.
__device__ __forceinline__ uint32_t shade_append(uint32_t* counter,
                                                 bool pred) {
  if constexpr (AJG_BLOCK_APPEND)
    return block_append<1, kShadeThreads / 32>(counter, pred ? 0 : -1);
  else
    return warp_append(counter, pred);
}
#ifndef AJG_SHADE_MIN_BLOCKS
// blocks per SM the shading kernels are compiled for: 512 threads, up to
// 128 registers, no spills (1024 threads: 64)
#define AJG_SHADE_MIN_BLOCKS (512 / AJG_SHADE_THREADS)
#endif
#ifndef AJG_SHADE_GRID
#define AJG_SHADE_GRID 256  // single-job shading grid: blocks per SM
#endif
#ifndef AJG_MJ_SHADE_GRID
#define AJG_MJ_SHADE_GRID 64  // multi-job shading grid: blocks per SM (8 for
                              // the rarer other materials).  16 batched jobs: Lambertian
                              // 8.15 -> 7.84 ms, Disney 7.20 -> 6.80 against 8
#endif
#ifndef AJG_SHADE_MIN_BLOCKS_DIFFUSE
// the Lambertian kernels: 1024 threads, 64 registers, no spills
#define AJG_SHADE_MIN_BLOCKS_DIFFUSE (1024 / AJG_SHADE_THREADS)
#endif
template <int MAT>
constexpr int shade_min_blocks() {
  return MAT == AJG_MAT_DIFFUSE ? AJG_SHADE_MIN_BLOCKS_DIFFUSE
                                : AJG_SHADE_MIN_BLOCKS;
}
constexpr int kMaxLights = 15;
constexpr unsigned kFull = 0xffffffffu;

struct WaveArgs {
  DeviceScene s;
  ajg_camera cam;
  JobParams j;
  uint32_t pix0, S, s0, n_paths;
  VisPointD* vp;  // SPPM camera pass: the visible points (else null)
};

// Where a kernel finds the job and the scene of a path: the kernel
// arguments (single job) or the wave tables (multi-job).
template <bool MJ>
struct Src;
template <>
struct Src<false> {
  static __device__ __forceinline__ const JobParams& job(const WaveArgs& a,
                                                         const MJTables&,
                                                         uint32_t) {
    return a.j;
  }
  static __device__ __forceinline__ const DeviceScene& scene(
      const WaveArgs& a, const MJTables&, uint32_t) {
    return a.s;
  }
};
template <>
struct Src<true> {
  static __device__ __forceinline__ const JobParams& job(const WaveArgs&,
                                                         const MJTables& t,
                                                         uint32_t jid) {
    return t.jobs[jid].j;
  }
  static __device__ __forceinline__ const DeviceScene& scene(
      const WaveArgs&, const MJTables& t, uint32_t jid) {
    return t.scenes[mj_scene(t, t.jobs[jid].scene)];
  }
};

__device__ __forceinline__ int dim_base(const JobParams& J, int b) {
  const int rr = b - J.min_b - 1;
  return 4 + b * J.nd + (rr > 0 ? rr : 0);
}

__device__ __forceinline__ void path_id(const WaveArgs& a, uint32_t p,
                                        uint32_t& pixel, uint32_t& sample) {
  pixel = a.pix0 + p / a.S;
  sample = a.s0 + p % a.S;
}

// Last index c in [0, n) with off[c] <= v (off ascending, off[0] == 0).
__device__ __forceinline__ uint32_t find_le(const uint32_t* off, uint32_t n,
                                            uint32_t v) {
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (off[mid] <= v)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// The camera sample of one path (pt.cpp:58-61) and the roulette before
// bounce 0.
__device__ __forceinline__ void raygen_path(const ajg_camera& cam,
                                            const JobParams& J, uint64_t key,
                                            int x, int y, F3& ro, F3& rd,
                                            F3& T, bool& alive) {
  const float u = x + key_float(key, 0);
  const float v = y + key_float(key, 1);
  const float l0 = key_float(key, 2), l1 = key_float(key, 3);
  camera_ray(cam, u, v, l0, l1, ro, rd);
  T = mk3(1.f, 1.f, 1.f);
  alive = J.max_b > 0;
  if (alive && 0 > J.min_b) {  // roulette before bounce 0
    if (key_float(key, dim_base(J, 0)) > J.cont) alive = false;
    T = T / J.cont;
  }
}

template <bool MJ>
__global__ void __launch_bounds__(kShadeThreads)
    k_raygen(WaveArgs a, MJTables t, WaveBufs w) {
  __shared__ uint32_t s_off[MJ ? kMaxWaveChunks : 1];
  uint32_t n_paths = a.n_paths, n_chunks = 0;
  const bool all_alive =
      AJG_BLOCK_APPEND && !MJ && a.j.max_b > 0 && !(0 > a.j.min_b);
  if (all_alive && blockIdx.x == 0 && threadIdx.x == 0)
    atomicAdd(&w.counts[0], n_paths);
  if constexpr (MJ) {
    if (!mj_wave_ok(t)) return;  // uniform: every thread reads one header
    n_paths = t.hdr->n_paths;
    n_chunks = t.hdr->n_chunks;
    for (uint32_t c = threadIdx.x; c < n_chunks; c += blockDim.x)
      s_off[c] = t.chunks[c].path_off;
    __syncthreads();
  }
  // block-uniform iterations (block_append synchronises the block)
  for (uint32_t pb = blockIdx.x * blockDim.x; pb < n_paths;
       pb += gridDim.x * blockDim.x) {
    const uint32_t p = pb + threadIdx.x;
    F3 ro = mk3(0, 0, 0), rd = mk3(0, 0, 1), T = mk3(1, 1, 1);
    bool alive = false;
    uint32_t sid = 0;
    if (p >= n_paths) {
      // past the wave: only the queue append below
    } else if constexpr (MJ) {
      const Chunk C = t.chunks[find_le(s_off, n_chunks, p)];
      const uint32_t q = p - C.path_off;
      const uint32_t i = C.pix0 + q / C.S;
      const uint32_t sample = C.s0 + q % C.S;
      const uint32_t jid = mj_job(t, C.job);
      const JobRec& R = t.jobs[jid];
      const int x = (int)(R.j.x0 + i % R.j.win_w);
      const int y = (int)(R.j.y0 + i / R.j.win_w);
      const uint64_t key =
          path_key(R.j.seed, (uint32_t)y * R.j.film_w + (uint32_t)x, sample);
      w.pjob[p] = jid;
      w.pkey[p] = key;
      sid = mj_scene(t, R.scene);
      raygen_path(R.cam, R.j, key, x, y, ro, rd, T, alive);
    } else {
      uint32_t pixel, sample;
      path_id(a, p, pixel, sample);
      const uint64_t key = path_key(a.j.seed, pixel, sample);
      const int x = (int)(pixel % a.cam.width), y = (int)(pixel / a.cam.width);
      raygen_path(a.cam, a.j, key, x, y, ro, rd, T, alive);
    }
    if (p < n_paths) {
      w.thr[p] = make_float4(T.x, T.y, T.z, 0.f);
      w.rad[p] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // a single job whose paths all start (no roulette before bounce 0) is
    // queued in path order without atomics (the count is added once above)
    const uint32_t k = all_alive ? p : shade_append(&w.counts[0], alive);
    if (alive) {
      w.qpath[0][k] = p;
      w.ro[0][k] = make_float4(ro.x, ro.y, ro.z, __uint_as_float(sid));
      w.rd[0][k] = make_float4(rd.x, rd.y, rd.z, 0.f);
    }
  }
}

// A light term: term_f holds throughput x f, counted once its ray is found
// unoccluded (kTermSeen, written by the traversal).  An occluded one adds
// throughput x 0: nothing, except in the rare path whose throughput is not
// finite (kTermUnseenBad; its throughput is then in thr_shade).
constexpr uint8_t kTermUnseen = 0, kTermSeen = 1, kTermUnseenBad = 2;
__device__ __forceinline__ uint8_t term_unseen(F3 T) {
  return isfinite(T.x) && isfinite(T.y) && isfinite(T.z) ? kTermUnseen
                                                         : kTermUnseenBad;
}
// In place of its path in a queue slot whose ray missed (set by k_classify).
constexpr uint32_t kMissed = 0x80000000u;

// Files every queue slot under its hit's shading class (delta types,
// Lambertian, Disney, the others), so that shading runs in class-specialised
// kernels, and ends the escaped paths: the environment counts only for camera
// rays (pt.cpp:114-121), or on every bounce without MIS (pt.cpp:245-249).
// (Beside the accumulation of the bounce before: no path of it is touched by
// both, as with MIS only camera rays add here.)
template <bool MJ>
__global__ void __launch_bounds__(kClassifyThreads)
    k_classify(WaveArgs a, MJTables t, WaveBufs w, int b, int cur,
               uint32_t list_cap) {
  const uint32_t n = w.counts[0];
  const uint32_t stride = gridDim.x * blockDim.x;
  // block-uniform iterations: block_append synchronises the block
  for (uint32_t bb = blockIdx.x * blockDim.x; bb < n; bb += stride) {
    const uint32_t k = bb + threadIdx.x;
    int cls = -1;
    if (k < n) {
      const int prim = w.hits[k].prim;
      if (prim >= 0) {
        const float4* shade = a.s.shade;
        const float* materials = a.s.materials;
        if constexpr (MJ) {
          const DeviceScene& sc =
              t.scenes[mj_scene(t, __float_as_uint(w.ro[cur][k].w))];
          shade = sc.shade;
          materials = sc.materials;
        }
        const uint32_t mat =
            __float_as_uint(__ldg(&shade[prim].w)) & 0xffffffu;
        const int type = (int)__ldg(materials + 16 * mat);
        cls = type == AJG_MAT_DIFFUSE  ? 1
              : type == AJG_MAT_DISNEY ? 2
                                       : ((kDeltaTypes >> type) & 1u ? 0 : 3);
      } else {
        if (MJ || ((b == 0 || !a.j.use_mis) && a.s.env >= 0)) {
          const uint32_t p = w.qpath[cur][k];
          const uint32_t jid = MJ ? mj_job(t, w.pjob[p]) : 0u;
          const JobParams& J = Src<MJ>::job(a, t, jid);
          if ((b == 0 || !J.use_mis) && Src<MJ>::scene(a, t, jid).env >= 0) {
            float4 L = w.rad[p];
            L.x += J.env_rgb.x;
            L.y += J.env_rgb.y;
            L.z += J.env_rgb.z;
            w.rad[p] = L;
          }
        }
        w.qpath[cur][k] = kMissed;
      }
    }
#if AJG_BLOCK_APPEND
    const uint32_t j = block_append<4, kClassifyThreads / 32>(&w.counts[4], cls);
    if (cls >= 0) w.lists[(uint64_t)cls * list_cap + j] = k;
#else
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint32_t j = warp_append(&w.counts[4 + c], cls == c);
      if (cls == c) w.lists[(uint64_t)c * list_cap + j] = k;
    }
#endif
  }
}

// The MIS BSDF term from its closest hit (helper.h:223-264): an escaped ray
// sees the environment, one that hits the lit side of an emitter its
// radiance, weighted against AreaLight::Pdf; anything else adds nothing.
template <bool MJ>
__global__ void __launch_bounds__(kShadeThreads)
    k_bsdf_emit(WaveArgs a, MJTables t, WaveBufs w, uint32_t NT, uint32_t cap,
                uint32_t n_max, const float* __restrict__ t_hit,
                const int32_t* __restrict__ prim_hit) {
  const uint32_t n = min(w.counts[9], n_max);
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += gridDim.x * blockDim.x) {
    const uint32_t i = cap - 1 - k;
    const float4 o4 = w.sq_o[i], d4 = w.sq_d[i];
    const uint32_t slot = __float_as_uint(d4.w);
    const uint32_t p = slot / NT;
    const uint32_t jid = MJ ? mj_job(t, w.pjob[p]) : 0u;
    const JobParams& J = Src<MJ>::job(a, t, jid);
    const DeviceScene& s = Src<MJ>::scene(a, t, jid);
    const F3 o = xyz(o4), d = xyz(d4);
    const bool delta = signbit(o4.w);  // see k_shade
    const float pdf = fabsf(o4.w);
    const float4 fs = w.term_f[slot];
    const F3 bf = xyz(fs);
    const float cosv = fs.w;
    const int prim = prim_hit[k];
    F3 fo = mk3(0.f, 0.f, 0.f);
    bool vis = false;
    if (prim < 0) {
      const F3 rad = mk3(J.env_rgb.x, J.env_rgb.y, J.env_rgb.z);
      if (s.env >= 0 && !black3(rad)) {
        const F3 fv = rad * bf * cosv;
        if (delta) {
          fo = mk3(0, 0, 0) + fv / pdf;
        } else {
          const float lp = env_pdf(J.env_mass != 0, d);
          fo = mk3(0, 0, 0) + fv / pdf * power_heuristic(pdf, lp);
        }
        vis = true;
      }
    } else {
      const int li = __ldg(s.tri_emit + prim);
      if (li >= 0) {
        F3 pos, ng;
        emitter_hit(s, o, d, t_hit[k], prim, pos, ng);
        const float* L = s.lights + 12 * li;
        const F3 le =
            dot3(ng, -d) > 0 ? mk3(L[1], L[2], L[3]) : mk3(0.f, 0.f, 0.f);
        if (!black3(le)) {
          const F3 fv = le * bf * cosv;
          if (delta) {
            fo = fv / pdf;
          } else {
            const float lp = area_pdf(L[9], o, pos, ng);
            fo = fv / pdf * power_heuristic(pdf, lp);
          }
          vis = true;
        }
      }
    }
    const F3 T = xyz(w.thr_shade[p]);
    fo = T * fo;
    w.term_f[slot] = make_float4(fo.x, fo.y, fo.z, 0.f);
    w.term_vis[slot] = vis ? kTermSeen : term_unseen(T);
  }
}

// A shadow ray: to the shadow queue, or -- `top`, the coherent rays of bounce
// 0 in waves without emitters -- to the coherent queue, whose entry k sits
// at cap - 1 - k of the same storage (the two cannot meet: a path appends at
// most NT entries to them together).  Without `split`, `top` is uniform over
// the block (one append); with `split` (uniform) each lane picks its queue
// (an append to each).
template <bool MJ>
__device__ __forceinline__ void emit_shadow(const WaveBufs& w, F3 o, F3 d,
                                            float tmax, uint32_t slot,
                                            uint32_t sid, bool pred,
                                            uint32_t cap, uint32_t* err,
                                            bool top = false,
                                            bool split = false) {
  uint32_t k;
  if (split) {
    const uint32_t kb = shade_append(&w.counts[2], pred && !top);
    const uint32_t kt = shade_append(&w.counts[11], pred && top);
    k = top ? kt : kb;
  } else {
    k = shade_append(&w.counts[top ? 11 : 2], pred);
  }
  if (!pred) return;
  if (k >= cap) {
    raise_device_error(err, kDevQueueOverflow);
    return;
  }
  const uint32_t i = top ? cap - 1 - k : k;
  w.sq_o[i] = make_float4(o.x, o.y, o.z, tmax);
  w.sq_d[i] = make_float4(d.x, d.y, d.z, __uint_as_float(slot));
  if constexpr (MJ) w.sq_scene[i] = (uint16_t)sid;
}

// The closest-hit queue of MIS BSDF rays in scenes with emitters: entry k
// sits at cap - 1 - k of the shadow queue's storage.  A path appends at most
// NT entries to the two queues together (its lights' shadow rays and one
// BSDF ray) and cap = P * NT, so the queues cannot meet.
template <bool MJ>
__device__ __forceinline__ void emit_closest(const WaveBufs& w, F3 o, F3 d,
                                             float pdf, uint32_t slot,
                                             uint32_t sid, bool pred,
                                             uint32_t cap, uint32_t* err) {
  const uint32_t k = shade_append(&w.counts[9], pred);
  if (!pred) return;
  if (k >= cap) {
    raise_device_error(err, kDevQueueOverflow);
    return;
  }
  const uint32_t i = cap - 1 - k;
  w.sq_o[i] = make_float4(o.x, o.y, o.z, pdf);
  w.sq_d[i] = make_float4(d.x, d.y, d.z, __uint_as_float(slot));
  if constexpr (MJ) w.sq_scene[i] = (uint16_t)sid;
}

// Shading of the hits on one material type: NEE to every light
// (helper.h:100-133), the MIS BSDF sample (helper.h:209-265), the
// continuation sample (pt.cpp:215-223) and the next bounce's roulette.
template <int MAT, bool MJ>
__global__ void __launch_bounds__(kShadeThreads, shade_min_blocks<MAT>())
    k_shade(WaveArgs a, MJTables t, WaveBufs w, int b, int cur,
            const uint32_t* __restrict__ list,
            const uint32_t* __restrict__ list_count, uint32_t NT,
            uint32_t shadow_cap, uint32_t* err, uint32_t coh = 0) {
  // coh: bit l set -- light term l's shadow rays go to the coherent queue
  // (bit 31: the MIS BSDF term's); multi-job waves: nonzero -- every lane's
  // directional-light rays go there.  Waves without emitters only.
  const uint32_t n = *list_count;
  const int nxt = cur ^ 1;
  // warp-uniform loop (block-uniform for a single job): every lane of a
  // warp (thread of the block) runs the same iterations, so the queue
  // appends see all of them
  constexpr bool kBlockLoop = AJG_BLOCK_APPEND;
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t first = kBlockLoop ? 0u : threadIdx.x - lane;
  for (uint32_t wb = blockIdx.x * blockDim.x + first; wb < n; wb += stride) {
    const uint32_t j = wb + (kBlockLoop ? threadIdx.x : lane);
    const bool hit = j < n;
    uint32_t p = 0, k = 0, jid = 0;
    if (hit) {
      k = list[j];
      p = w.qpath[cur][k];
      if constexpr (MJ) jid = mj_job(t, w.pjob[p]);
    }
    const JobParams& J = Src<MJ>::job(a, t, jid);
    const DeviceScene& s = Src<MJ>::scene(a, t, jid);
    const uint32_t sid = MJ ? mj_scene(t, t.jobs[jid].scene) : 0u;
    HitInfo hi;
    BsdfT<MAT> f;
    F3 T = mk3(0, 0, 0);
    uint64_t key = 0;
    int emitter = -1;
    if (hit) {
      const ajg_hit h = w.hits[k];
      if (s.tri_emit) emitter = __ldg(s.tri_emit + h.prim);
      const F3 ro = xyz(w.ro[cur][k]), rd = xyz(w.rd[cur][k]);
      if constexpr (MJ) {
        key = w.pkey[p];
      } else {
        uint32_t pixel, sample;
        path_id(a, p, pixel, sample);
        key = path_key(a.j.seed, pixel, sample);
      }
      T = xyz(w.thr[p]);
      hi = complete_hit(s, ro, rd, h.t, h.u, h.v, h.prim);
      f.prepare(s.materials + 16 * hi.mat, __ldg(&s.mat_lum[hi.mat].x), hi.ng,
                hi.ns, hi.wr);
      if (s.tri_emit || term_unseen(T) != kTermUnseen)
        w.thr_shade[p] = make_float4(T.x, T.y, T.z, 0.f);
      // an emitter seen by a camera ray, or by any ray without MIS
      // (pt.cpp:185-190, 282-286; AreaLight::Radiance, area_light.cpp:30-34)
      if (emitter >= 0 && (b == 0 || !J.use_mis)) {
        const float* L = s.lights + 12 * emitter;
        const F3 le = dot3(hi.ng, hi.wr) > 0 ? mk3(L[1], L[2], L[3])
                                               : mk3(0.f, 0.f, 0.f);
        const F3 c = T * le;
        float4 R = w.rad[p];
        R.x += c.x;
        R.y += c.y;
        R.z += c.z;
        w.rad[p] = R;
      }
    }
    int dim = dim_base(J, b) + (b > J.min_b ? 1 : 0);
    // lanes of a multi-job block differ in lights and MIS: loop over the
    // block's maximum with the lanes past their own count idle
    const int nl = (int)s.num_lights;
    const bool mis = hit && J.use_mis;
    int nl_loop = nl;
    bool any_mis = J.use_mis != 0;
    if constexpr (MJ && kBlockLoop) {
      nl_loop = (int)block_max<kShadeThreads / 32>(mis ? (unsigned)nl : 0u);
      any_mis = __syncthreads_or(mis) != 0;
    } else if constexpr (MJ) {
      nl_loop = (int)__reduce_max_sync(kFull, mis ? (unsigned)nl : 0u);
      any_mis = __any_sync(kFull, mis);
    }

    // SPPM's camera pass ends a path at its first diffuse surface or its
    // last bounce with a visible point (sppm.cpp:77-92)
    bool vp_here = false;
    if constexpr (!MJ) {
      if (a.vp && hit) {
        bool diffuse;
        if (MAT == AJG_MAT_DIFFUSE)
          diffuse = true;
        else if (MAT == AJG_MAT_DISNEY)
          diffuse = f.m[5] < 1.f;  // DisneyBSDF: metallic < 1
        else
          diffuse = (int)f.m[0] == AJG_MAT_PLASTIC;
        vp_here = diffuse || b == J.max_b - 1;
        if (vp_here && isfinite(T.x) && isfinite(T.y) && isfinite(T.z)) {
          VisPointD v;
          v.pos = make_float4(hi.pos.x, hi.pos.y, hi.pos.z,
                              __uint_as_float(hi.mat));
          v.wr = make_float4(hi.wr.x, hi.wr.y, hi.wr.z, 0.f);
          v.thr = make_float4(T.x, T.y, T.z, 0.f);
          v.ng = make_float4(hi.ng.x, hi.ng.y, hi.ng.z, 0.f);
          v.ns = make_float4(hi.ns.x, hi.ns.y, hi.ns.z, 0.f);
          a.vp[a.pix0 + p / a.S] = v;
        }
      }
    }

    // The hit's directions, a round each: a sample per light, the MIS BSDF
    // sample, the continuation.  A round draws a direction, evaluates the BSDF
    // there and appends its ray.  Lanes without MIS only continue.
    // (What no hit changes of a light comes in its record, and the lights share
    // ns1: Lambertian shading of 256x256x64 paths in a box 1.72 -> 1.66 ms, of
    // 16 batched jobs 7.94 -> 7.55.)
    F3 ns1 = mk3(0, 0, 0);
    if (hit) ns1 = normalize3(hi.ns);
    DisneyB::Stretched stretched;
    if constexpr (BsdfT<MAT>::kDisney)
      if (hit) stretched = f.b.stretched();
    // The Lambertian kernels re-read the throughput (L1) where they need it:
    // held over the rounds it would spill.
    auto thr = [&]() __attribute__((always_inline)) {
      return MAT == AJG_MAT_DIFFUSE ? xyz(w.thr[p]) : T;
    };
    enum Kind { kLight, kMisBsdf, kContinue };
    auto round = [&](Kind kind, int t_) __attribute__((always_inline)) {
      const bool is_light = kind == kLight, is_mis = kind == kMisBsdf;
      if constexpr (MAT == kMatDelta) {
        if (is_light) {  // f is 0: the light's draws are passed over
          if (MJ ? (mis && t_ < nl) : hit) {
            w.term_vis[p * NT + t_] = term_unseen(T);
            dim += (int)s.lights[12 * t_] == kLightArea ? 3 : 2;
          }
          return;
        }
      }
      bool on, lit = false;  // lit: `wl` is a direction to evaluate
      F3 wl = mk3(0, 0, 1), lrad = mk3(0, 0, 0);
      float lpdf = 0.f, len = 0.f;
      int type = -1, draws = 3;
      const float* L = s.lights;
      BsdfSample bs = invalid_sample();
      if (is_light) {
        on = MJ ? (mis && t_ < nl) : hit;
        L = s.lights + 12 * (MJ ? (t_ < nl ? t_ : 0) : t_);
        draws = 2;
        if (on) {
          F3 lpos;
          type = (int)L[0];
          bool ok = true;
          if (type == kLightArea) {
            // AreaLight::Sample (area_light.cpp:36-57): three draws
            draws = 3;
            const AreaSample g =
                area_sample(L, s.emit_pts, key_float(key, dim),
                            key_float(key, dim + 1), key_float(key, dim + 2));
            lrad = mk3(L[1], L[2], L[3]);
            lpos = g.pos;
            lpdf = 0.f;
            if (dot3(g.ng, hi.pos - g.pos) <= 0) {
              ok = false;
            } else {
              const F3 i2r = hi.pos - g.pos;
              const float dist2 = dot3(i2r, i2r);
              lpdf = g.pdf * dist2 / fabsf(dot3(g.ng, i2r));
            }
          } else if (type == AJG_LIGHT_DIRECTIONAL) {
            const float u0 = key_float(key, dim), u1 = key_float(key, dim + 1);
            const Frame fr(mk3(L[8], L[9], L[10]), L[11]);
            const F3 r2l = fr.to_world(uniform_cone(u0, u1, L[7]));
            lpdf = uniform_cone_pdf(L[7]);
            lpos = hi.pos + 2.f * s.radius * r2l;
            lrad = mk3(L[1], L[2], L[3]);
          } else {
            // g++ evaluates SampleContinuous's two Next1D() arguments right
            // to left: the first draw is v (env_light.cpp:71-72)
            const float v = key_float(key, dim);
            float u = key_float(key, dim + 1);
            lrad = mk3(L[1], L[2], L[3]);
            lpdf = 0.f;
            lpos = hi.pos;
            if (L[10] == 0.f) {  // the 1x1 distribution has no mass
              ok = false;
            } else {
              constexpr float two_pi = 2.f * kPi;
              u -= L[4];
              if (u > 1.f) u -= 1.f;
              if (u < 0.f) u += 1.f;
              const float phi = u * two_pi;
              const float theta = v * kPi;
              const float st = sinf(theta);
              lpdf = st != 0.f ? 1.f / (2.f * kPi * kPi * st) : 0.f;
              const F3 dir = mk3(-st * cosf(phi), cosf(theta), -st * sinf(phi));
              lpos = hi.pos + 2.f * s.radius * dir;
            }
          }
          if (ok && !(black3(lrad) || lpdf <= 0.f)) {
            len = len3(lpos - hi.pos) - kRayEps;
            if (!(len < kRayEps)) {
              wl = normalize3(lpos - hi.pos);
              lit = true;
            }
          }
        }
      } else {
        on = is_mis ? (MJ ? mis : hit) : hit && !vp_here && b + 1 < J.max_b;
        if (on) {
          const F3 sam = mk3(key_float(key, dim), key_float(key, dim + 1),
                             key_float(key, dim + 2));
          if constexpr (BsdfT<MAT>::kDisney) {
            const F3 lwi = f.b.sample_dir(sam, stretched);
            if (!(lwi.z <= 0.0f)) {
              wl = f.b.frame().to_world(lwi);
              lit = true;
            }
          } else {
            bs = f.sample(sam);
          }
        }
      }
      F3 bf = mk3(0, 0, 0);
      float bp = 0.f;
      if (lit) f.eval_pdf(wl, bf, bp, !is_light);
      if constexpr (BsdfT<MAT>::kDisney) {
        if (!is_light && lit) {
          bs.dir = wl;
          bs.f = bf;
          bs.pdf = bp;
        }
      }

      if (kind == kContinue) {
        // the continuation sample (pt.cpp:215-223)
        bool alive = false;
        F3 nro = mk3(0, 0, 0), nrd = mk3(0, 0, 1);
        if (on) {
          if (!(black3(bs.f) || bs.pdf < 0.f)) {
            T = thr() * (bs.f * fabsf(dot3(hi.ng, bs.dir)) / bs.pdf);
            make_ray(eps_offset(hi, bs.dir), bs.dir, nro, nrd);
            alive = true;
            if (b + 1 > J.min_b) {
              if (key_float(key, dim_base(J, b + 1)) > J.cont)
                alive = false;
              else
                T = T / J.cont;
            }
          }
          if (alive) w.thr[p] = make_float4(T.x, T.y, T.z, 0.f);
        }
        // the next bounce's queue
        const uint32_t kn = shade_append(&w.counts[kCounterWords], alive);
        if (alive) {
          w.qpath[nxt][kn] = p;
          w.ro[nxt][kn] = make_float4(nro.x, nro.y, nro.z, __uint_as_float(sid));
          w.rd[nxt][kn] = make_float4(nrd.x, nrd.y, nrd.z, 0.f);
        }
        return;
      }

      // a shadow ray (or an emitter scene's closest-hit ray) of the term
      bool emit = false, closest = false;
      F3 fo = mk3(0, 0, 0), so = mk3(0, 0, 0), sd = mk3(0, 0, 1);
      float tmax = __int_as_float(0x7f800000);
      float w_o = __int_as_float(0x7f800000), cosv = 0.f;
      if (is_light) {
        if (lit && !black3(bf)) {
          // MISSampleAreaLight takes the shading normal as it is, the
          // others normalise it (helper.h:64, 91, 120)
          const F3 nn = type == kLightArea ? hi.ns : ns1;
          F3 fv;
          if (type != AJG_LIGHT_ENV)
            fv = mk3(1.f, 1.f, 1.f) * lrad * bf * fabsf(dot3(wl, nn));
          else
            fv = lrad * bf * fabsf(dot3(wl, nn));
          fo = fv / lpdf * power_heuristic(lpdf, bp);
          make_ray(hi.pos, wl, so, sd);
          tmax = 0.99f * len;
          emit = true;
        }
      } else if (on && !(black3(bs.f) || bs.pdf == 0.f)) {
        // MISSampleBsdf (helper.h:209-265).  Without emitters only the
        // environment can answer, and an any-hit escape test decides; with
        // emitters the closest hit decides, so the ray goes to the closest
        // queue with the BSDF value and |cos| parked in its term and the pdf
        // in the ray (k_bsdf_emit completes the term).
        if (s.tri_emit) {
          bs.dir = normalize3(bs.dir);
          make_ray(eps_offset(hi, bs.dir), bs.dir, so, sd);
          fo = bs.f;
          cosv = fabsf(dot3(hi.ns, sd));
          w_o = bs.delta ? -bs.pdf : bs.pdf;  // a delta sample: negated
          closest = true;
        } else if (s.env >= 0) {
          bs.dir = normalize3(bs.dir);
          make_ray(eps_offset(hi, bs.dir), bs.dir, so, sd);
          const F3 rad = mk3(J.env_rgb.x, J.env_rgb.y, J.env_rgb.z);
          if (!black3(rad)) {
            const F3 fv = rad * bs.f * fabsf(dot3(hi.ns, sd));
            // a delta sample is not weighted (helper.h:236-241)
            if (bs.delta) {
              fo = mk3(0, 0, 0) + fv / bs.pdf;
            } else {
              const float lp = env_pdf(J.env_mass != 0, sd);
              fo = mk3(0, 0, 0) +
                   fv / bs.pdf * power_heuristic(bs.pdf, lp);
            }
            emit = true;
          }
        }
      }
      const uint32_t slot = p * NT + (is_mis ? NT - 1 : (uint32_t)t_);
      if (on) {
        // (a closest-hit term is completed, and multiplied, by k_bsdf_emit)
        const F3 Th = thr();
        if (!closest) fo = Th * fo;
        w.term_f[slot] = make_float4(fo.x, fo.y, fo.z, cosv);
        w.term_vis[slot] = term_unseen(Th);
        dim += draws;
      }
      // to the packet queue: this term's rays (a single job), or a lane's
      // directional-light rays when its job's footprint allows packets
      // (multi-job lanes differ in their t-th light and their job)
      bool top;
      if (is_mis)
        top = !MJ && ((coh >> 31) & 1u);
      else
        top = MJ ? (coh != 0 && on && J.packets &&
                    (int)L[0] == AJG_LIGHT_DIRECTIONAL)
                 : (t_ < 31 && ((coh >> t_) & 1u));
      emit_shadow<MJ>(w, so, sd, tmax, slot, sid, emit, shadow_cap, err, top,
                      MJ && coh != 0 && is_light);
      // (a single job's scene without emitters never fills this queue: skip
      // its block-wide append; the condition is uniform)
      if (is_mis && (MJ || s.tri_emit))
        emit_closest<MJ>(w, so, sd, w_o, slot, sid, closest, shadow_cap, err);
    };
    if constexpr (BsdfT<MAT>::kDisney) {
      // one loop: the BSDF's sample and evaluation are at one site each, so
      // they are inlined with the hit's terms in registers and the kernel
      // fits the instruction cache.  (Three sites with out-of-line calls:
      // 9.7 ms of shading a 1024x1024x32 render of the 1.3 M-triangle
      // sphere, its terms prepared in local memory 10.7, this loop 7.6.)
      for (int t = any_mis ? 0 : nl_loop + 1; t < nl_loop + 2; ++t)
        round(t < nl_loop ? kLight : (t == nl_loop ? kMisBsdf : kContinue), t);
    } else {
      // the kinds apart: each is short and needs fewer registers (256x256x64
      // Cornell box: 1.67 ms, one loop 1.82)
      if (any_mis) {
        for (int t = 0; t < nl_loop; ++t) round(kLight, t);
        round(kMisBsdf, nl_loop);
      }
      round(kContinue, nl_loop + 1);
    }
  }
}

// direct_illum += throughput * MISSampleLight(...) for each light, then
// += throughput * MISSampleBsdf(...); pixel.value += direct (pt.cpp:200-213)
template <bool MJ>
__global__ void __launch_bounds__(kShadeThreads)
    k_accumulate(WaveArgs a, MJTables t, WaveBufs w, int cur, uint32_t NT) {
  const uint32_t n = w.counts[0];
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += gridDim.x * blockDim.x) {
    const uint32_t p = w.qpath[cur][k];
    if (p == kMissed) continue;
    int nl = (int)a.s.num_lights;
    if constexpr (MJ) {
      const JobParams& J = t.jobs[mj_job(t, w.pjob[p])].j;
      if (!J.use_mis) continue;
      nl = J.nl;
      if (nl + 1 > (int)NT) {  // the arena holds NT terms per path
        raise_device_error(t.err, kDevTableOutOfBounds);
        continue;
      }
    }
    F3 direct = mk3(0.f, 0.f, 0.f);
    for (int j = 0; j <= nl; ++j) {
      const uint32_t slot = p * NT + (j < nl ? (uint32_t)j : NT - 1);
      const uint8_t seen = w.term_vis[slot];
      if (seen == kTermSeen)
        direct = direct + xyz(w.term_f[slot]);
      else if (seen == kTermUnseenBad)
        direct = direct + xyz(w.thr_shade[p]) * mk3(0, 0, 0);
    }
    float4 L = w.rad[p];
    const F3 d1 = 1.f / 1 * direct;
    L.x += d1.x;
    L.y += d1.y;
    L.z += d1.z;
    w.rad[p] = L;
  }
}

// Adds S consecutive samples to one film pixel in sample order
// (Kahan-compensated float32, or float64).
__device__ __forceinline__ void film_pixel(const float4* __restrict__ rad,
                                           uint64_t base, uint32_t S,
                                           uint64_t pixel, float4* sum,
                                           float4* comp, double* sum64,
                                           bool drop_nonfinite) {
  if (sum64) {
    double* o = sum64 + 4 * pixel;
    double x = o[0], y = o[1], z = o[2], wsum = o[3];
    for (uint32_t j = 0; j < S; ++j) {
      const float4 L = rad[base + j];
      if (drop_nonfinite &&
          !(isfinite(L.x) && isfinite(L.y) && isfinite(L.z)))
        continue;
      x += L.x;
      y += L.y;
      z += L.z;
      wsum += 1.0;
    }
    o[0] = x;
    o[1] = y;
    o[2] = z;
    o[3] = wsum;
    return;
  }
  float4 s4 = sum[pixel], c4 = comp[pixel];
  for (uint32_t j = 0; j < S; ++j) {
    const float4 L = rad[base + j];
    if (drop_nonfinite && !(isfinite(L.x) && isfinite(L.y) && isfinite(L.z)))
      continue;
    s4.w += 1.f;
    float y, t;
    y = L.x - c4.x; t = s4.x + y; c4.x = (t - s4.x) - y; s4.x = t;
    y = L.y - c4.y; t = s4.y + y; c4.y = (t - s4.y) - y; s4.y = t;
    y = L.z - c4.z; t = s4.z + y; c4.z = (t - s4.z) - y; s4.z = t;
  }
  sum[pixel] = s4;
  comp[pixel] = c4;
}

// Each pixel of the wave adds its S samples in sample order.
template <bool MJ>
__global__ void k_film_add(WaveArgs a, MJTables t,
                           const float4* __restrict__ rad,
                           float4* __restrict__ sum, float4* __restrict__ comp,
                           double* __restrict__ sum64, uint32_t n_pix) {
  __shared__ uint32_t s_off[MJ ? kMaxWaveChunks : 1];
  uint32_t n_chunks = 0;
  if constexpr (MJ) {
    if (!mj_wave_ok(t)) return;  // uniform: every thread reads one header
    n_pix = t.hdr->n_pix;
    n_chunks = t.hdr->n_chunks;
    for (uint32_t c = threadIdx.x; c < n_chunks; c += blockDim.x)
      s_off[c] = t.chunks[c].pix_off;
    __syncthreads();
  }
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_pix;
       i += gridDim.x * blockDim.x) {
    if constexpr (MJ) {
      const Chunk C = t.chunks[find_le(s_off, n_chunks, i)];
      const JobRec& R = t.jobs[mj_job(t, C.job)];
      const uint32_t li = i - C.pix_off;
      if (C.path_off + (uint64_t)(li + 1) * C.S > t.hdr->n_paths) {
        raise_device_error(t.err, kDevTableOutOfBounds);
        continue;
      }
      film_pixel(rad, C.path_off + (uint64_t)li * C.S, C.S, C.pix0 + li,
                 R.fsum, R.fcomp, R.fsum64, R.j.drop_nonfinite != 0);
    } else {
      film_pixel(rad, (uint64_t)i * a.S, a.S, a.pix0 + i, sum, comp, sum64,
                 a.j.drop_nonfinite != 0);
    }
  }
}

// The reference's film convention (film.cpp:27-63, film.h:119-129,
// image.h:38-42): a sample at (x, y) lands on (x-1..x, y-1..y) with weight
// 1, and row/column -1 folds into 0.  Target (tx, ty) thus sums sources
// tx (twice when tx == 0) and tx + 1, likewise in y.  For a window of the
// image the fold applies only where the window starts at row/column 0, and
// sources past the window are absent.  The four terms are summed in
// double: the compensated float32 film carries more than float precision.
__global__ void k_resolve(const float4* __restrict__ sum,
                          const float4* __restrict__ comp,
                          const double* __restrict__ sum64, uint32_t W,
                          uint32_t H, int fold_x, int fold_y,
                          float4* __restrict__ out) {
  const uint64_t npix = (uint64_t)W * H;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < npix;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t tx = (uint32_t)(i % W), ty = (uint32_t)(i / W);
    double r = 0, g = 0, bl = 0, wt = 0;
    for (int dy = 0; dy < 2; ++dy) {
      const uint32_t sy = ty + dy;
      if (sy >= H) continue;
      const int my = (dy == 0 && ty == 0 && fold_y) ? 2 : 1;
      for (int dx = 0; dx < 2; ++dx) {
        const uint32_t sx = tx + dx;
        if (sx >= W) continue;
        const int mx = (dx == 0 && tx == 0 && fold_x) ? 2 : 1;
        const uint64_t src = (uint64_t)sy * W + sx;
        double x, y, z, ww;
        if (sum64) {
          x = sum64[4 * src];
          y = sum64[4 * src + 1];
          z = sum64[4 * src + 2];
          ww = sum64[4 * src + 3];
        } else {
          const float4 s4 = sum[src], c4 = comp[src];
          x = (double)s4.x - (double)c4.x;
          y = (double)s4.y - (double)c4.y;
          z = (double)s4.z - (double)c4.z;
          ww = s4.w;
        }
        const int m = mx * my;
        r += m * x;
        g += m * y;
        bl += m * z;
        wt += m * ww;
      }
    }
    out[i] = make_float4((float)r, (float)g, (float)bl, (float)wt);
  }
}

__global__ void k_copy_li(WaveArgs a, const float4* __restrict__ rad,
                          uint64_t pixel_begin, uint32_t spp,
                          float* __restrict__ out) {
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < a.n_paths;
       p += gridDim.x * blockDim.x) {
    uint32_t pixel, sample;
    path_id(a, p, pixel, sample);
    float* o = out + 3 * (((uint64_t)pixel - pixel_begin) * spp + sample);
    const float4 L = rad[p];
    o[0] = L.x;
    o[1] = L.y;
    o[2] = L.z;
  }
}

int fail(ajg_ctx* ctx, int code, const std::string& m) {
  ctx->last_error = m;
  return code;
}

// SPPM's camera pass: each pixel's direct light (one path per pixel).
__global__ void k_copy_direct(WaveArgs a, const float4* __restrict__ rad,
                              float4* __restrict__ direct) {
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < a.n_paths;
       p += gridDim.x * blockDim.x)
    direct[a.pix0 + p] = rad[p];
}

}  // namespace

cudaError_t Scratch::take(ajg_ctx* ctx, uint64_t bytes, cudaStream_t st) {
  bytes = std::max<uint64_t>(bytes, 16);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(st, &cap);
  if (bytes > kScratchKeep || cap != cudaStreamCaptureStatusNone) {
    own = st;
    owned = device_malloc_async(ctx, (void**)&p, bytes, st);
    return owned ? cudaSuccess : cudaErrorMemoryAllocation;
  }
  if (ctx->scratch.bytes < bytes) {
    scratch_drop(ctx);
    const uint64_t want = std::max<uint64_t>(bytes, 8ull << 20);
    const cudaError_t e = cudaMalloc(&ctx->scratch.ptr, want);
    if (e != cudaSuccess) {
      ctx->scratch = Buffer{};
      cudaGetLastError();
      return e;
    }
    ctx->scratch.bytes = want;
  }
  p = static_cast<char*>(ctx->scratch.ptr);
  return cudaSuccess;
}

bool scratch_drop(ajg_ctx* ctx) {
  if (!ctx->scratch.ptr) return false;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(ctx->stream, &cap);
  if (cap != cudaStreamCaptureStatusNone) return false;
  cudaStreamSynchronize(ctx->stream);
  cudaFree(ctx->scratch.ptr);
  ctx->scratch = Buffer{};
  return true;
}

bool scratch_yield(ajg_ctx* ctx) {
  if (!ctx->mu.try_lock()) return false;
  const bool dropped = scratch_drop(ctx);
  ctx->mu.unlock();
  return dropped;
}

template <class Alloc, class Drop>
static bool alloc_or_drop(Alloc&& alloc, Drop&& drop, void** p) {
  if (alloc() == cudaSuccess) return true;
  cudaGetLastError();
  if (drop() && alloc() == cudaSuccess) return true;
  cudaGetLastError();
  *p = nullptr;
  return false;
}

bool device_malloc(ajg_ctx* ctx, void** p, uint64_t bytes, bool locked) {
  return alloc_or_drop(
      [&] { return cudaMalloc(p, bytes); },
      [&] { return locked ? scratch_drop(ctx) : scratch_yield(ctx); }, p);
}

bool device_malloc_async(ajg_ctx* ctx, void** p, uint64_t bytes, cudaStream_t st,
                         bool locked) {
  return alloc_or_drop(
      [&] { return cudaMallocAsync(p, bytes, st); },
      [&] { return locked ? scratch_drop(ctx) : scratch_yield(ctx); }, p);
}

int resident_grid(const void* fn, int threads, int carveout) {
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, int> cache;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  auto key = std::make_pair(fn, dev);
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  if (carveout >= 0)
    cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                         carveout);
  int sms = kSMs, per_sm = 1;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, 0) !=
          cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  const int g = sms * per_sm;
  cache[key] = g;
  return g;
}

uint64_t wave_bytes(uint64_t P, int nt, bool mj) {
  const uint64_t slots = P * nt;
  uint64_t b = 0;
  auto add = [&](uint64_t bytes) { b += ((bytes + 255) / 256) * 256; };
  add(P * 16); add(P * 16); add(P * 16);  // thr, thr_shade, rad
  if (mj) {
    add(P * 4);  // pjob
    add(P * 8);  // pkey
  }
  add(P * 4); add(P * 4);      // qpath
  add(P * 16); add(P * 16);    // ro
  add(P * 16); add(P * 16);    // rd
  add(P * sizeof(ajg_hit));
  add(slots * 16);             // term_f
  add(slots);                  // term_vis
  add(slots * 16); add(slots * 16);  // shadow queue
  if (mj) add(slots * 2);      // sq_scene
  add(P * 4 * 4);              // shading-class lists
  add(64);                     // (the counters' first 64 bytes)
  return b;
}

WaveBufs carve_wave(char* base, uint64_t P, int nt, bool mj) {
  char* cur = base;
  WaveBufs w{};
  w.thr = carve<float4>(cur, P);
  w.thr_shade = carve<float4>(cur, P);
  w.rad = carve<float4>(cur, P);
  if (mj) {
    w.pjob = carve<uint32_t>(cur, P);
    w.pkey = carve<uint64_t>(cur, P);
  }
  w.qpath[0] = carve<uint32_t>(cur, P);
  w.qpath[1] = carve<uint32_t>(cur, P);
  w.ro[0] = carve<float4>(cur, P);
  w.ro[1] = carve<float4>(cur, P);
  w.rd[0] = carve<float4>(cur, P);
  w.rd[1] = carve<float4>(cur, P);
  w.hits = carve<ajg_hit>(cur, P);
  w.term_f = carve<float4>(cur, P * nt);
  w.term_vis = carve<uint8_t>(cur, P * nt);
  w.sq_o = carve<float4>(cur, P * nt);
  w.sq_d = carve<float4>(cur, P * nt);
  if (mj) w.sq_scene = carve<uint16_t>(cur, P * nt);
  w.lists = carve<uint32_t>(cur, P * 4);
  w.counts = carve<uint32_t>(cur, 16);  // and behind: counter_bytes in all
  return w;
}

// The wave arena: one device allocation reused across renders of the
// context, grown when a render needs more paths or light terms.
static int ensure_arena(ajg_ctx* ctx, uint64_t P, int nt, char** base) {
  const uint64_t need = wave_bytes(P, nt, false) + counter_bytes(kMaxBounces);
  if (ctx->arena.empty() || ctx->arena[0].bytes < need) {
    for (auto& b : ctx->arena) cudaFree(b.ptr);
    ctx->arena.clear();
    Buffer b;
    if (!device_malloc(ctx, &b.ptr, need))
      return fail(ctx, AJG_ERR_OOM, "device allocation failed (wave arena)");
    b.bytes = need;
    ctx->arena.push_back(b);
  }
  *base = static_cast<char*>(ctx->arena[0].ptr);
  return AJG_OK;
}

// Paths per wave of a single-job render: the context's wave size, but no
// more than the render needs (its paths, in whole KiB) and no more than
// kArenaBytes of wave state for its light count.
constexpr uint64_t kArenaBytes = 96ull << 30;
static uint64_t job_wave_paths(const ajg_ctx* ctx, uint64_t needed, int nt) {
  const uint64_t per_path = (wave_bytes(1u << 20, nt, false) >> 20) + 1;
  uint64_t P = std::min<uint64_t>(ctx->wave_paths, (needed + 1023) / 1024 * 1024);
  P = std::min<uint64_t>(P, kArenaBytes / per_path);
  // the shadow queue (P x nt entries) is indexed by the traversal's 32-bit
  // signed ray numbers, with 2^31 - 1 reserved
  P = std::min<uint64_t>(P, ((1ull << 31) - 2) / (uint64_t)nt);
  return std::max<uint64_t>(1024, P / 1024 * 1024);
}

int check_render(ajg_ctx* ctx, const DeviceScene& s, const ajg_camera& cam,
                 const ajg_render_params& prm) {
  if (cam.width == 0 || cam.height == 0 || prm.spp == 0)
    return fail(ctx, AJG_ERR_INVALID, "empty film or zero spp");
  if (prm.max_bounces < 0 || prm.max_bounces > kMaxBounces)
    return fail(ctx, AJG_ERR_INVALID, "max_bounces must be in [0, 1024]");
  if (s.num_lights > kMaxLights)
    return fail(ctx, AJG_ERR_UNSUPPORTED, "at most 15 lights");
  if ((uint64_t)cam.width * cam.height > (1ull << 31))
    return fail(ctx, AJG_ERR_INVALID, "film too large");
  return AJG_OK;
}

// Bounce 0's directional-light shadow rays as packets (trace_packet_any): a
// packet walks the union of its rays' traversals, which near their origins
// grows with the triangles they span.  The measure is a pixel's footprint at
// the world box's centre -- the angle between the rays through the film
// centre and the pixel beside it, times the camera's distance to that centre
// -- in median triangle edges (kPacketSpread of them: packet_spread), times
// the pixels a packet of 32 spans when a wave holds S samples of each.
static float packet_ratio(const ajg_scene* sc, const ajg_camera& cam) {
  auto apply = [](const float* m, const float v[4], float o[4]) {
    for (int r = 0; r < 4; ++r) {
      o[r] = 0.f;
      for (int c = 0; c < 4; ++c) o[r] += m[c * 4 + r] * v[c];
    }
  };
  const float cx = 0.5f * (float)cam.width, cy = 0.5f * (float)cam.height;
  const float p0[4] = {cx, cy, 1.f, 1.f}, p1[4] = {cx + 1.f, cy, 1.f, 1.f};
  float q0[4], q1[4];
  apply(cam.raster2camera, p0, q0);
  apply(cam.raster2camera, p1, q1);
  auto unit = [](const float q[4], double u[3]) {
    const double n = std::sqrt((double)q[0] * q[0] + (double)q[1] * q[1] +
                               (double)q[2] * q[2]);
    for (int k = 0; k < 3; ++k) u[k] = n > 0 ? q[k] / n : 0.0;
  };
  double u0[3], u1[3];
  unit(q0, u0);
  unit(q1, u1);
  const double angle = std::sqrt((u1[0] - u0[0]) * (u1[0] - u0[0]) +
                                 (u1[1] - u0[1]) * (u1[1] - u0[1]) +
                                 (u1[2] - u0[2]) * (u1[2] - u0[2]));
  const float* m = cam.camera2world;  // column-major: translation in 12..14
  double dist2 = 0.0;
  for (int k = 0; k < 3; ++k) {
    const double c = 0.5 * ((double)sc->world[k] + sc->world[k + 3]);
    const double e = (double)m[12 + k] / (m[15] != 0.f ? m[15] : 1.f) - c;
    dist2 += e * e;
  }
  return (float)(angle * std::sqrt(dist2) / (double)sc->d.packet_spread);
}
// Packets pay up to one edge in waves of 4 Mi paths, half of one at 2 Mi (a
// packet's walk is longer than a ray's, and a short launch waits for it), not
// at all below.  Per-lane time over packet time of whole one-bounce renders
// of displaced spheres, by span in edges: 2 Mi paths 0.24 1.015, 0.49 0.999,
// 0.98 0.97; 4 Mi 0.49 1.03, 0.98 0.99 to 1.01, 1.96 0.91 to 0.95; 16 Mi and
// more 0.98 1.03 to 1.05, 1.96 0.99, 3.9 0.90; 1 Mi 0.49 0.99, 3.9 0.79;
// 262,144 paths 15.7 0.67, 31 0.61.
bool packets_pay(const JobParams& j, uint64_t S, uint64_t paths) {
  return paths >= (1u << 21) &&
         j.packet_ratio * (float)((31 + S) / S) <=
             std::min(1.f, (float)paths / (float)(1u << 22));
}

JobParams make_job_params(const ajg_scene* sc, const ajg_camera& cam,
                          const ajg_render_params& prm) {
  const DeviceScene& s = sc->d;
  JobParams j{};
  j.seed = prm.seed;
  j.min_b = prm.min_bounces;
  j.max_b = prm.max_bounces;
  j.cont = prm.cont_prob;
  j.use_mis = prm.use_mis ? 1 : 0;
  j.nl = (int)s.num_lights;
  // draws per bounce: 2 per directional or env light, 3 per area light,
  // 3 for the MIS BSDF sample and 3 for the continuation
  j.nd = j.use_mis ? (2 * j.nl + (int)s.num_area + 6) : 3;
  j.env_rgb = make_float4(0, 0, 0, 0);
  j.env_mass = 0;
  if (s.env >= 0) {
    const float* L = sc->host_lights.data() + 12 * s.env;
    // EnvLight::Radiance = scaler * texel (env_light.cpp:65)
    j.env_rgb = make_float4(L[8] * L[1], L[8] * L[2], L[8] * L[3], 0.f);
    j.env_mass = L[11] != 0.f ? 1 : 0;
  }
  j.drop_nonfinite = (prm.flags & AJG_RENDER_DROP_NONFINITE) ? 1 : 0;
  j.film_w = cam.width;
  j.film_h = cam.height;
  j.x0 = j.y0 = 0;
  j.win_w = cam.width;
  j.win_h = cam.height;
  j.packet_ratio = packet_ratio(sc, cam);
  return j;
}

// The sample loop of one render over zeroed film accumulators: waves of S
// samples of a pixel range, the bounce loop per wave, the film update per
// wave and the footprint resolve at the end.  `timers` enables the
// profiling events of the traversal and shading launches.
static void run_waves(ajg_scene* sc, const ajg_camera& cam,
                      const ajg_render_params& prm, const WaveBufs& w,
                      uint64_t P, float4* fsum, float4* fcomp, double* fsum64,
                      float4* d_out, uint64_t li_begin, uint64_t li_end,
                      float* d_li, cudaStream_t st, bool timers,
                      VisPointD* vp = nullptr, float4* d_direct = nullptr) {
  ajg_ctx* ctx = sc->ctx;
  const DeviceScene& s = sc->d;
  const int nt = (int)s.num_lights + 1;
  const uint64_t npix_all = (uint64_t)cam.width * cam.height;
  const bool want_film = d_out != nullptr;
  const int kc = timers ? kKindClosest : -1;
  const int ka = timers ? kKindAny : -1;
  const int ks = timers ? kKindShade : -1;
  const int kcp = timers ? kKindClosestPacket : -1;
  const int kap = timers ? kKindAnyPacket : -1;
  const MJTables t{};

  WaveArgs a;
  a.s = s;
  a.cam = cam;
  a.j = make_job_params(sc, cam, prm);
  a.vp = vp;

  const uint64_t pb = d_li ? li_begin : 0;
  const uint64_t pe = d_li ? li_end : npix_all;
  const uint64_t npix = pe - pb;
  uint64_t S = std::min<uint64_t>(prm.spp, std::max<uint64_t>(1, P / npix));
  const uint64_t chunk = std::min<uint64_t>(npix, P / S);
  const uint32_t shadow_cap = (uint32_t)(P * nt);
  const int gs = kSMs * 8;
  // persistent traversal: resident blocks only
  const DeviceScene s_closest = closest_view(s);
  // bounce 0's camera rays (a pixel's samples side by side in the queue) as
  // masked packets over the binary layout (AJG_PACKET_CAMERA)
  const bool cam_packets = ctx->packet_camera && s_closest.width == 2;
  // the wave's buffers with bounce b's counters
  auto at_bounce = [&](int b) {
    WaveBufs wb = w;
    wb.counts = w.counts + kCounterWords * b;
    return wb;
  };
  auto extend = [&](const WaveBufs& wb, int q, cudaStream_t es, bool cam) {
    if (cam)
      launch_wave_extend_packet(false, s_closest.tri_test, s_closest, t,
                                w.ro[q], w.rd[q], &wb.counts[0], &wb.counts[8],
                                wb.hits, &ctx->d_counters[0], ctx->d_error, es);
    else
      launch_wave_extend(false, s_closest.tri_test, s_closest.width, s_closest,
                         t, w.ro[q], w.rd[q], &wb.counts[0], &wb.counts[8],
                         wb.hits, &ctx->d_counters[0], ctx->d_error, es);
  };
  auto classify = [&](const WaveBufs& wb, int b, int q, cudaStream_t es) {
    KernelTimer tm(ctx, es, -1);
    k_classify<false><<<gs, kClassifyThreads, 0, es>>>(a, t, wb, b, q, (uint32_t)P);
  };
  // Bounce b+1's closest hits run on the trace stream beside bounce b's
  // shadow rays: the two persistent launches fill each other's drain.  The
  // queues alternate by bounce parity, the hits have been shaded; everything
  // else bounce b+1 touches is written after k_accumulate of bounce b on the
  // render stream.  Its classification follows the hits there, except in
  // scenes with emitters, whose MIS BSDF hits borrow the lists.
  const bool overlap = ctx->overlap && !ctx->profiling;
  const bool classify_ahead = overlap && !s.tri_emit;
  cudaStream_t ts = ctx->trace_stream;
  auto extend_ahead = [&](int b, int q, bool cam) {
    const WaveBufs wb = at_bounce(b);
    cudaEventRecord(ctx->ev_queue, st);
    cudaStreamWaitEvent(ts, ctx->ev_queue, 0);
    {
      KernelTimer tm(ctx, ts, cam ? kcp : kc);
      extend(wb, q, ts, cam);
    }
    if (classify_ahead) classify(wb, b, q, ts);
    cudaEventRecord(ctx->ev_hits, ts);
  };
  auto bsdf_closest = [&](const WaveBufs& wb) {
    launch_wave_bsdf_trace(false, s_closest.tri_test, s_closest.width, s_closest, t,
                           w.sq_o, w.sq_d,
                           nullptr, &wb.counts[9], &wb.counts[10], shadow_cap,
                           (uint32_t)P, reinterpret_cast<float*>(w.lists),
                           reinterpret_cast<int32_t*>(w.lists + P),
                           &ctx->d_counters[0], ctx->d_error, st);
  };
  auto shadow = [&](const WaveBufs& wb) {
    launch_wave_shadow(false, s.tri_test, s.width, s, t, w.sq_o, w.sq_d, nullptr,
                       &wb.counts[2], &wb.counts[3], w.term_vis,
                       &ctx->d_counters[1], ctx->d_error, st);
  };
  // Coherent shadow rays: at bounce 0 a shading block's rays of one light
  // term are a pixel's samples (one origin region; toward a directional
  // light, one direction), traced as masked packets from a queue of their
  // own.  Single jobs without emitters (the BSDF rays of scenes with
  // emitters use the top of the storage) over the plain 4-wide tree.
  uint32_t coh0 = 0;
  if (ctx->packet_shadow > 0 && !s.tri_emit && s.width == 4 && a.j.use_mis &&
      (packets_pay(a.j, S, S * chunk) || ctx->packet_shadow >= 2)) {
    for (int l = 0; l < (int)s.num_lights && l < 31; ++l)
      if (ctx->packet_shadow == 2 ||
          (int)sc->host_lights[12 * l] == AJG_LIGHT_DIRECTIONAL)
        coh0 |= 1u << l;
    if (ctx->packet_shadow >= 2) coh0 |= 1u << 31;  // 3: directional + BSDF
  }
  auto shadow_packets = [&](const WaveBufs& wb) {
    launch_wave_shadow_packet(false, s.tri_test, s, t, w.sq_o, w.sq_d, nullptr,
                              &wb.counts[11], &wb.counts[12], shadow_cap,
                              w.term_vis, &ctx->d_counters[1], ctx->d_error,
                              st);
  };
  for (uint64_t s0 = 0; s0 < prm.spp; s0 += S) {
    const uint64_t Sw = std::min<uint64_t>(S, prm.spp - s0);
    for (uint64_t p0 = pb; p0 < pe; p0 += chunk) {
      const uint64_t n_pix = std::min<uint64_t>(chunk, pe - p0);
      a.pix0 = (uint32_t)p0;
      a.S = (uint32_t)Sw;
      a.s0 = (uint32_t)s0;
      a.n_paths = (uint32_t)(n_pix * Sw);
      // shading grids: many short blocks (the block-wide loop waits on its
      // slowest warp each round; small blocks of work keep the SMs evenly
      // busy to the end), never more than the wave's paths need
      const int gsh = grid_for(a.n_paths, kShadeThreads, kSMs * AJG_SHADE_GRID);
      cudaMemsetAsync(w.counts, 0, counter_bytes(a.j.max_b), st);
      KernelTimer{ctx, st, -1};
      k_raygen<false><<<grid_for(a.n_paths, kShadeThreads, gs), kShadeThreads,
                        0, st>>>(a, t, w);
      int q = 0;
      if (overlap && a.j.max_b > 0) extend_ahead(0, 0, cam_packets);
      for (int b = 0; b < a.j.max_b; ++b) {
        const WaveBufs wb = at_bounce(b);
        const uint32_t coh = b < ctx->packet_bounces ? coh0 : 0u;
        if (overlap) {
          cudaStreamWaitEvent(st, ctx->ev_hits, 0);
        } else {
          const bool cam = b == 0 && cam_packets;
          KernelTimer tm(ctx, st, cam ? kcp : kc);
          extend(wb, q, st, cam);
        }
        if (!classify_ahead) classify(wb, b, q, st);
        // one shading launch per material class the scene has
        if (s.mat_mask & (1u << AJG_MAT_DIFFUSE)) {
          KernelTimer tm(ctx, st, ks);
          k_shade<AJG_MAT_DIFFUSE, false><<<gsh, kShadeThreads, 0, st>>>(
              a, t, wb, b, q, w.lists + P, &wb.counts[5], (uint32_t)nt,
              shadow_cap, ctx->d_error, coh);
        }
        if (s.mat_mask & (1u << AJG_MAT_DISNEY)) {
          KernelTimer tm(ctx, st, ks);
          k_shade<AJG_MAT_DISNEY, false><<<gsh, kShadeThreads, 0, st>>>(
              a, t, wb, b, q, w.lists + 2 * P, &wb.counts[6], (uint32_t)nt,
              shadow_cap, ctx->d_error, coh);
        }
        if (s.mat_mask & kOtherTypes) {
          KernelTimer tm(ctx, st, ks);
          k_shade<kMatOther, false><<<gsh, kShadeThreads, 0, st>>>(
              a, t, wb, b, q, w.lists + 3 * P, &wb.counts[7], (uint32_t)nt,
              shadow_cap, ctx->d_error, coh);
        }
        if (s.mat_mask & kDeltaTypes) {
          KernelTimer tm(ctx, st, ks);
          k_shade<kMatDelta, false><<<gsh, kShadeThreads, 0, st>>>(
              a, t, wb, b, q, w.lists, &wb.counts[4], (uint32_t)nt, shadow_cap,
              ctx->d_error, coh);
        }
        if (overlap && b + 1 < a.j.max_b)
          extend_ahead(b + 1, q ^ 1, false);
        if (a.j.use_mis) {
          {
            KernelTimer tm(ctx, st, ka);
            shadow(wb);
          }
          if (coh) {
            KernelTimer tm(ctx, st, kap);
            shadow_packets(wb);
          }
          if (s.tri_emit) {
            {
              KernelTimer tm(ctx, st, kc);
              bsdf_closest(wb);
            }
            KernelTimer{ctx, st, -1};
            k_bsdf_emit<false><<<gs, kShadeThreads, 0, st>>>(
                a, t, wb, (uint32_t)nt, shadow_cap, (uint32_t)P,
                reinterpret_cast<const float*>(w.lists),
                reinterpret_cast<const int32_t*>(w.lists + P));
          }
          KernelTimer{ctx, st, -1};
          k_accumulate<false><<<gs, kShadeThreads, 0, st>>>(a, t, wb, q,
                                                            (uint32_t)nt);
        }
        q ^= 1;
      }
      if (want_film) KernelTimer{ctx, st, -1};
      if (want_film)
        k_film_add<false><<<grid_for(n_pix, 256, gs), 256, 0, st>>>(
            a, t, w.rad, fsum, fcomp, fsum64, (uint32_t)n_pix);
      if (d_li) KernelTimer{ctx, st, -1};
      if (d_li)
        k_copy_li<<<grid_for(a.n_paths, 256, gs), 256, 0, st>>>(
            a, w.rad, li_begin, prm.spp, d_li);
      if (d_direct) {
        KernelTimer{ctx, st, -1};
        k_copy_direct<<<grid_for(a.n_paths, 256, gs), 256, 0, st>>>(
            a, w.rad, d_direct);
      }
    }
  }
  if (want_film) {
    KernelTimer{ctx, st, -1};
    k_resolve<<<grid_for(npix_all, 256, gs), 256, 0, st>>>(
        fsum, fcomp, fsum64, cam.width, cam.height, 1, 1, d_out);
  }
  ctx->paths_total += (unsigned long long)npix * prm.spp;
}

void enqueue_mj_wave(const MJTables& t, const WaveBufs& w, uint64_t P,
                     int NT, int bounces, int tri_test, int width, bool emit,
                     uint32_t mat_mask, TraceCounters* ctr, uint32_t* err, cudaStream_t st,
                     cudaStream_t ts, cudaEvent_t ev_queue,
                     cudaEvent_t ev_hits, bool cam_packets,
                     bool shadow_packets) {
  const DeviceScene s{};
  WaveArgs a{};
  const uint32_t shadow_cap = (uint32_t)(P * NT);
  const int gs = kSMs * 8;
  const int gsh = grid_for(P, kShadeThreads, kSMs * AJG_MJ_SHADE_GRID);
  const int gso = grid_for(P, kShadeThreads, kSMs * 8);
  // bounce 0's camera rays (each chunk's paths a pixel's samples side by
  // side) as masked packets when the closest hits walk binary trees
  const bool cam_ok = cam_packets && closest_width(width) == 2;
  // and its directional-light shadow rays, in waves without emitters over
  // plain 4-wide trees
  const bool shadow_ok = shadow_packets && !emit && width == 4;
  // bounce b+1's closest hits on the trace stream beside bounce b's shadow
  // rays, as in the single-job waves (run_waves)
  const bool overlap = ts && ev_queue && ev_hits;
  const bool classify_ahead = overlap && !emit;
  auto at_bounce = [&](int b) {
    WaveBufs wb = w;
    wb.counts = w.counts + kCounterWords * b;
    return wb;
  };
  auto extend = [&](const WaveBufs& wb, int q, cudaStream_t es, bool cam) {
    if (cam)
      launch_wave_extend_packet(true, tri_test, s, t, w.ro[q], w.rd[q],
                                &wb.counts[0], &wb.counts[8], wb.hits, ctr, err,
                                es);
    else
      launch_wave_extend(true, tri_test, closest_width(width), s, t, w.ro[q],
                         w.rd[q], &wb.counts[0], &wb.counts[8], wb.hits, ctr, err,
                         es);
  };
  auto classify = [&](const WaveBufs& wb, int b, int q, cudaStream_t es) {
    k_classify<true><<<gs, kClassifyThreads, 0, es>>>(a, t, wb, b, q, (uint32_t)P);
  };
  auto extend_ahead = [&](int b, int q, bool cam) {
    const WaveBufs wb = at_bounce(b);
    cudaEventRecord(ev_queue, st);
    cudaStreamWaitEvent(ts, ev_queue, 0);
    extend(wb, q, ts, cam);
    if (classify_ahead) classify(wb, b, q, ts);
    cudaEventRecord(ev_hits, ts);
  };
  cudaMemsetAsync(w.counts, 0, counter_bytes(bounces), st);
  k_raygen<true><<<gs, kShadeThreads, 0, st>>>(a, t, w);
  int q = 0;
  if (overlap && bounces > 0) extend_ahead(0, 0, cam_ok);
  for (int b = 0; b < bounces; ++b) {
    const WaveBufs wb = at_bounce(b);
    const uint32_t coh = b == 0 && shadow_ok ? 1u : 0u;
    if (overlap)
      cudaStreamWaitEvent(st, ev_hits, 0);
    else
      extend(wb, q, st, b == 0 && cam_ok);
    if (!classify_ahead) classify(wb, b, q, st);
    k_shade<AJG_MAT_DIFFUSE, true><<<gsh, kShadeThreads, 0, st>>>(
        a, t, wb, b, q, w.lists + P, &wb.counts[5], (uint32_t)NT, shadow_cap,
        err, coh);
    k_shade<AJG_MAT_DISNEY, true><<<gsh, kShadeThreads, 0, st>>>(
        a, t, wb, b, q, w.lists + 2 * P, &wb.counts[6], (uint32_t)NT,
        shadow_cap, err, coh);
    if (mat_mask & kOtherTypes)
      k_shade<kMatOther, true><<<gso, kShadeThreads, 0, st>>>(
          a, t, wb, b, q, w.lists + 3 * P, &wb.counts[7], (uint32_t)NT,
          shadow_cap, err, coh);
    if (mat_mask & kDeltaTypes)
      k_shade<kMatDelta, true><<<gso, kShadeThreads, 0, st>>>(
          a, t, wb, b, q, w.lists, &wb.counts[4], (uint32_t)NT, shadow_cap, err,
          coh);
    if (overlap && b + 1 < bounces)
      extend_ahead(b + 1, q ^ 1, false);
    launch_wave_shadow(true, tri_test, width, s, t, w.sq_o, w.sq_d, w.sq_scene,
                       &wb.counts[2], &wb.counts[3], w.term_vis, ctr + 1, err, st);
    if (coh)
      launch_wave_shadow_packet(true, tri_test, s, t, w.sq_o, w.sq_d,
                                w.sq_scene, &wb.counts[11], &wb.counts[12],
                                shadow_cap, w.term_vis, ctr + 1, err, st);
    if (emit) {
      launch_wave_bsdf_trace(true, tri_test, closest_width(width), s, t, w.sq_o, w.sq_d,
                             w.sq_scene, &wb.counts[9], &wb.counts[10], shadow_cap,
                             (uint32_t)P, reinterpret_cast<float*>(w.lists),
                             reinterpret_cast<int32_t*>(w.lists + P), ctr, err,
                             st);
      k_bsdf_emit<true><<<gs, kShadeThreads, 0, st>>>(
          a, t, wb, (uint32_t)NT, shadow_cap, (uint32_t)P,
          reinterpret_cast<const float*>(w.lists),
          reinterpret_cast<const int32_t*>(w.lists + P));
    }
    k_accumulate<true><<<gs, kShadeThreads, 0, st>>>(a, t, wb, q,
                                                     (uint32_t)NT);
    q ^= 1;
  }
  k_film_add<true><<<gs, 256, 0, st>>>(a, t, w.rad, nullptr, nullptr, nullptr,
                                       0);
}

void enqueue_resolve(const float4* fsum, const float4* fcomp,
                     const double* fsum64, uint32_t w, uint32_t h,
                     bool fold_x, bool fold_y, float4* out, cudaStream_t st) {
  k_resolve<<<grid_for((uint64_t)w * h, 256, kSMs * 8), 256, 0, st>>>(
      fsum, fcomp, fsum64, w, h, fold_x ? 1 : 0, fold_y ? 1 : 0, out);
}

int reserve_wave(ajg_scene* sc, const ajg_camera& cam,
                 const ajg_render_params& prm, uint64_t npix) {
  int rc = check_render(sc->ctx, sc->d, cam, prm);
  if (rc) return rc;
  const int nt = (int)sc->d.num_lights + 1;
  char* base = nullptr;
  return ensure_arena(sc->ctx, job_wave_paths(sc->ctx, npix * prm.spp, nt), nt,
                      &base);
}

int render_impl(ajg_scene* sc, const ajg_camera& cam,
                const ajg_render_params& prm, float4* d_out, void* film,
                uint64_t li_begin, uint64_t li_end, float* d_li,
                cudaStream_t st) {
  ajg_ctx* ctx = sc->ctx;
  const DeviceScene& s = sc->d;
  int rc = check_render(ctx, s, cam, prm);
  if (rc) return rc;
  const int nt = (int)s.num_lights + 1;
  const uint64_t npix_all = (uint64_t)cam.width * cam.height;
  const uint64_t npix_job = d_li ? std::min(li_end, npix_all) - li_begin : npix_all;
  const uint64_t P = job_wave_paths(ctx, npix_job * prm.spp, nt);
  char* base = nullptr;
  rc = ensure_arena(ctx, P, nt, &base);
  if (rc) return rc;
  const WaveBufs w = carve_wave(base, P, nt, false);

  // film accumulators: per pixel a float32 sum and Kahan compensation, or a
  // float64 sum
  float4 *fsum = nullptr, *fcomp = nullptr;
  double* fsum64 = nullptr;
  if (d_out) {
    if (prm.flags & AJG_RENDER_FP64_FILM) {
      fsum64 = static_cast<double*>(film);
    } else {
      fsum = static_cast<float4*>(film);
      fcomp = fsum + npix_all;
    }
    cudaMemsetAsync(film, 0, npix_all * 32, st);
  }
  run_waves(sc, cam, prm, w, P, fsum, fcomp, fsum64, d_out, li_begin, li_end,
            d_li, st, true);
  return AJG_OK;
}

int render_in_scratch(ajg_scene* sc, const ajg_camera& cam,
                      const ajg_render_params& prm, float4* d_out,
                      cudaStream_t st, char* scratch, uint64_t bytes) {
  ajg_ctx* ctx = sc->ctx;
  const DeviceScene& s = sc->d;
  int rc = check_render(ctx, s, cam, prm);
  if (rc) return rc;
  const int nt = (int)s.num_lights + 1;
  const uint64_t npix = (uint64_t)cam.width * cam.height;
  const uint64_t film_bytes = ((npix * 32 + 255) / 256) * 256;
  const uint64_t min_wave = wave_bytes(1024, nt, false);
  if (film_bytes + min_wave > bytes)
    return fail(ctx, AJG_ERR_INVALID,
                "film of " + std::to_string(npix) + " pixels needs " +
                    std::to_string(film_bytes + min_wave) +
                    " bytes of scratch; the static scratch holds " +
                    std::to_string(bytes) + " (at most " +
                    std::to_string((bytes - min_wave) / 32) + " pixels)");
  uint64_t P = 1024;
  while (wave_bytes(P + 1024, nt, false) + film_bytes <= bytes) P += 1024;
  float4* fsum = nullptr;
  float4* fcomp = nullptr;
  double* fsum64 = nullptr;
  // the scratch keeps the previous call's contents: zero the film
  if (prm.flags & AJG_RENDER_FP64_FILM) {
    fsum64 = reinterpret_cast<double*>(scratch);
  } else {
    fsum = reinterpret_cast<float4*>(scratch);
    fcomp = fsum + npix;
  }
  cudaMemsetAsync(scratch, 0, npix * 32, st);
  const WaveBufs w = carve_wave(scratch + film_bytes, P, nt, false);
  run_waves(sc, cam, prm, w, P, fsum, fcomp, fsum64, d_out, 0, 0, nullptr, st,
            false);
  return AJG_OK;
}

// TracerVP is TraceMIS without roulette that stops at a visible point:
// min = max bounces = fmd, sample 0 of each pixel (SetSeed(x + y W))
static ajg_render_params sppm_camera_params(int fmd, uint64_t seed) {
  ajg_render_params prm{};
  prm.spp = 1;
  prm.min_bounces = fmd;
  prm.max_bounces = fmd;
  prm.cont_prob = 1.f;
  prm.use_mis = 1;
  prm.seed = seed;
  return prm;
}

int sppm_reserve(ajg_scene* sc, const ajg_camera& cam, int fmd) {
  return reserve_wave(sc, cam, sppm_camera_params(fmd, 0),
                      (uint64_t)cam.width * cam.height);
}

int sppm_camera_pass(ajg_scene* sc, const ajg_camera& cam, int fmd,
                     uint64_t seed, VisPointD* vp, float4* direct,
                     cudaStream_t st) {
  ajg_ctx* ctx = sc->ctx;
  const ajg_render_params prm = sppm_camera_params(fmd, seed);
  int rc = check_render(ctx, sc->d, cam, prm);
  if (rc) return rc;
  const int nt = (int)sc->d.num_lights + 1;
  const uint64_t npix = (uint64_t)cam.width * cam.height;
  const uint64_t P = job_wave_paths(ctx, npix, nt);
  char* base = nullptr;
  rc = ensure_arena(ctx, P, nt, &base);
  if (rc) return rc;
  const WaveBufs w = carve_wave(base, P, nt, false);
  cudaMemsetAsync(vp, 0xff, npix * sizeof(VisPointD), st);
  run_waves(sc, cam, prm, w, P, nullptr, nullptr, nullptr, nullptr, 0, 0,
            nullptr, st, false, vp, direct);
  return AJG_OK;
}

}  // namespace ajg
