// wavefront.cu -- the path integrator (render/path-integ.cc:134-407) as a
// wavefront on sm_100a.
//
// A job's render pattern (the image plus the Mitchell filter's 2-pixel
// margin, snogray.lua:543-550) times its samples per pixel is processed in
// waves of whole pixels.  Per wave:
//   k_camera                 eye rays for every path (camera/camera.cc:108-160)
//   per bounce b = 0..max_len:
//     k_trace_closest        octree closest hit for the live rays
//     k_shade                emission, BSDF continuation, Russian
//                            roulette; appends surviving rays to the other
//                            queue with warp-aggregated atomics and lists
//                            the vertices to light
//     k_direct               direct lighting with MIS of the listed
//                            vertices (emits shadow rays)
//     k_trace_shadow         any-hit for the shadow rays; unoccluded ones add
//                            their contribution to the path's radiance; on a
//                            stream of its own, beside the next bounce's
//                            k_trace_closest, and joined before its k_shade
//   k_splat                  Mitchell filter of the wave's samples, by image tiles
//                            into the image accumulator
// and finally k_resolve divides by the filter weight
// (image/image-sampled-output.cc:79-123).
//
// Path state is SoA of 16-byte records (float4 throughput+rr ratio, float4
// radiance+alpha) plus a 32-bit word: path length (8 bits), after-specular
// (1 bit), media-stack depth (3 bits) and up to four medium ids (5 bits
// each).  Queues hold rays as two float4 (origin+t0, direction+t1) in queue
// order, so the trace kernels read them with coalesced 128-bit loads.

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <type_traits>

#include "launch.h"
#include "pathstate.cuh"
#include "scene.h"
#include "wavefront.h"

namespace cg = cooperative_groups;

namespace snog {

namespace {

struct PathPtrs {
  float4 *thr, *rad;
  uint32_t *pstate;
  float2 *jit;
};
struct RayQ {
  float4 *o, *d;
  uint32_t *path;
};
struct ShadowQ {
  float4 *o, *d, *c;
};
struct DirectL {             // vertices to light, written by k_shade
  uint32_t *idx;             // queue index
  float4 *thr;               // throughput before the continuation, path state word in w
};

// ---- kernels -----------------------------------------------------------------

// A bounce is a chain of kernels, of a few microseconds each on a small image, and
// between two of them the device drains, launches and fills again for 2 to 3 more.
// A kernel that calls this first, in every thread, lets the next kernel's blocks
// take the room that its own leave, and touches nothing before the kernel
// before it has completed (which implies that the ones before that have).
// 64x48 Cornell 463 -> 437 us, 256x256x16 2.19 -> 2.16 ms, 853x479 terrain
// unchanged at 7.4.  The engine's iterations lost by it (terrain frame 162.2 ->
// 165.3 ms, 1024x1024x16 Cornell 30.8 -> 31.8): the next closest hits then hold
// the room that the shadow rays, whose launch is the longer one there, start in.
__device__ __forceinline__ void start_after_previous() {
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
}

// Launch K, which calls start_after_previous(), on ST: if EARLY, set up while the
// kernel before it there still runs.  Errors are left for cudaGetLastError().
template <class... P, class... A>
void launch_after(bool early, void (*k)(P...), dim3 grid, uint32_t block, cudaStream_t st, A... a) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = early ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k, P(a)...);
}

__global__ void __launch_bounds__(256) k_camera(JobConsts jc, uint64_t base, uint32_t n, PathPtrs P, RayQ q,
                                                uint32_t *counters) {
  start_after_previous();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    counters[0] = n;
    counters[1] = 0;
    counters[2] = 0;
    counters[4] = 0;          // closest kernel's dispenser
  }
  const Strata st = strata_for(jc.S);
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
    const uint64_t g = base + p;
    const uint32_t pixel = uint32_t(g / jc.S), s = uint32_t(g % jc.S);
    const int px = jc.PX + int(pixel % jc.PW), py = jc.PY + int(pixel / jc.PW);
    Rng rng{jc.seed_lo, jc.seed_hi, uint32_t(g), uint32_t(g >> 32)};
    float2 j = strat_uv(st, rng, pixel, s, dim_of(0, K_CAMERA));
    // Renderer::render_packet (render-mgr/renderer.cc:69-88) and
    // Camera::eye_vec (camera/camera.h:384-389).
    float cu = float(px) + j.x, cv = float(py) + j.y;
    float fu = cu / float(jc.FW), fv = (float(jc.FH) - cv) / float(jc.FH);
    float x = 2.f * fu - 1.f, y = 2.f * fv - 1.f;
    float3 d = add(add(load3(jc.cam_fwd), mul(mul(load3(jc.cam_right), x), jc.tan_x)),
                   mul(mul(load3(jc.cam_up), y), jc.tan_y));
    q.o[p] = make_float4(jc.cam_pos[0], jc.cam_pos[1], jc.cam_pos[2], 0.f);
    q.d[p] = make_float4(d.x, d.y, d.z, jc.max_trace);
    q.path[p] = p;
    P.thr[p] = make_float4(1.f, 1.f, 1.f, 1.f);
    P.rad[p] = make_float4(0.f, 0.f, 0.f, 1.f);
    P.pstate[p] = 0;
    P.jit[p] = j;
  }
}

// Add a thread's node/test counts to P[0..1] with one atomic per warp; every
// lane of the block must call it.
__device__ __forceinline__ void warp_count(unsigned long long *p, unsigned long long nodes,
                                           unsigned long long tests) {
  for (int off = 16; off > 0; off >>= 1) {
    nodes += __shfl_down_sync(0xffffffffu, nodes, off);
    tests += __shfl_down_sync(0xffffffffu, tests, off);
  }
  if ((threadIdx.x & 31u) == 0) {
    atomicAdd(p, nodes);
    atomicAdd(p + 1, tests);
  }
}

// Persistent closest-hit kernel: warps take rays from the queue through a
// RayDispenser (counters[4]) and interleave one octree entry per ray per
// iteration, so finished lanes are refilled instead of idling.
template <int STACK, int PER, bool COUNT>
__global__ void __launch_bounds__(kTraceBlock, SNOG_TRACE_MINBLOCKS)
    k_trace_closest(DevScene s, RayQ q, uint32_t *counters, uint32_t cur, uint32_t *hit_ref, float *hit_t,
                    unsigned long long *stats) {
  start_after_previous();
  const uint32_t n = counters[cur];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    counters[cur ^ 1u] = 0;   // the next queue and the direct-lighting list start empty
    counters[6] = 0;
    stats[0] += n;
  }
  TraceCounters c{0, 0, 0};
  trace_loop<STACK, kClosestOnly, PER, COUNT>(
      counters + 4, n, c,
      [&](uint32_t ray, Traversal<STACK> &tr, bool &any) {
        const float4 o = q.o[ray], d = q.d[ray];
        tr.init(s, xyz(o), xyz(d), o.w, d.w);
        any = false;
      },
      [&](uint32_t ray, Traversal<STACK> &tr, bool) {
        hit_ref[ray] = tr.hit_ref;
        hit_t[ray] = tr.t1;
      });
  if (c.overflow) atomicOr(counters + 3, 1u);
  if (COUNT) warp_count(stats + 2, c.nodes, c.tests);
}

// Persistent any-hit kernel for the shadow queue (dispenser counters[5]);
// an unoccluded ray adds its contribution to its path's radiance.
template <int STACK, bool COUNT>
__global__ void __launch_bounds__(kTraceBlock, SNOG_TRACE_MINBLOCKS)
    k_trace_shadow(DevScene s, ShadowQ q, uint32_t *counters, float4 *rad, unsigned long long *stats) {
  const uint32_t n = counters[2];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    stats[1] += n;
  }
  TraceCounters c{0, 0, 0};
  trace_loop<STACK, kAnyOnly, 1, COUNT>(
      counters + 5, n, c,
      [&](uint32_t ray, Traversal<STACK> &tr, bool &any) {
        const float4 o = q.o[ray], d = q.d[ray];
        tr.init(s, xyz(o), xyz(d), o.w, d.w);
        any = true;
      },
      [&](uint32_t ray, Traversal<STACK> &tr, bool) {
        if (tr.hit_ref != PREF_END) return;
        const float4 cc = q.c[ray];
        float4 *r = rad + __float_as_uint(cc.w);
        atomicAdd(&r->x, cc.x);
        atomicAdd(&r->y, cc.y);
        atomicAdd(&r->z, cc.z);
      });
  if (c.overflow) atomicOr(counters + 3, 1u);
  if (COUNT) warp_count(stats + 4, c.nodes, c.tests);
}

// 6 blocks of 128 per SM (80 registers), as the engine's shading kernels.
__global__ void __launch_bounds__(128, 6) k_shade(DevScene s, JobConsts jc, uint64_t base, uint32_t bounce,
                                               RayQ qin, uint32_t *counters, uint32_t cur,
                                               const uint32_t *hit_ref, const float *hit_t, PathPtrs P,
                                               RayQ qout, DirectL dl) {
  start_after_previous();
  const uint32_t n = counters[cur];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    counters[4] = 0;   // next bounce's dispenser
    counters[2] = 0;   // the last bounce's shadow rays are traced: the queue
    counters[5] = 0;   // starts empty, as does its dispenser
  }
  uint32_t *count_out = counters + (cur ^ 1u);
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const Strata st = strata_for(jc.S);
  const bool strat = bounce < jc.min_len;

  for (uint32_t wb = warp * 32; wb < n; wb += nwarps * 32) {
    const uint32_t i = wb + lane;
    const bool active = i < n;
    uint32_t path = 0, ps = 0, ref = PREF_END;
    float4 o4 = make_float4(0, 0, 0, 0), d4 = o4;
    float3 thr = f3(0, 0, 0), rad = f3(0, 0, 0);
    float rr_ratio = 1.f, alpha = 1.f;
    bool alive = false;       // path reaches direct lighting
    Isec I;
    BsdfCtx B{nullptr, 1.f, 1.f};
    DevMedium med{1.f, {0, 0, 0}};
    Rng rng{jc.seed_lo, jc.seed_hi, 0, 0};
    uint32_t pixel = 0, sidx = 0;
    if (active) {
      path = qin.path[i];
      o4 = qin.o[i];
      d4 = qin.d[i];
      ref = hit_ref[i];
      float t = hit_t[i];
      ps = P.pstate[path];
      float4 t4 = P.thr[path], r4 = P.rad[path];
      thr = xyz(t4);
      rr_ratio = t4.w;
      rad = xyz(r4);
      alpha = r4.w;
      const uint64_t g = base + path;
      pixel = uint32_t(g / jc.S);
      sidx = uint32_t(g % jc.S);
      rng.path_lo = uint32_t(g);
      rng.path_hi = uint32_t(g >> 32);
      const uint32_t depth = ps_depth(ps);
      const uint32_t mid = depth ? ps_medium(ps, depth - 1) : 0u;
      med = s.media[mid];
      const uint32_t len = ps_len(ps);
      // Volume integrator: attenuation over the ray (render/filter-volume-integ.h:55-68).
      const float t1 = ref == PREF_END ? d4.w : t;
      thr = mul3(thr, medium_transmittance(med, length(xyz(d4)) * (t1 - o4.w)));
      const bool include_emitters = len == 0 || ps_spec(ps) || jc.direct_samples == 0;
      if (ref == PREF_END) {
        if (include_emitters) rad = add(rad, mul3(background(s, xyz(d4)), thr));
        if (len == 0 && rad.x == 0.f && rad.y == 0.f && rad.z == 0.f) alpha = jc.bg_alpha;
      } else {
        I = make_isec(s, ref, xyz(o4), xyz(d4), t);
        const DevMaterial &M = s.mats[I.mat];
        // Glow::Le (material/glow.cc:37-40)
        if (include_emitters && M.type == MAT_GLOW && !I.back) rad = add(rad, mul3(load3(M.color), thr));
        const DevMaterial *bm = bsdf_material(s, I.mat);
        if (bm) {
          B.m = bm;
          B.medium_ior = med.ior;
          // Media::enclosing_medium (material/media.h:76-79)
          B.enclosing_ior = depth >= 2 ? s.media[ps_medium(ps, depth - 2)].ior : 1.f;
          alive = true;
        }
      }
    }

    // Vertices with lights to sample go to the direct-lighting list, with the
    // throughput and path state the continuation below replaces.
    const bool lit = alive && jc.direct_samples != 0u && s.n_lights != 0u;
    const uint32_t dslot = warp_append(counters + 6, lit);
    if (lit) {
      dl.idx[dslot] = i;
      dl.thr[dslot] = make_float4(thr.x, thr.y, thr.z, __uint_as_float(ps));
    }

    // ---- BSDF continuation, roulette, next ray (path-integ.cc:309-403) ----
    bool cont = false;
    float3 next_d = f3(0, 0, 0);
    if (alive) {
      const uint32_t len = ps_len(ps);
      float2 prm = strat ? strat_uv(st, rng, pixel, sidx, dim_of(bounce, K_BSDF)) : rng.uv(dim_of(bounce, K_BSDF));
      BSample bs = bsdf_sample(B, I, prm, B_ALL);
      if (bs.pdf != 0.f && !(bs.val.x == 0.f && bs.val.y == 0.f && bs.val.z == 0.f)) {
        thr = mul3(thr, mul(bs.val, fabsf(I.cos_n(bs.dir)) / bs.pdf));
        bool stop = false;
        if (len > jc.min_len) {
          float p = fminf(intensity(thr) * rr_ratio, 1.f);
          if (rng.u(dim_of(bounce, K_RR)) > p) {
            stop = true;
          } else {
            thr = mul(thr, 1.f / p);
            rr_ratio *= p;
          }
        }
        if (!stop && len != jc.max_len) {
          cont = true;
          next_d = I.nf.from(bs.dir);
          uint32_t nps = (ps & ~0x1ffu) | (len + 1) | ((bs.flags & B_SPECULAR) ? 0x100u : 0u);
          if (bs.flags & B_TRANSMISSIVE) {
            uint32_t mid = s.mats[I.mat].medium_id;
            if (mid && I.back) {
              nps = ps_pop(nps);
            } else if (mid && !ps_push(nps, mid)) {
              atomicOr(counters + 3, 2u);   // a fifth nested medium: the path ends here
              cont = false;
            }
          }
          if (cont) ps = nps;
        }
      }
    }
    uint32_t slot = warp_append(count_out, cont);
    if (cont) {
      // Intersect::recursive_ray (dir) (render/intersect.cc:196-202)
      qout.o[slot] = make_float4(I.pos.x, I.pos.y, I.pos.z, jc.min_trace);
      qout.d[slot] = make_float4(next_d.x, next_d.y, next_d.z, jc.horizon);
      qout.path[slot] = path;
    }
    if (active) {
      P.rad[path] = make_float4(rad.x, rad.y, rad.z, alpha);
      if (cont) {
        P.thr[path] = make_float4(thr.x, thr.y, thr.z, rr_ratio);
        P.pstate[path] = ps;
      }
    }
  }
}

// Direct lighting of the vertices k_shade listed (render/direct-illum.cc:83-255),
// one list entry per thread: the vertex is rebuilt from its queue entry (the
// same arithmetic as in k_shade, so the same bits) and every light sampled.
// Kept out of k_shade so neither body outgrows the instruction cache, and run
// over a compacted list so escaped and absorbed paths leave no idle lanes.
__global__ void __launch_bounds__(128, 6) k_direct(DevScene s, JobConsts jc, uint64_t base, uint32_t bounce,
                                                RayQ qin, uint32_t *counters, const uint32_t *hit_ref,
                                                const float *hit_t, DirectL dl, ShadowQ sq,
                                                unsigned long long *stats) {
  start_after_previous();
  const uint32_t n = counters[6];
  if (blockIdx.x == 0 && threadIdx.x == 0) stats[6] += n;   // DirectIllum::sample_all_lights calls
  uint32_t *count_sq = counters + 2;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const Strata st_direct = strata_for(jc.S * (jc.direct_samples ? jc.direct_samples : 1));
  const Strata st_rand = strata_for(jc.direct_samples ? jc.direct_samples : 1);
  const bool strat = bounce < jc.min_len;
  const float inv_ns = jc.direct_samples ? 1.f / float(jc.direct_samples) : 0.f;

  for (uint32_t wb = warp * 32; wb < n; wb += nwarps * 32) {
    const uint32_t k = wb + lane;
    const bool alive = k < n;
    uint32_t path = 0;
    float3 thr = f3(0, 0, 0);
    Isec I;
    BsdfCtx B{nullptr, 1.f, 1.f};
    DevMedium med{1.f, {0, 0, 0}};
    Rng rng{jc.seed_lo, jc.seed_hi, 0, 0};
    uint32_t pixel = 0, sidx = 0;
    if (alive) {
      const uint32_t i = dl.idx[k];
      const float4 t4 = dl.thr[k];
      thr = xyz(t4);
      const uint32_t ps = __float_as_uint(t4.w);
      path = qin.path[i];
      const float4 o4 = qin.o[i], d4 = qin.d[i];
      const uint64_t g = base + path;
      pixel = uint32_t(g / jc.S);
      sidx = uint32_t(g % jc.S);
      rng.path_lo = uint32_t(g);
      rng.path_hi = uint32_t(g >> 32);
      const uint32_t depth = ps_depth(ps);
      med = s.media[depth ? ps_medium(ps, depth - 1) : 0u];
      I = make_isec(s, hit_ref[i], xyz(o4), xyz(d4), hit_t[i]);
      B.m = bsdf_material(s, I.mat);
      B.medium_ior = med.ior;
      B.enclosing_ior = depth >= 2 ? s.media[ps_medium(ps, depth - 2)].ior : 1.f;
    }

    // ---- direct lighting (render/direct-illum.cc:83-255) ----------------
    // Every lane runs the same loop so that shadow-ray appends stay
    // warp-synchronous; lanes without a live vertex append nothing.
    if (jc.direct_samples) {
      const uint32_t flags = B_ALL & ~B_SPECULAR;
      for (uint32_t l = 0; l < s.n_lights; l++) {
        const DevLight &L = s.lights[l];
        const bool point = is_point_light(L);
        for (uint32_t jn = 0; jn < jc.direct_samples; jn++) {
          bool emit_l = false, emit_b = false;
          float3 c_l = f3(0, 0, 0), c_b = f3(0, 0, 0), dir_l = c_l, dir_b = c_l;
          float dist_l = 0.f, dist_b = 0.f;
          if (alive) {
            const uint32_t kl = K_LIGHT0 + 3 * l;
            float2 pl, pb;
            if (strat) {
              pl = strat_uv(st_direct, rng, pixel, sidx * jc.direct_samples + jn, dim_of(bounce, kl));
              pb = strat_uv(st_direct, rng, pixel, sidx * jc.direct_samples + jn, dim_of(bounce, kl + 1));
            } else {
              pl = strat_uv(st_rand, rng, uint32_t(rng.path_lo ^ (bounce << 24)), jn, dim_of(bounce, kl));
              pb = strat_uv(st_rand, rng, uint32_t(rng.path_lo ^ (bounce << 24)), jn, dim_of(bounce, kl + 1));
            }
            const float extra = rng.u(dim_of(bounce, kl + 2) ^ (jn << 20));
            LSample ls = light_sample(s, L, I, pl, extra);
            if (ls.pdf > 0.f && csum(ls.val) > 0.f) {
              float bpdf;
              float3 bv = bsdf_eval(B, I, ls.dir, flags, bpdf);
              if (csum(bv) > 0.f) {
                float3 c = ls.val;
                float slen = (ls.dist == 0.f ? jc.horizon : ls.dist) - 2.f * jc.min_trace;
                c = mul3(c, medium_transmittance(med, slen));
                if (!point) c = mul(c, mis_weight(ls.pdf, bpdf));
                c = mul3(c, bv);
                c = mul(c, fabsf(I.cos_n(ls.dir)) / ls.pdf);
                c_l = mul(mul3(c, thr), inv_ns);
                dir_l = ls.dir;
                dist_l = ls.dist;
                emit_l = true;
              }
            }
            if (!point) {
              BSample bs = bsdf_sample(B, I, pb, flags);
              if (bs.pdf > 0.f && csum(bs.val) > 0.f) {
                LSample lv = light_eval(s, L, I, bs.dir);
                if (lv.pdf > 0.f && csum(lv.val) > 0.f) {
                  float3 c = lv.val;
                  float slen = (lv.dist == 0.f ? jc.horizon : lv.dist) - 2.f * jc.min_trace;
                  c = mul3(c, medium_transmittance(med, slen));
                  c = mul(c, mis_weight(bs.pdf, lv.pdf));
                  c = mul3(c, bs.val);
                  c = mul(c, fabsf(I.cos_n(bs.dir)) / bs.pdf);
                  c_b = mul(mul3(c, thr), inv_ns);
                  dir_b = bs.dir;
                  dist_b = lv.dist;
                  emit_b = true;
                }
              }
            }
          }
          // Intersect::recursive_ray (dir, max_dist) (render/intersect.cc:211-218)
          uint32_t slot = warp_append(count_sq, emit_l);
          if (emit_l) {
            float3 wd = I.nf.from(dir_l);
            float t1 = (dist_l == 0.f ? jc.horizon : dist_l) - jc.min_trace;
            sq.o[slot] = make_float4(I.pos.x, I.pos.y, I.pos.z, jc.min_trace);
            sq.d[slot] = make_float4(wd.x, wd.y, wd.z, t1);
            sq.c[slot] = make_float4(c_l.x, c_l.y, c_l.z, __uint_as_float(path));
          }
          slot = warp_append(count_sq, emit_b);
          if (emit_b) {
            float3 wd = I.nf.from(dir_b);
            float t1 = (dist_b == 0.f ? jc.horizon : dist_b) - jc.min_trace;
            sq.o[slot] = make_float4(I.pos.x, I.pos.y, I.pos.z, jc.min_trace);
            sq.d[slot] = make_float4(wd.x, wd.y, wd.z, t1);
            sq.c[slot] = make_float4(c_b.x, c_b.y, c_b.z, __uint_as_float(path));
          }
        }
      }
    }

  }
}

// ImageMitchellFilt::mitchell1 with B = C = 1/3, radius 2
// (image/image-mitchell-filt.h:50-65): both cubics by fused Horner steps, which
// round once where the reference's expression rounds three times, and a select.
__device__ __forceinline__ float mitchell1(float x) {
  constexpr double b = 1.0 / 3.0, c = 1.0 / 3.0;
  x = fabsf(x);
  const float inner = fmaf(fmaf(float((12 - 9 * b - 6 * c) / 6), x, float((-18 + 12 * b + 6 * c) / 6)), x * x,
                           float((6 - 2 * b) / 6));
  const float outer = fmaf(fmaf(fmaf(float((-b - 6 * c) / 6), x, float((6 * b + 30 * c) / 6)), x,
                                float((-12 * b - 48 * c) / 6)),
                           x, float((8 * b + 24 * c) / 6));
  return x > 2.f ? 0.f : x > 1.f ? outer : inner;
}

// A splat block's target pixels -- a thread takes ROWS of one column -- and the
// pattern pixels around them.
constexpr int kSplatW = 32, kSplatWarps = 4, kSplatBlock = 32 * kSplatWarps, kHaloW = kSplatW + 4;
constexpr uint32_t kSplatSplit = 16;   // most blocks per tile
constexpr int splat_height(int rows) { return rows * kSplatWarps; }
constexpr int splat_tile(int rows) { return kSplatW * splat_height(rows); }
constexpr int splat_halo(int rows) { return kHaloW * (splat_height(rows) + 4); }

// What a splat block keeps of one sample of each pattern pixel around its tile.
template <int ROWS>
struct SplatSlice {
  float4 col[splat_halo(ROWS)];   // alpha-scaled colour, alpha
  float wlo[splat_halo(ROWS)];    // the least weight the clamp lets pass
  // [d]: weight for the target d - 2 pixels to the left / above
  float wx[5][splat_halo(ROWS)], wy[5][splat_halo(ROWS)];
};

// Its sums (colour, alpha, weight), for the other blocks of its tile.
template <int ROWS>
struct SplatSums {
  double v[5][splat_tile(ROWS)];
};

template <int ROWS>
union SplatShared {
  SplatSlice<ROWS> slice;
  SplatSums<ROWS> sums;
  __device__ SplatShared() {}
};

// Gather the wave's samples into the target pixels they reach
// (ImageFilterConv::add_sample, image/image-filter-conv.h:109-186): every
// sample within the filter's support of a target pixel centre adds
// Tint * w and w, with the negative-lobe clamp (neg_clamp = -0.1).
//
// Every sample reaches 25 pixels, so what a pixel and a sample cost together
// is what counts.  A block takes one sample of each pattern pixel around its
// 32x16 targets (32x4 in small images) at a time: first each sample's colour, its
// five weights per axis and its clamp go to shared memory, then every thread adds
// the products for its four targets (one) -- two products, five fused additions
// and no branch each, with a sample's colour read once for up to four.  The clamp
// scales a product whose smallest component lies below -0.1 to it, which is
// to say that the weight is at least -0.1 / largest component.
//
// A slice's 25 products per target are summed in 32 bits, and the slices in 64:
// all products in one 32-bit sum round worse by the square root of the samples
// (rms of a pixel 3.2e-7 at 16 samples, 6e-7 at 64; 6e-8 so).  The blocks of one
// tile are a cluster and take every SPLIT-th sample each; their sums are
// added in the order of the blocks, so that an image repeats bit for bit.
// (Bound by shared-memory latency at 16 warps per SM; at 20 the 64-bit sums do not
// fit the registers: 1920x1080 at 16 samples 1.64 ms, 2.75 at 20 warps.  Against
// lanes that each evaluated the filter for every pair of sample and target, with
// k_camera and k_resolve: 853x479 pixels at 9 samples 876 -> 208 us, 256x256 at 16
// 162 -> 81, at 64 579 -> 235.  Two or one target per thread in more warps:
// slower by half and by a quarter.)
template <int ROWS, bool CLUSTER>
__global__ void __launch_bounds__(kSplatBlock, 4) k_splat(JobConsts jc, uint64_t base, uint32_t n,
                                                          const float4 *__restrict__ rad,
                                                          const float2 *__restrict__ jit, float4 *accum, float *wsum,
                                                          int ty0, int nrows, uint32_t across, uint32_t split) {
  start_after_previous();
  constexpr int kHalo = splat_halo(ROWS), kTile = splat_tile(ROWS);
  __shared__ SplatShared<ROWS> shared;
  SplatSlice<ROWS> &sl = shared.slice;
  const uint32_t p0 = uint32_t(base / jc.S), p1 = uint32_t((base + n) / jc.S);
  const int lane = threadIdx.x & 31, group = threadIdx.x >> 5;
  const uint32_t tile_id = blockIdx.x / split, rank = blockIdx.x % split;   // tile, block of the tile
  const int x0 = int(tile_id % across) * kSplatW, y0 = ty0 + int(tile_id / across) * splat_height(ROWS);
  double sum[ROWS][5] = {};   // colour, alpha, weight
  // This thread's pattern pixels around the tile, from the wave's first on.
  constexpr int kRounds = (kHalo + kSplatBlock - 1) / kSplatBlock;
  uint32_t pix[kRounds];
#pragma unroll
  for (int q = 0; q < kRounds; q++) {
    const int i = int(threadIdx.x) + q * kSplatBlock;
    const int pc = jc.OX + x0 - 2 + i % kHaloW - jc.PX, pr = jc.OY + y0 - 2 + i / kHaloW - jc.PY;
    const uint32_t pidx = uint32_t(pr) * jc.PW + uint32_t(pc);
    const bool in = i < kHalo && pc >= 0 && pc < int(jc.PW) && pr >= 0 && pr < int(jc.PH) && pidx >= p0 && pidx < p1;
    pix[q] = in ? pidx - p0 : ~0u;
  }
  for (uint32_t k = rank; k < jc.S; k += split) {
    // All loads of the slice first: their latency is paid once.
    bool wild = false;   // a colour that is not finite
    float2 jq[kRounds];
    float4 rq[kRounds];
#pragma unroll
    for (int q = 0; q < kRounds; q++) {
      jq[q] = make_float2(0.f, 0.f);
      rq[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (pix[q] != ~0u) {
        const size_t s = size_t(pix[q]) * jc.S + k;
        jq[q] = jit[s];
        rq[q] = rad[s];
      }
    }
#pragma unroll
    for (int q = 0; q < kRounds; q++) {
      const int i = int(threadIdx.x) + q * kSplatBlock;
      if (i >= kHalo) break;
      const float4 r = rq[q];
      // Tint (radiance, alpha) stores alpha-scaled colour (color/tint.h:45-49)
      const float4 c = make_float4(r.x * r.w, r.y * r.w, r.z * r.w, r.w);
      sl.col[i] = c;
      sl.wlo[i] = -0.1f / fmaxf(fmaxf(c.x, fmaxf(c.y, c.z)), 0.f);   // (-inf where nothing is positive)
      wild |= !(fabsf(c.x) < INFINITY && fabsf(c.y) < INFINITY && fabsf(c.z) < INFINITY && fabsf(c.w) < INFINITY);
      const int px = jc.OX + x0 - 2 + i % kHaloW, py = jc.OY + y0 - 2 + i / kHaloW;
      const float sx = float(px) + jq[q].x, sy = float(py) + jq[q].y;
#pragma unroll
      for (int d = 0; d < 5; d++) {
        sl.wx[d][i] = pix[q] != ~0u ? mitchell1(sx - (float(px - (d - 2)) + 0.5f)) : 0.f;
        sl.wy[d][i] = mitchell1(sy - (float(py - (d - 2)) + 0.5f));
      }
    }
    float4 acc[ROWS];
    float wacc[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
      acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
      wacc[r] = 0.f;
    }
    // Where a colour is not finite, zero weights are skipped (a weight that the clamp
    // brings to zero is not: the sample then counts as NaN, as an infinite one
    // scaled to -0.1 does).
    auto add = [&](auto guard) {
#pragma unroll 1
      for (int dx = 0; dx < 5; dx++) {
#pragma unroll
        for (int h = 0; h < ROWS + 4; h++) {
          const int i = (group * ROWS + h) * kHaloW + lane + dx;
          const float4 c = sl.col[i];
          const float ux = sl.wx[dx][i], lo = sl.wlo[i];
#pragma unroll
          for (int r = 0; r < ROWS; r++) {
            if (h < r || h > r + 4) continue;
            const float product = ux * sl.wy[h - r][i];
            if (guard() && product == 0.f) continue;
            const float w = fmaxf(product, lo);
            acc[r].x = fmaf(c.x, w, acc[r].x);
            acc[r].y = fmaf(c.y, w, acc[r].y);
            acc[r].z = fmaf(c.z, w, acc[r].z);
            acc[r].w = fmaf(c.w, w, acc[r].w);
            wacc[r] += w;
          }
        }
      }
    };
    if (__syncthreads_or(wild)) add(std::true_type{});
    else add(std::false_type{});
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
      sum[r][0] += acc[r].x;
      sum[r][1] += acc[r].y;
      sum[r][2] += acc[r].z;
      sum[r][3] += acc[r].w;
      sum[r][4] += wacc[r];
    }
    __syncthreads();
  }
  auto store = [&](int i, const double *v) {   // add V to target I of the tile
    const int x = x0 + i % kSplatW, y = y0 + i / kSplatW;
    if (x >= int(jc.W) || y >= ty0 + nrows) return;
    const size_t o = size_t(y) * jc.W + size_t(x);
    const float4 a = accum[o];
    accum[o] = make_float4(a.x + float(v[0]), a.y + float(v[1]), a.z + float(v[2]), a.w + float(v[3]));
    wsum[o] += float(v[4]);
  };
  if (!CLUSTER) {
#pragma unroll
    for (int r = 0; r < ROWS; r++) store((group * ROWS + r) * kSplatW + lane, sum[r]);
    return;
  }
#pragma unroll
  for (int r = 0; r < ROWS; r++)
    for (int c = 0; c < 5; c++) shared.sums.v[c][(group * ROWS + r) * kSplatW + lane] = sum[r][c];
  const cg::cluster_group tile = cg::this_cluster();
  tile.sync();
  // Each block adds up its share of the tile's targets.
  const int share = kTile / int(split);
  for (int i = int(threadIdx.x); i < share; i += kSplatBlock) {
    const int t = int(rank) * share + i;
    double v[5] = {};
    for (uint32_t b = 0; b < split; b++) {
      const SplatSums<ROWS> *s = tile.map_shared_rank(&shared.sums, b);
      for (int c = 0; c < 5; c++) v[c] += s->v[c][t];
    }
    store(t, v);
  }
  tile.sync();   // the others read this block's sums
}

template <int ROWS, bool CLUSTER>
void launch_splat_tiles(uint32_t tiles, uint32_t across, uint32_t split, cudaStream_t st, const JobConsts &jc,
                        uint64_t base, uint32_t n, const float4 *rad, const float2 *jit, float4 *accum, float *wsum,
                        int ty0, int nrows) {
  const auto kernel = k_splat<ROWS, CLUSTER>;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = split;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(tiles * split);   // one-dimensional: an image may be millions of pixels wide or high
  cfg.blockDim = dim3(kSplatBlock);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = CLUSTER ? 1 : 0;
  if (split > 8u) cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaLaunchKernelEx(&cfg, kernel, jc, base, n, rad, jit, accum, wsum, ty0, nrows, across, split);
}

// The splat of NROWS target rows from TY0 on.
void launch_splat(const JobConsts &jc, uint64_t base, uint32_t n, const float4 *rad, const float2 *jit,
                  float4 *accum, float *wsum, int ty0, int nrows, cudaStream_t st) {
  const uint32_t across = (jc.W + kSplatW - 1) / kSplatW;
  auto down = [&](int rows) { return (uint32_t(nrows) + splat_height(rows) - 1) / splat_height(rows); };
  auto tiles = [&](int rows) { return uint64_t(across) * down(rows); };
  // Images too small for a block per SM take tiles of a quarter of the height,
  // whose slices take a third of the time (with k_camera and k_resolve: 64x48 at 64
  // samples 45 -> 40 us, 20x20 at 1000 356 -> 216; from one to two blocks per SM the
  // larger tiles are as fast or faster, 200x150 at 4 samples 29 and 33 us).
  const bool small = tiles(4) * (jc.S < kSplatSplit ? jc.S : kSplatSplit) < uint64_t(num_sms());
  const int rows = small ? 1 : 4;
  // Four blocks fit an SM: split the samples while the blocks fill the device no
  // more than three times over (256x256 at 16 samples 77, 81, 81, 98 us for once,
  // twice, three, four times, 640x360 at 16 225, 210, 211, 212), among at most the
  // blocks of a cluster (of 8, the portable size: 64x48 at 64 samples 65 us).
  const uint64_t want = uint64_t(num_sms()) * 4 * 3;
  uint32_t split = 1;
  while (split < kSplatSplit && 2 * split <= jc.S && 2 * split * tiles(rows) <= want) split *= 2;
  const auto launch = small ? (split > 1u ? launch_splat_tiles<1, true> : launch_splat_tiles<1, false>)
                            : (split > 1u ? launch_splat_tiles<4, true> : launch_splat_tiles<4, false>);
  launch(uint32_t(tiles(rows)), across, split, st, jc, base, n, rad, jit, accum, wsum, ty0, nrows);
}

// ImageSampledOutput::set_raw_min_y row flush (image/image-sampled-output.cc:79-123).
__global__ void __launch_bounds__(256) k_resolve(uint32_t npix, const float4 *accum, const float *wsum, float *out) {
  start_after_previous();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += gridDim.x * blockDim.x) {
    float4 a = accum[i];
    float w = wsum[i];
    float r = a.x, g = a.y, b = a.z, al = a.w;
    if (w > 0.f && w != 1.f) {
      float iw = 1.f / w;
      r *= iw; g *= iw; b *= iw; al *= iw;
    }
    al = fminf(fmaxf(al, 0.f), 1.f);
    r = fmaxf(r, 0.f); g = fmaxf(g, 0.f); b = fmaxf(b, 0.f);
    if (al != 0.f && al != 1.f) {
      float ia = 1.f / al;
      r *= ia; g *= ia; b *= ia;
    }
    out[3 * size_t(i)] = r;
    out[3 * size_t(i) + 1] = g;
    out[3 * size_t(i) + 2] = b;
  }
}

template <int STACK, bool COUNT>
void launch_bounce(const DevScene &s, const JobConsts &jc, WaveBuffers &wb, uint64_t base, uint32_t b,
                   uint32_t cur, uint32_t grid128, cudaStream_t st, RenderProfile *prof, ShadowStream *side) {
  RayQ qin{wb.q_o[cur], wb.q_d[cur], wb.q_path[cur]};
  RayQ qout{wb.q_o[cur ^ 1], wb.q_d[cur ^ 1], wb.q_path[cur ^ 1]};
  ShadowQ sq{wb.s_o, wb.s_d, wb.s_c};
  DirectL dl{wb.d_idx, wb.d_thr};
  PathPtrs P{wb.thr, wb.rad, wb.pstate, wb.jit};
  const auto closest = s.pair_lists ? k_trace_closest<STACK, 2, COUNT> : k_trace_closest<STACK, 1, COUNT>;
  const auto shadow = k_trace_shadow<STACK, COUNT>;
  if (prof) prof->begin(st, RenderProfile::CLOSEST);
  launch_after(!prof, closest, resident_grid(closest, kTraceBlock), kTraceBlock, st, s, qin, wb.counters, cur,
               wb.hit_ref, wb.hit_t, wb.stats);
  if (prof) prof->end(st), prof->begin(st, RenderProfile::SHADE);
  // The last bounce's shadow rays add to the radiance that shading reads.
  if (side && b) cudaStreamWaitEvent(st, side->done, 0);
  launch_after(!prof, k_shade, grid128, 128, st, s, jc, base, b, qin, wb.counters, cur, wb.hit_ref, wb.hit_t, P,
               qout, dl);
  launch_after(!prof, k_direct, grid128, 128, st, s, jc, base, b, qin, wb.counters, wb.hit_ref, wb.hit_t, dl, sq,
               wb.stats);
  if (prof) prof->end(st), prof->begin(st, RenderProfile::SHADOW);
  const cudaStream_t on = side ? side->st : st;
  if (side) {
    cudaEventRecord(side->lit, st);
    cudaStreamWaitEvent(on, side->lit, 0);
  }
  shadow<<<resident_grid(shadow, kTraceBlock), kTraceBlock, 0, on>>>(s, sq, wb.counters, wb.rad, wb.stats);
  if (side) cudaEventRecord(side->done, on);
  if (prof) prof->end(st);
}

__global__ void k_cdf_guide(const float *cdf, uint32_t n, uint32_t rows, uint32_t cells, uint32_t *guide) {
  const uint64_t width = uint64_t(cells) + 2u;
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < rows * width;
       i += uint64_t(gridDim.x) * blockDim.x) {
    const uint64_t row = i / width;
    const uint32_t b = uint32_t(i % width);
    guide[i] = b == 0u ? 0u : b > cells ? n : lower_bound_f(cdf + row * n, 0u, n, float(b) / float(cells));
  }
}

}  // namespace

cudaError_t build_cdf_guide(const float *cdf, uint32_t n, uint32_t rows, uint32_t cells, uint32_t *guide,
                            cudaStream_t st) {
  k_cdf_guide<<<uint32_t(num_sms()) * 8, 256, 0, st>>>(cdf, n, rows, cells, guide);
  return cudaGetLastError();
}

cudaError_t RenderProfile::begin(cudaStream_t st, int kind) {
  if (n == cap) {
    uint32_t nc = cap ? 2 * cap : 256;
    Mark *m = new Mark[nc];
    for (uint32_t i = 0; i < n; i++) m[i] = marks[i];
    delete[] marks;
    marks = m;
    cap = nc;
  }
  Mark &mk = marks[n];
  mk.kind = kind;
  cudaError_t e = cudaEventCreate(&mk.a);
  if (e == cudaSuccess) e = cudaEventCreate(&mk.b);
  if (e == cudaSuccess) e = cudaEventRecord(mk.a, st);
  return e;
}

cudaError_t RenderProfile::end(cudaStream_t st) {
  cudaError_t e = cudaEventRecord(marks[n].b, st);
  n++;
  return e;
}

cudaError_t RenderProfile::collect() {
  cudaError_t err = cudaSuccess;
  for (uint32_t i = 0; i < n; i++) {
    float ms = 0.f;
    cudaError_t e = cudaEventElapsedTime(&ms, marks[i].a, marks[i].b);
    if (e != cudaSuccess) err = e;
    this->ms[marks[i].kind] += ms;
    launches[marks[i].kind]++;
    cudaEventDestroy(marks[i].a);
    cudaEventDestroy(marks[i].b);
  }
  n = 0;
  return err;
}

RenderProfile::~RenderProfile() {
  for (uint32_t i = 0; i < n; i++) {
    cudaEventDestroy(marks[i].a);
    cudaEventDestroy(marks[i].b);
  }
  delete[] marks;
}

uint64_t wave_bytes_per_path(uint32_t n_lights) {
  // thr 16 + rad 16 + pstate 4 + 2 queues x 36 + hit 8 + jitter 8
  // + direct-lighting list 20 + shadow queue 48 per entry, 2 entries per light sample
  return 16 + 16 + 4 + 72 + 8 + 8 + 20 + 48ull * 2 * (n_lights ? n_lights : 1);
}

cudaError_t wave_alloc(WaveBuffers &wb, uint64_t cap, uint32_t n_lights) {
  wave_free(wb);
  const uint64_t nl = n_lights ? n_lights : 1;
  size_t bytes = 0;
  auto take = [&](size_t b) {
    size_t off = bytes;
    bytes += (b + 255) & ~size_t(255);
    return off;
  };
  size_t o_thr = take(16 * cap), o_rad = take(16 * cap), o_ps = take(4 * cap);
  size_t o_qo0 = take(16 * cap), o_qd0 = take(16 * cap), o_qp0 = take(4 * cap);
  size_t o_qo1 = take(16 * cap), o_qd1 = take(16 * cap), o_qp1 = take(4 * cap);
  size_t o_href = take(4 * cap), o_ht = take(4 * cap), o_jit = take(8 * cap);
  size_t o_didx = take(4 * cap), o_dthr = take(16 * cap);
  size_t o_so = take(16 * cap * 2 * nl), o_sd = take(16 * cap * 2 * nl), o_sc = take(16 * cap * 2 * nl);
  size_t o_cnt = take(64), o_stats = take(64);
  char *base = nullptr;
  cudaError_t e = device_malloc(reinterpret_cast<void **>(&base), bytes);
  if (e != cudaSuccess) return e;
  wb.block = base;
  wb.bytes = bytes;
  wb.wave_cap = cap;
  wb.n_lights = n_lights;
  wb.thr = reinterpret_cast<float4 *>(base + o_thr);
  wb.rad = reinterpret_cast<float4 *>(base + o_rad);
  wb.pstate = reinterpret_cast<uint32_t *>(base + o_ps);
  wb.q_o[0] = reinterpret_cast<float4 *>(base + o_qo0);
  wb.q_d[0] = reinterpret_cast<float4 *>(base + o_qd0);
  wb.q_path[0] = reinterpret_cast<uint32_t *>(base + o_qp0);
  wb.q_o[1] = reinterpret_cast<float4 *>(base + o_qo1);
  wb.q_d[1] = reinterpret_cast<float4 *>(base + o_qd1);
  wb.q_path[1] = reinterpret_cast<uint32_t *>(base + o_qp1);
  wb.hit_ref = reinterpret_cast<uint32_t *>(base + o_href);
  wb.hit_t = reinterpret_cast<float *>(base + o_ht);
  wb.jit = reinterpret_cast<float2 *>(base + o_jit);
  wb.d_idx = reinterpret_cast<uint32_t *>(base + o_didx);
  wb.d_thr = reinterpret_cast<float4 *>(base + o_dthr);
  wb.s_o = reinterpret_cast<float4 *>(base + o_so);
  wb.s_d = reinterpret_cast<float4 *>(base + o_sd);
  wb.s_c = reinterpret_cast<float4 *>(base + o_sc);
  wb.counters = reinterpret_cast<uint32_t *>(base + o_cnt);
  wb.stats = reinterpret_cast<unsigned long long *>(base + o_stats);
  return cudaSuccess;
}

void wave_free(WaveBuffers &wb) {
  if (wb.block) cudaFree(wb.block);
  wb = WaveBuffers{};
}

void check_window(const SnogRenderParams &p, const SnogRenderWindow &w) {
  if (w.pat_width == 0 || w.pat_height == 0 || w.out_width == 0 || w.out_height == 0)
    throw Error{SNOG_EINVAL, "render window: empty pattern or output"};
  if (w.out_width > 65536 || w.out_height > 65536 || w.pat_width > 65540 || w.pat_height > 65540)
    throw Error{SNOG_EINVAL, "render window too large"};
  const int64_t lim = int64_t(1) << 20;
  if (w.pat_x < -lim || w.pat_x > lim || w.pat_y < -lim || w.pat_y > lim || w.out_x < -lim || w.out_x > lim ||
      w.out_y < -lim || w.out_y > lim)
    throw Error{SNOG_EINVAL, "render window offsets out of range"};
  if (uint64_t(w.pat_width) * w.pat_height >= (1ull << 32)) throw Error{SNOG_EINVAL, "render pattern too large"};
  if (uint64_t(w.pat_width) * w.pat_height * p.spp >= (1ull << 40))
    throw Error{SNOG_EINVAL, "too many paths in one job"};
}

JobConsts make_job(const DevScene &s, const SnogCamera &cam, const SnogRenderParams &p,
                   const SnogRenderWindow *win) {
  JobConsts jc;
  std::memset(&jc, 0, sizeof jc);
  jc.FW = p.width;
  jc.FH = p.height;
  if (win) {
    jc.W = win->out_width;
    jc.H = win->out_height;
    jc.OX = win->out_x;
    jc.OY = win->out_y;
    jc.PW = win->pat_width;
    jc.PH = win->pat_height;
    jc.PX = win->pat_x;
    jc.PY = win->pat_y;
  } else {
    jc.W = p.width;
    jc.H = p.height;
    jc.OX = jc.OY = 0;
    jc.PW = p.width + 4;
    jc.PH = p.height + 4;
    jc.PX = jc.PY = -2;
  }
  jc.S = p.spp;
  jc.min_len = p.min_path_len;
  jc.max_len = p.max_path_len;
  jc.direct_samples = p.direct_samples;
  jc.min_trace = p.min_trace;
  jc.bg_alpha = p.bg_alpha;
  jc.horizon = s.horizon;
  // (scene.bbox () + camera.pos).diameter () (render-mgr/renderer.cc:54)
  float lo[3], hi[3];
  for (int k = 0; k < 3; k++) {
    lo[k] = s.bbox_min[k] < cam.pos[k] ? s.bbox_min[k] : cam.pos[k];
    hi[k] = s.bbox_max[k] > cam.pos[k] ? s.bbox_max[k] : cam.pos[k];
  }
  float ex = hi[0] - lo[0], ey = hi[1] - lo[1], ez = hi[2] - lo[2];
  jc.max_trace = std::sqrt(ex * ex + ey * ey + ez * ez);
  for (int k = 0; k < 3; k++) {
    jc.cam_pos[k] = cam.pos[k];
    jc.cam_fwd[k] = cam.forward[k];
    jc.cam_right[k] = cam.right[k];
    jc.cam_up[k] = cam.up[k];
  }
  jc.tan_x = cam.tan_half_fov_x;
  jc.tan_y = cam.tan_half_fov_y;
  jc.seed_lo = uint32_t(p.seed) * 2654435761u + 0x1234567u;
  jc.seed_hi = uint32_t(p.seed >> 32) ^ 0x9e3779b9u;
  jc.integ = p.integrator;
  return jc;
}

cudaError_t ShadowStream::create() {
  cudaError_t e = cudaSuccess;
  if (!lit) e = cudaEventCreateWithFlags(&lit, cudaEventDisableTiming);
  if (e == cudaSuccess && !done) e = cudaEventCreateWithFlags(&done, cudaEventDisableTiming);
  if (e == cudaSuccess && !st) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  return e;
}

cudaError_t render_job(const DevScene &s, const JobConsts &jc, WaveBuffers &wb, float4 *accum, float *wsum,
                       float *out_rgb, cudaStream_t st, uint32_t *waves, uint32_t *launches,
                       RenderProfile *prof, bool count, ShadowStream *side) {
  if (prof) side = nullptr;   // the profile's events bracket launches of one stream
  const uint64_t npix = uint64_t(jc.W) * jc.H;
  cudaError_t e = cudaMemsetAsync(accum, 0, npix * sizeof(float4), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(wsum, 0, npix * sizeof(float), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(wb.stats, 0, 64, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(wb.counters, 0, 64, st);
  if (e == cudaSuccess && side) e = side->create();
  if (e != cudaSuccess) return e;
  const int sms = num_sms();
  const uint32_t grid128 = uint32_t(sms) * 12, grid256 = uint32_t(sms) * 8;
  const uint64_t total = job_total(jc);
  const uint64_t wave_paths = (wb.wave_cap / jc.S) * jc.S;
  if (wave_paths == 0) return cudaErrorInvalidValue;
  const int sc = stack_class_for_depth(s.max_depth);
  uint32_t nl = 0;
  for (uint64_t base = 0; base < total; base += wave_paths) {
    const uint32_t n = uint32_t(total - base < wave_paths ? total - base : wave_paths);
    PathPtrs P{wb.thr, wb.rad, wb.pstate, wb.jit};
    RayQ q0{wb.q_o[0], wb.q_d[0], wb.q_path[0]};
    if (prof) prof->begin(st, RenderProfile::OTHER);
    k_camera<<<grid256, 256, 0, st>>>(jc, base, n, P, q0, wb.counters);
    if (prof) prof->end(st);
    nl++;
    for (uint32_t b = 0; b <= jc.max_len; b++) {
      const uint32_t cur = b & 1u;
      auto bounce = [&](auto stack) {
        if (prof || count) launch_bounce<stack(), true>(s, jc, wb, base, b, cur, grid128, st, prof, side);
        else launch_bounce<stack(), false>(s, jc, wb, base, b, cur, grid128, st, prof, side);
      };
      switch (sc) {
        case 32: bounce(std::integral_constant<int, 32>{}); break;
        case 64: bounce(std::integral_constant<int, 64>{}); break;
        case 128: bounce(std::integral_constant<int, 128>{}); break;
        case 256: bounce(std::integral_constant<int, 256>{}); break;
        default: return cudaErrorInvalidValue;
      }
      nl += 4;
    }
    if (side && (e = cudaStreamWaitEvent(st, side->done, 0)) != cudaSuccess) return e;
    // Output rows reached by this wave's pattern rows (a sample reaches
    // the film rows within 2 of its own).
    const uint32_t p0 = uint32_t(base / jc.S), p1 = uint32_t((base + n) / jc.S);
    const int r0 = int(p0 / jc.PW), r1 = int((p1 - 1) / jc.PW);
    const int a0 = jc.PY + r0 - jc.OY - 2, a1 = jc.PY + r1 - jc.OY + 2;
    const int ty0 = a0 < 0 ? 0 : a0, ty1 = a1 > int(jc.H) - 1 ? int(jc.H) - 1 : a1;
    if (ty1 >= ty0) {
      if (prof) prof->begin(st, RenderProfile::OTHER);
      launch_splat(jc, base, n, wb.rad, P.jit, accum, wsum, ty0, ty1 - ty0 + 1, st);
      if (prof) prof->end(st);
      nl++;
    }
    if (waves) (*waves)++;
  }
  if (prof) prof->begin(st, RenderProfile::OTHER);
  launch_after(!prof, k_resolve, grid256, 256, st, uint32_t(npix), accum, wsum, out_rgb);
  if (prof) prof->end(st);
  nl++;
  if (launches) *launches += nl;
  return cudaGetLastError();
}

}  // namespace snog

namespace snog {

cudaError_t splat_job(const JobConsts &jc, const float4 *rad, const float2 *jit, uint64_t total, float4 *accum,
                      float *wsum, float *out_rgb, cudaStream_t st) {
  const uint64_t npix = uint64_t(jc.W) * jc.H;
  cudaError_t e = cudaMemsetAsync(accum, 0, npix * sizeof(float4), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(wsum, 0, npix * sizeof(float), st);
  if (e != cudaSuccess) return e;
  const uint32_t grid256 = uint32_t(num_sms()) * 8;
  launch_splat(jc, 0, uint32_t(total), rad, jit, accum, wsum, 0, int(jc.H), st);
  launch_after(true, k_resolve, grid256, 256, st, uint32_t(npix), accum, wsum, out_rgb);
  return cudaGetLastError();
}

}  // namespace snog
