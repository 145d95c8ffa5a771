// Device code of the wave kernels shared by the translation units that
// instantiate them (kernels.cu: surfaces; wave_media.cu: volume scattering;
// wave_adjoint.cu: the path-replay adjoint). Each unit holds its own copy of
// the constant-memory scene table (dev_constants.cuh), which every upload
// writes.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "dev_sampler.cuh"
#include "dev_shade.cuh"
#include <cooperative_groups.h>

#include "dev_traverse.cuh"
#include "dev_volume.cuh"
#include "kernels.h"

namespace ym {

namespace cg = cooperative_groups;



// ---------------------------------------------------------------- paths ---

__device__ __forceinline__ void store_path(const PathPool& P, uint32_t i, vec3 o, vec3 d, vec3 tp, vec3 rad, uint32_t pixel,
                                           uint32_t flags, uint32_t last_inst, uint32_t last_tri, const PathSampler& hs,
                                           uint32_t path_id) {
  P.path_id[i] = path_id;
  P.ray_o[i] = make_float4(o.x, o.y, o.z, 0.0f);
  P.ray_d[i] = make_float4(d.x, d.y, d.z, 0.0f);
  P.throughput[i] = make_float4(tp.x, tp.y, tp.z, 0.0f);
  P.radiance[i] = make_float4(rad.x, rad.y, rad.z, 0.0f);
  P.pixel_flags[i] = make_uint2(pixel, flags);
  P.last_hit[i] = make_uint2(last_inst, last_tri);
  P.sampler[i] = make_uint4((uint32_t)hs.index, (uint32_t)(hs.index >> 32), hs.dim, hs.aux);
}

// Per-pixel accumulation (the reference adds the four channels with four
// float atomics, src/Shading.cu:1859-1862): one vector atomic that adds each
// channel atomically.
__device__ __forceinline__ void accumulate_pixel(float4* image, uint32_t pixel, vec3 light, float inv_spp) {
  atomicAdd(image + pixel, make_float4(light.x * inv_spp, light.y * inv_spp, light.z * inv_spp, inv_spp));
}

// A path ends: its radiance into its pixel, and (differentiable renders)
// into the job's per-path record.
__device__ __forceinline__ void finish_path(const JobDesc& J, uint32_t pixel, uint32_t path_id, vec3 rad,
                                            float inv_spp) {
  accumulate_pixel(J.image, pixel, rad, inv_spp);
  // added, not stored: deferred shadow rays of the path add to the same record
  if (J.path_radiance) atomicAdd(J.path_radiance + path_id, make_float4(rad.x, rad.y, rad.z, 0.0f));
}

template <bool kAdj>
__device__ __forceinline__ void end_path(const JobDesc& J, uint32_t pixel, uint32_t path_id, vec3 rad, float inv_spp) {
  if (!kAdj) finish_path(J, pixel, path_id, rad, inv_spp);
}

// Warp-aggregated slot allocation in the output pool.
__device__ __forceinline__ uint32_t warp_append(uint32_t* counter, bool want) {
  const uint32_t mask = __ballot_sync(0xFFFFFFFFu, want);
  if (!want) return kEmpty;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(mask) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
  base = __shfl_sync(mask, base, leader);
  return base + (uint32_t)__popc(mask & ((1u << lane) - 1u));
}

__device__ __forceinline__ uint32_t flags_pack(int depth, bool never_scatter, bool camera_ray, uint32_t job) {
  return (uint32_t)depth | (never_scatter ? kFlagNeverScatter : 0u) | (camera_ray ? kFlagCameraRay : 0u) |
         (job << kFlagJobShift);
}

// ------------------------------------------------------------ generate ---

// The job holding path g of the batch's path space (binary search; jobs are
// in path order).
__device__ __forceinline__ uint32_t find_job(const JobDesc* __restrict__ jobs, uint32_t n_jobs, unsigned long long g) {
  uint32_t lo = 0, hi = n_jobs;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (jobs[mid].path_begin <= g) lo = mid;
    else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ void generate_path(const PathPool& P, uint32_t base, uint32_t tid,
                                              unsigned long long path_cursor, const JobDesc* __restrict__ jobs,
                                              uint32_t n_jobs);

// The wave's continuing rays, when there are enough of them to be grouped (else 0).
__device__ __forceinline__ uint32_t grouped_rays(const WaveControl* ctl) {
  return ctl->live >= kMinGroupedRays ? ctl->live : 0u;
}

// -------------------------------------------------------------- extend ---

// Counts this lane's hit under its shading bucket (kBucketNone: no hit), one
// atomic per bucket present in the warp, and the warp's hits in hit_count.
__device__ __forceinline__ void file_bucket(WaveCounters* counters, uint32_t bucket) {
  const bool has = bucket != kBucketNone;
  const uint32_t act = __ballot_sync(0xFFFFFFFFu, has);
  const uint32_t hits = __ballot_sync(0xFFFFFFFFu, has && bucket != kBucketMiss);
  const int lane = threadIdx.x & 31;
  if (lane == 0 && hits) atomicAdd(&counters->hit_count, (uint32_t)__popc(hits));
  if (!has) return;
  const uint32_t peers = __match_any_sync(act, bucket);
  if (lane == __ffs(peers) - 1) atomicAdd(&counters->bucket_count[bucket], (uint32_t)__popc(peers));
}

// Walks the wave's paths warp by warp (every lane of a warp takes part in each
// iteration, for the warp-collective bucket filing); the wave's size comes
// from the wave-control block, so any grid works (launched with one thread
// per pool slot, each thread takes at most one path).
//
// kF: the batch's scene features (kFeatSpheres, kFeatGrids); a batch without
// spheres or grids runs the instantiation without their code.
//
// kAdj (with kVol): the adjoint pass; each free-flight segment also adds its
// density-grid gradient terms to grid_grads, weighted by dLoss/dI times the
// radiance the path gathers after the segment (its recorded total minus what
// it gathered so far).
//
// ray_order (surfaces, optional): the continuing slots [0, live) in the order
// to trace them (k_ray_scatter: grouped by origin cell and direction), so that
// neighbouring lanes take similar walks; the new camera paths keep slot order.
//
// Launched with kTraceBlock threads by default, or any block size up to
// kMaxTraceBlock (YMRT_OPT_TRACE_BLOCK, tuned by ymrt_b200.autotune); the
// traversal stacks are in dynamic shared memory (traversal_shared_bytes).
// Registers a thread: 96, five resident 128-thread blocks per SM (instanced
// 1080p 64 spp, closest hits 97.8 ms at 128 registers and 86.7 at 96, 107 at
// 80; Cornell 256x256 16 spp 1.07 and 0.97; media with fBm 47.7 and 46.4). The
// media instantiation with every texture node spills at 96: 128 (smoke grid
// 33.2 and 34.2 ms).
template <bool kVol, uint32_t kF>
constexpr uint32_t extend_registers() {
  return kVol && (kF & (kFeatGrids | kFeatTextures)) ? 128 : 96;
}

template <bool kVol, uint32_t kF, bool kAdj = false>
__global__ void __maxnreg__((extend_registers<kVol, kF>())) k_extend(PathPool P, const WaveControl* __restrict__ ctl, HitPool H,
                                                           const JobDesc* __restrict__ jobs, WaveCounters* counters,
                                                           float* grid_grads = nullptr, uint32_t grid_tex = kEmpty,
                                                           const uint32_t* __restrict__ ray_order = nullptr) {
  YM_TRAVERSAL_SHARED_DYNAMIC(s_stack);
  const uint32_t count = ctl->count;
  const uint32_t live = ray_order ? grouped_rays(ctl) : 0u;
  uint32_t tests = 0, nodes = 0, n_rays = 0;
  bool overflow = false;
  for (uint32_t warp_base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); warp_base < count;
       warp_base += gridDim.x * blockDim.x) {
  const uint32_t j = warp_base + (threadIdx.x & 31u);
  uint32_t i = j;
  if (j < live) {
    i = ray_order[j];
    if (i >= live) {  // not a continuing slot: the order is broken (never expected)
      atomicOr(&counters->errors, (uint32_t)kDevErrQueue);
      i = j;
    }
  }
  bool active = j < count;
  uint2 pf = active ? P.pixel_flags[i] : make_uint2(kEmpty, kFlagDead);
  if (active && (pf.y & kFlagDead)) active = false;
  uint32_t bucket = kBucketNone;
  if (active) {
    const JobDesc& J = jobs[pf.y >> kFlagJobShift];
    const uint32_t slot = J.scene_slot;
    const DeviceScene& S = c_scenes[slot];
    const float4 o4 = P.ray_o[i], d4 = P.ray_d[i];
    (void)J;
    const vec3 o(o4.x, o4.y, o4.z), d(d4.x, d4.y, d4.z);
    const uint2 lh = P.last_hit[i];
    TraversalStack st;
    st.bind(s_stack);
    ClosestHit ch;
    bool hit = trace_closest_impl<(kF & kFeatSpheres) != 0, false>(slot, st, o, d, kTMax, lh.x, lh.y, &ch, &tests, &nodes);
    overflow = overflow || st.overflow;
    bool volume_hit = false;
    vec3 vol_pos(0.0f);
    if (kVol && J.setting.enable_volume_scattering) {
      // volume free flight before the surface (src/Shading.cu:1828-1853)
      RayTransfer rt;
      rt.record_count = P.transfer_count[i];
      rt.max_priority_record_index = -1;
      if (rt.record_count > 0) rt = P.transfer[i];
      const uint4 s4 = P.sampler[i];
      PathSampler hs{(uint64_t)s4.x | ((uint64_t)s4.y << 32), s4.z, s4.w};
      int vidx[kMaxBoundaryRecord];
      const int n = current_volumes(rt, S.volume_count, vidx);
      vec3 trw(1.0f);
      float dist = 0.0f;
      float vw[kMaxBoundaryRecord];
      bool hv;
      if constexpr (kAdj) {
        MediumAdj am{vec3(0.0f), grid_tex, grid_grads};
        if (grid_grads && J.dloss) {
          const float4 dl = J.dloss[pf.x], lt = J.path_radiance[P.path_id[i]], r4 = P.radiance[i];
          const float inv_spp = 1.0f / gmax(J.setting.ssp, 1);
          am.scale = vec3(dl.x, dl.y, dl.z) * inv_spp * (vec3(lt.x, lt.y, lt.z) - vec3(r4.x, r4.y, r4.z));
        }
        hv = sample_volume_scattering<kF, true>(S, o, d, n, vidx, hit ? ch.t : kTMax, &trw, &dist, vw, hs,
                                                &counters->errors, &am);
      } else {
        hv = sample_volume_scattering<kF>(S, o, d, n, vidx, hit ? ch.t : kTMax, &trw, &dist, vw, hs,
                                          &counters->errors);
      }
      const float4 t4 = P.throughput[i];
      vec3 tp(t4.x, t4.y, t4.z);
      tp *= trw;
      P.throughput[i] = make_float4(tp.x, tp.y, tp.z, 0.0f);
      P.sampler[i] = make_uint4((uint32_t)hs.index, (uint32_t)(hs.index >> 32), hs.dim, hs.aux);
      if (hv) {
        volume_hit = true;
        vol_pos = o + d * dist;
        for (int k = 0; k < n; ++k) H.vol_w[(size_t)i * kMaxBoundaryRecord + k] = vw[k];
        if (!hit) {
          ch.inst = kEmpty;
          ch.tri = kEmpty;
          ch.back = 0;
          ch.t = kTMax;
          ch.nearby_count = 0;
        }
      }
      hit = hit || hv;
    }
    if (!hit) {
      // a miss: listed in its own bucket; k_shade adds the background and
      // ends the path (the miss branch of Ray_trace_path_tracing,
      // src/Shading.cu:1855-1864)
      H.ids[i] = make_uint4(kEmpty, kEmpty, 0u, 0u);
      bucket = kBucketMiss;
    } else {
      if (volume_hit) H.bary_t[i] = make_float4(vol_pos.x, vol_pos.y, vol_pos.z, ch.t);
      else H.bary_t[i] = make_float4(ch.b0, ch.b1, ch.b2, ch.t);
      uint32_t nearby_word = (uint32_t)ch.nearby_count;
      if (!(ch.nearby_count == 1 && ch.nearby[0].prim == ch.inst && ch.nearby[0].t == ch.t &&
            ch.nearby[0].back == ch.back)) {
        for (int k = 0; k < ch.nearby_count; ++k)
          H.nearby[(size_t)i * kMaxNearby + k] =
              make_uint4(ch.nearby[k].prim, __float_as_uint(ch.nearby[k].t), (uint32_t)ch.nearby[k].back, 0u);
        nearby_word |= kNearbyExplicit;
      }
      H.ids[i] = make_uint4(ch.inst, ch.tri, (uint32_t)ch.back | (volume_hit ? 2u : 0u), nearby_word);
      bucket = volume_hit ? kBucketVolume : (uint32_t)S.inst_bucket[ch.inst];
    }
  }
  if (j < count) H.bucket[i] = (uint8_t)bucket;
  file_bucket(counters, bucket);
  n_rays += __popc(__ballot_sync(0xFFFFFFFFu, active));
  }
  // counters: one atomic per warp
  uint32_t t_sum = tests, n_sum = nodes;
  for (int off = 16; off > 0; off >>= 1) {
    t_sum += __shfl_down_sync(0xFFFFFFFFu, t_sum, off);
    n_sum += __shfl_down_sync(0xFFFFFFFFu, n_sum, off);
  }
  if ((threadIdx.x & 31) == 0) {
    if (n_rays) atomicAdd(&counters->extension_rays, (unsigned long long)n_rays);
    if (t_sum) atomicAdd(&counters->tri_tests, (unsigned long long)t_sum);
    if (n_sum) atomicAdd(&counters->node_visits, (unsigned long long)n_sum);
  }
  if (overflow) atomicOr(&counters->errors, (uint32_t)kDevErrStack);
}

// --------------------------------------------------------------- shade ---

__device__ __forceinline__ int find_record(const RayTransfer& rt, uint32_t prim) {
  for (int r = rt.record_count - 1; r >= 0; --r)
    if (rt.records[r].prim_idx == prim) return r;
  return -1;
}
__device__ __forceinline__ int find_max_priority_record(const RayTransfer& rt) {
  if (rt.record_count == 0) return -1;
  uint32_t mp = rt.records[0].ior_priority;
  int mi = 0;
  for (int r = 1; r < rt.record_count; ++r)
    if (rt.records[r].ior_priority >= mp) {
      mp = rt.records[r].ior_priority;
      mi = r;
    }
  return mi;
}
// RayTransfer::PushRecord / PopRecord (src/Ray.h:179-224).
__device__ __forceinline__ bool push_record(RayTransfer& rt, uint32_t prim, float ior, uint32_t prio, int vol,
                                            uint32_t* errors) {
  if (rt.record_count == kMaxBoundaryRecord) {
    atomicOr(errors, (uint32_t)kDevErrStack);
    return false;
  }
  BoundaryRecord& r = rt.records[rt.record_count];
  r.prim_idx = prim;
  r.ior = ior;
  r.ior_priority = prio;
  r.vol_idx = vol;
  ++rt.record_count;
  if (rt.record_count == 1) {
    rt.max_priority_record_index = 0;
    return true;
  }
  if (prio >= rt.records[rt.max_priority_record_index].ior_priority) rt.max_priority_record_index = rt.record_count - 1;
  return true;
}
__device__ __forceinline__ void pop_record(RayTransfer& rt, int idx) {
  if (rt.record_count == 0 || !(idx >= 0 && idx < rt.record_count)) return;
  for (int k = idx + 1; k < rt.record_count; ++k) rt.records[k - 1] = rt.records[k];
  --rt.record_count;
  rt.max_priority_record_index = find_max_priority_record(rt);
}
// Material::FetchIOR (src/Material.h:262-278); a light material reports ior 1
// and priority 0.
__device__ __forceinline__ float fetch_ior(const Material& m, uint32_t* prio) {
  if (m.material_type == kDefaultMtl) {
    *prio = m.default_mtl.ior_priority;
    return m.default_mtl.ior_n;
  }
  *prio = 0;
  return 1.0f;
}
// BoundaryTransitionBunch (src/ShadingUtilities.cuh:954-990).
__device__ __forceinline__ void boundary_transition(const DeviceScene& S, RayTransfer& rt, const NearbyHit* nb, int n,
                                                    uint32_t* errors) {
  for (int k = 0; k < n; ++k) {
    if (nb[k].back) continue;
    const Instance inst = S.instances[nb[k].prim];
    uint32_t prio;
    const float ior = fetch_ior(S.materials[inst.material_idx], &prio);
    if (find_record(rt, nb[k].prim) == -1) push_record(rt, nb[k].prim, ior, prio, inst.inner_volume_idx, errors);
  }
  for (int k = 0; k < n; ++k) {
    if (!nb[k].back) continue;
    const int r = find_record(rt, nb[k].prim);
    if (r != -1) pop_record(rt, r);
  }
}
// RayTransfer::GetRayIOR / GetExIOR (src/Ray.h:239-258).
__device__ __forceinline__ float ray_ior(const RayTransfer& rt) {
  return rt.record_count > 0 ? rt.records[rt.max_priority_record_index].ior : 1.0f;
}
__device__ __forceinline__ float ex_ior(const RayTransfer& rt, uint32_t hit_prim) {
  uint32_t mp = 0;
  int mi = -1;
  for (int r = 0; r < rt.record_count; ++r) {
    if (rt.records[r].prim_idx == hit_prim) continue;
    if (rt.records[r].ior_priority >= mp) {
      mp = rt.records[r].ior_priority;
      mi = r;
    }
  }
  return mi == -1 ? 1.0f : rt.records[mi].ior;
}

// Closest boundary crossing of a ray (TraceVolume, src/ShadingUtilities.cuh:434-561)
// and the transmittance along a shadow ray through every medium it crosses
// (TraceTr, src/VolumeEval.cuh:420-468). `rt` is the shadow ray's own copy of
// the nested-media stack; `o`/`d`/`tmax` and the last hit are the shadow ray.
template <uint32_t kF, bool kAdj = false>
__device__ __noinline__ vec3 trace_tr(uint32_t scene, TraversalStack& st, vec3 o, vec3 d, float tmax,
                                      uint32_t last_inst, uint32_t last_tri, RayTransfer& rt, PathSampler& hs,
                                      uint32_t* errors, uint32_t* tests, uint32_t* nodes,
                                      const MediumAdj* am = nullptr) {
  const DeviceScene& S = c_scenes[scene];
  if (S.volume_count == 0) return vec3(1.0f);
  vec3 tr(1.0f);
  const float max_d = tmax;
  float traced = kTMin;
  float ray_t = tmax;
  int guard = 0;
  while (traced < max_d) {
    if (++guard > 4 * kMaxRayDepth) {
      atomicOr(errors, (uint32_t)kDevErrIter);
      note_bound(kBoundShadowCrossings, (uint32_t)(guard - 1), o, d, max_d - traced, last_inst, last_tri, &rt);
      break;
    }
    ClosestHit ch;
    const bool hit = trace_closest_impl<(kF & kFeatSpheres) != 0, true>(scene, st, o, d, ray_t, last_inst, last_tri, &ch, tests, nodes);
    tr *= eval_tr<kF, kAdj>(S, o, d, rt, hit ? ch.t : gmax(max_d - traced, 0.0f), hs, errors, am);
    if (!hit) break;
    traced += ch.t;
    vec3 hp, herr, hng;
    fetch_geometry_normal<kF>(S, ch.inst, ch.tri, vec3(ch.b0, ch.b1, ch.b2), &hp, &herr, &hng);
    boundary_transition(S, rt, ch.nearby, ch.nearby_count, errors);
    o = offset_ray_origin(hp, herr, d, hng);
    d = normalize(d);
    last_inst = ch.inst;
    last_tri = ch.tri;
    ray_t = kTMax;
  }
  return tr;
}

// A direction toward a light: radiance and pdf, and (shape lights) the point
// reached on it with its error and geometric normal.
struct LightSample {
  vec3 dir, pos, err, ng, Li;
  float pdf;
};

// DistantLight::SampleLi / EvalLi (src/Light.h:343-386).
__device__ __forceinline__ void distant_sample_li(const DeviceScene& S, const DistantLight& L, float u0, float u1, vec3* wi,
                                                  vec3* Li, float* pdf) {
  const mat4& otw = S.transforms[L.transform_idx];
  const float cone = 2.0f * kPi * (1.0f - L.cos_theta_max);
  vec3 cs(0.0f);
  if (cone < 1E-10f) {
    cs = vec3(0.0f, 1.0f, 0.0f);
  } else {
    const float c = (1.0f - u0) + u0 * L.cos_theta_max;
    const float sn = sqrtf(gmax(0.0f, 1.0f - c * c));
    const float phi = u1 * 2.0f * kPi;
    cs = vec3(cosf(phi) * sn, sinf(phi) * sn, c);
    cs = vec3(cs.x, cs.z, cs.y);
  }
  *wi = -normalize(transform_vector(otw, cs));
  *pdf = 1.0f / gmax(cone, 1E-10f);
  *Li = L.light_color * L.intensity;
}
__device__ __forceinline__ vec3 distant_eval_li(const DeviceScene& S, const DistantLight& L, vec3 wi, float* pdf) {
  const vec3 lwi = transform_vector(S.i_transforms[L.transform_idx], wi);
  const float c = -lwi.y;
  if (c < L.cos_theta_max) {
    *pdf = 0.0f;
    return vec3(0.0f);
  }
  const float cone = 2.0f * kPi * (1.0f - L.cos_theta_max);
  *pdf = 1.0f / cone;
  return L.light_color * L.intensity * (*pdf);
}

// ------------------------------------------------- path-replay adjoint ---
//
// Gradients of an image loss with respect to each material's diffuse albedo
// (rgb) and roughness (alpha_x and alpha_y together), by path replay: the
// adjoint pass re-traces every path with its own sampler (same directions as
// the forward pass, which recorded each path's radiance), and at every
// surface vertex adds, for each parameter p of the vertex's material,
//   dLoss/dI . ( tp * dNEE/dp  +  L_after * (df/dp) / f )
// where L_after is the radiance the path gathers after the vertex (its
// recorded total minus what it gathered so far). Sampling and MIS weights are
// held fixed (detached), so only BSDF values are differentiated; df/dp is the
// central difference of the closed-form layered BSDF at the vertex's fixed
// directions.

constexpr int kMaxGradMaterials = 64;     // materials with shared-memory gradient slots per block
constexpr float kParamStep = 1e-3f;       // central-difference step of df/dp

struct AdjCtx {
  vec3 weight;                            // dLoss/dI (per path) * throughput: the weight of this vertex's NEE
  float g[kGradParams];                   // accumulated dLoss/dp
  // Per-lobe derivative data of the vertex's layered BSDF (channel-diagonal
  // in albedo: each channel's albedo moves only that channel of f):
  vec3 lambert_coeff;                     // the diffuse lobe's colour per unit albedo
  vec3 metal_n[2], metal_k[2];            // the conductor's complex IOR at albedo +-h
  float ax[2], ay[2];                     // the microfacet lobes' alpha at roughness +-h
};

// m: the material's parameters as read at the vertex. A parameter a texture
// supplies does not depend on the material's constant: its derivative is 0.
static __device__ __noinline__ void init_adjoint(AdjCtx& a, const LayeredBsdf& B, const DefaultMtl& m) {
  const bool albedo_const = m.diffuse_albedo_tex == kEmpty;
  const float ha = albedo_const ? kParamStep : 0.0f;
  const float hx = m.alpha_x_tex == kEmpty ? kParamStep : 0.0f;
  const float hy = m.alpha_y_tex == kEmpty ? kParamStep : 0.0f;
  a.lambert_coeff = vec3(0.0f);
  for (int i = 0; i < B.count; ++i)
    if (B.lobe[i].role == kRoleDiffuse && albedo_const)
      for (int c = 0; c < 3; ++c)
        a.lambert_coeff[c] = m.diffuse_albedo[c] > 0.0f ? B.lobe[i].albedo[c] / m.diffuse_albedo[c] : 0.0f;
  edge_tint_to_conductor(m.diffuse_albedo + vec3(ha), m.specular_albedo, &a.metal_n[0], &a.metal_k[0]);
  edge_tint_to_conductor(m.diffuse_albedo - vec3(ha), m.specular_albedo, &a.metal_n[1], &a.metal_k[1]);
  a.ax[0] = sqr(gclamp(m.alpha_x + hx, 0.001f, 0.999f));
  a.ax[1] = sqr(gclamp(m.alpha_x - hx, 0.001f, 0.999f));
  a.ay[0] = sqr(gclamp(m.alpha_y + hy, 0.001f, 0.999f));
  a.ay[1] = sqr(gclamp(m.alpha_y - hy, 0.001f, 0.999f));
  for (int k = 0; k < kGradParams; ++k) a.g[k] = 0.0f;
}

// Adds weight . (c * (df/dp) / f) for every parameter at the fixed
// directions (wo, wi) in the frame of B. df/d(albedo): exact for the diffuse
// lobe (linear), a central difference of the conductor's Fresnel term
// through its edge-tint IOR; df/d(roughness): central differences of the
// metal, specular and transmission lobes (the coat has its own roughness).
static __device__ __noinline__ void add_relative_grads(AdjCtx* a, const LayeredBsdf& B, vec3 wo, vec3 wi, vec3 weight,
                                                vec3 c) {
  float pdf;
  const float inv2h = 0.5f / kParamStep;
  vec3 f(0.0f), da(0.0f), dr(0.0f);
  for (int i = 0; i < B.count; ++i) {
    const Lobe& L = B.lobe[i];
    f += lobe_eval(L, wo, wi, &pdf);
    if (L.role == kRoleDiffuse) {
      Lobe u = L;
      u.albedo = a->lambert_coeff;
      da += lobe_eval(u, wo, wi, &pdf);
    }
    if (L.role == kRoleMetal) {
      Lobe hi = L, lo = L;
      hi.nt = a->metal_n[0];
      hi.kt = a->metal_k[0];
      lo.nt = a->metal_n[1];
      lo.kt = a->metal_k[1];
      da += (lobe_eval(hi, wo, wi, &pdf) - lobe_eval(lo, wo, wi, &pdf)) * inv2h;
    }
    if (L.role == kRoleMetal || L.role == kRoleSpecular || L.role == kRoleTransmission) {
      Lobe hi = L, lo = L;
      hi.ax = a->ax[0];
      hi.ay = a->ay[0];
      lo.ax = a->ax[1];
      lo.ay = a->ay[1];
      dr += (lobe_eval(hi, wo, wi, &pdf) - lobe_eval(lo, wo, wi, &pdf)) * inv2h;
    }
  }
  float rough = 0.0f;
  for (int ch = 0; ch < 3; ++ch) {
    if (!(f[ch] > 0.0f)) continue;
    const float s = weight[ch] * c[ch] / f[ch];
    a->g[ch] += s * da[ch];
    rough += s * dr[ch];
  }
  a->g[3] += rough;
}

// Where a surface shadow ray goes when shadow rays are deferred: the queue
// k_connect traces, the pixel it lights and the path's weight on it
// (throughput / spp).
struct ShadowEmit {
  ShadowQueue q;
  uint32_t* count;
  uint32_t* errors;
  uint32_t pixel;
  uint32_t job;
  uint32_t path;
  vec3 weight;
};

// Queues one shadow ray with its contribution (warp-aggregated slot claim
// over the lanes that reach this point together).
__device__ __forceinline__ void emit_shadow_ray(const ShadowEmit& em, vec3 o, vec3 d, float maxd, vec3 contribution) {
  cg::coalesced_group g = cg::coalesced_threads();
  uint32_t base = 0;
  if (g.thread_rank() == 0) base = atomicAdd(em.count, g.size());
  const uint32_t slot = g.shfl(base, 0) + g.thread_rank();
  if (slot >= em.q.capacity) {
    atomicOr(em.errors, kDevErrQueue);
    return;
  }
  const vec3 w = em.weight * contribution;
  em.q.o[slot] = make_float4(o.x, o.y, o.z, maxd);
  em.q.d[slot] = make_float4(d.x, d.y, d.z, __uint_as_float(em.pixel));
  em.q.c[slot] = make_float4(w.x, w.y, w.z, __uint_as_float(em.job));
  em.q.path[slot] = em.path;
}

// A light chosen for next-event estimation: a shape light (triangle or
// sphere) or a distant light, and the probability of the choice.
struct ChosenLight {
  bool distant;
  int index;        // into S.distant_lights or S.shape_lights
  float area;       // shape lights
  float select_pdf;
  LightTri tri;     // shape lights
};
template <uint32_t kF>
__device__ __forceinline__ void choose_light(const DeviceScene& S, bool distant, float u, ChosenLight& L) {
  L.distant = distant;
  if (distant) {
    L.select_pdf = 1.0f / float(S.distant_light_count);
    L.index = gmax(gmin((int)(u * S.distant_light_count), (int)S.distant_light_count - 1), 0);
    return;
  }
  L.index = sample_light_power(S, u, &L.select_pdf);
  const ShapeLight sl = S.shape_lights[L.index];
  L.area = sl.area;
  L.tri = load_light_tri<kF>(S, sl);
}
// The light of an earlier choice (L.index, L.select_pdf).
template <uint32_t kF>
__device__ __forceinline__ void reload_light(const DeviceScene& S, bool distant, ChosenLight& L) {
  L.distant = distant;
  if (distant) return;
  const ShapeLight sl = S.shape_lights[L.index];
  L.area = sl.area;
  L.tri = load_light_tri<kF>(S, sl);
}
// A direction toward the light from `p` (false: none), its radiance and pdf;
// shape lights also give the point on the light with its error and normal.
template <uint32_t kF>
__device__ __forceinline__ bool sample_chosen_light(const DeviceScene& S, const ChosenLight& L, vec3 p, float u0, float u1,
                                                 LightSample& q) {
  if (L.distant) {
    distant_sample_li(S, S.distant_lights[L.index], u0, u1, &q.dir, &q.Li, &q.pdf);
    return true;
  }
  return light_sample_li<kF>(L.tri, L.area, p, u0, u1, &q.dir, &q.pos, &q.err, &q.ng, &q.Li, &q.pdf);
}
// The light's radiance along a direction from `p` (zero: not hit) and the pdf
// sample_chosen_light would give it.
template <uint32_t kF>
__device__ __forceinline__ void eval_chosen_light(const DeviceScene& S, const ChosenLight& L, vec3 p, LightSample& q) {
  q.Li = L.distant ? distant_eval_li(S, S.distant_lights[L.index], q.dir, &q.pdf)
                   : light_eval_li<kF>(L.tri, L.area, p, q.dir, &q.pos, &q.err, &q.ng, &q.pdf);
}

// kDefer (surfaces only, no indirect clamp): next-event shadow rays are queued
// for k_connect instead of traced here, which keeps traversal out of this
// kernel.
//
// kAdj: the path-replay adjoint pass, in phases (launch_shade_phases). Paths
// are shaded exactly as in the forward pass, nothing is added to the image,
// and each material vertex adds its terms of dLoss/dParam (see AdjCtx) to
// `grads` (per-block sums in shared memory, then one atomic per touched slot).
//
// The block works stage by stage: fetch the vertex, build its BSDF (mapped
// frame, textured parameters, lobes), and for each of the (up to four) shadow
// rays set it up, test its occlusion, follow its transmittance, then the
// continuation, with a barrier between the stages. The kernel is 150-470 KB of
// code, more than an SM's instruction caches hold, and warps left to run on
// their own spread over all of it: they waited for instructions 21-32 of 28-40
// cycles per issue. Behind barriers the warps of an SM run the same few KB at
// a time, and the wait falls to 1.3 (solid textures; surfaces 1.4). So the block is as wide as an SM
// has registers for (512 threads of 128) where the code is widest: media and
// textures (one B200, without barriers at 128 threads -> 512: volumetric
// 1280x720 16 spp 528 -> 299 ms, solid textures 8 spp 197 -> 72 ms, image
// textures 640x480 16 spp 37.2 -> 20.3 ms; 256 threads 334, 96 and 23.4 ms).
// Surfaces without textures need less of the code at a time and lose more to
// the barriers: 128 threads, four blocks per SM (instanced 1080p 64 spp
// shading 48.4 ms without barriers, 41.3 at 128, 40.5 at 256, 42.6 at 512;
// Cornell 256x256 16 spp 1.28, 1.31, 1.37, 1.45 ms). Surface adjoint 256
// threads (41.1 ms for 4 views 512x512 16 spp; 61.7 without barriers, 46.9 at
// 128, 43.5 at 512). Finer stages where they are the long ones: occlusion and
// transmittance apart (shading of the fog gradients' forward pass 12.1 ->
// 11.3 ms, of solid textures 44.8 -> 43.1), mapped frame and parameters apart
// (44.8 -> 42.1, image textures 11.65 -> 11.3); one between a light's sampling
// and its BSDF value gained nothing.
template <bool kVol, bool kDefer, bool kAdj, uint32_t kF>
constexpr uint32_t shade_threads() {
  if (kVol || (kF & kFeatTextures)) return 512;
  return kAdj ? 256 : 128;
}
template <bool kVol, bool kDefer, bool kAdj, uint32_t kF>
constexpr uint32_t shade_blocks_per_sm() {  // 128 registers a thread
  return 512 / shade_threads<kVol, kDefer, kAdj, kF>();
}

// The coincident hits of path slot i (at least the hit itself); returns their number.
__device__ __forceinline__ int load_nearby(const HitPool& H, uint32_t i, uint4 ids, float t, NearbyHit* nb) {
  const int n = (int)(ids.w & 0xFFu);
  if (ids.w & kNearbyExplicit) {
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
      const uint4 e = H.nearby[(size_t)i * kMaxNearby + k];
      nb[k] = NearbyHit{e.x, __uint_as_float(e.y), (int)e.z};
    }
  } else {
    nb[0] = NearbyHit{ids.x, t, (int)(ids.z & 1u)};
  }
  return n;
}

// A vertex kept between the launches of a phased k_shade: surface point and
// shading frame in six 16-byte words, each lobe in four, word k of all
// vertices together (a warp's accesses are contiguous).
__device__ __forceinline__ void store_vertex(const VertexQueue& X, uint32_t t, const SurfacePoint& sp,
                                             const LayeredBsdf& B) {
  const size_t n = X.capacity;
  uint4* v = X.state + 2 * n + t;
  v[0] = make_uint4(f2u(sp.p.x), f2u(sp.p.y), f2u(sp.p.z), f2u(sp.p_err.x));
  v[n] = make_uint4(f2u(sp.p_err.y), f2u(sp.p_err.z), f2u(sp.ng.x), f2u(sp.ng.y));
  v[2 * n] = make_uint4(f2u(sp.ng.z), f2u(B.t.x), f2u(B.t.y), f2u(B.t.z));
  v[3 * n] = make_uint4(f2u(B.b.x), f2u(B.b.y), f2u(B.b.z), f2u(B.n.x));
  v[4 * n] = make_uint4(f2u(B.n.y), f2u(B.n.z), (uint32_t)B.count, f2u(B.w[0]));
  if (B.count > 1) v[5 * n] = make_uint4(f2u(B.w[1]), f2u(B.w[2]), f2u(B.w[3]), f2u(B.w[4]));
#pragma unroll 1
  for (int c = 0; c < B.count; ++c) {
    const Lobe& l = B.lobe[c];
    uint4* q = X.lobes + (size_t)c * 4 * n + t;
    q[0] = make_uint4((uint32_t)l.type, f2u(l.albedo.x), f2u(l.albedo.y), f2u(l.albedo.z));
    q[n] = make_uint4(f2u(l.nt.x), f2u(l.nt.y), f2u(l.nt.z), f2u(l.ni));
    q[2 * n] = make_uint4(f2u(l.kt.x), f2u(l.kt.y), f2u(l.kt.z), f2u(l.ax));
    q[3 * n] = make_uint4(f2u(l.ay), (uint32_t)l.is_metal, (uint32_t)l.role, 0u);
  }
}
__device__ __forceinline__ void load_vertex(const VertexQueue& X, uint32_t t, SurfacePoint& sp, LayeredBsdf& B) {
  const size_t n = X.capacity;
  const uint4* v = X.state + 2 * n + t;
  const uint4 a = v[0], b = v[n], c = v[2 * n], d = v[3 * n], e = v[4 * n];
  sp.p = vec3(u2f(a.x), u2f(a.y), u2f(a.z));
  sp.p_err = vec3(u2f(a.w), u2f(b.x), u2f(b.y));
  sp.ng = vec3(u2f(b.z), u2f(b.w), u2f(c.x));
  B.t = vec3(u2f(c.y), u2f(c.z), u2f(c.w));
  B.b = vec3(u2f(d.x), u2f(d.y), u2f(d.z));
  B.n = vec3(u2f(d.w), u2f(e.x), u2f(e.y));
  B.count = (int)e.z;
  B.w[0] = u2f(e.w);
  if (B.count > 1) {
    const uint4 f = v[5 * n];
    B.w[1] = u2f(f.x);
    B.w[2] = u2f(f.y);
    B.w[3] = u2f(f.z);
    B.w[4] = u2f(f.w);
  }
#pragma unroll 1
  for (int k = 0; k < B.count; ++k) {
    const uint4* q = X.lobes + (size_t)k * 4 * n + t;
    const uint4 q0 = q[0], q1 = q[n], q2 = q[2 * n], q3 = q[3 * n];
    Lobe& l = B.lobe[k];
    l.type = (int)q0.x;
    l.albedo = vec3(u2f(q0.y), u2f(q0.z), u2f(q0.w));
    l.nt = vec3(u2f(q1.x), u2f(q1.y), u2f(q1.z));
    l.ni = u2f(q1.w);
    l.kt = vec3(u2f(q2.x), u2f(q2.y), u2f(q2.z));
    l.ax = u2f(q2.w);
    l.ay = u2f(q3.x);
    l.is_metal = (int)q3.y;
    l.role = (int)q3.z;
  }
}
// The adjoint's data of the vertex: its gradients so far, and (once) the rest.
__device__ __forceinline__ void store_adjoint(const VertexQueue& X, uint32_t t, const AdjCtx& a, bool gradients_only) {
  const size_t n = X.capacity;
  uint4* v = X.adjoint + t;
  v[0] = make_uint4(f2u(a.g[0]), f2u(a.g[1]), f2u(a.g[2]), f2u(a.g[3]));
  if (gradients_only) return;
  v[n] = make_uint4(f2u(a.weight.x), f2u(a.weight.y), f2u(a.weight.z), f2u(a.lambert_coeff.x));
  v[2 * n] = make_uint4(f2u(a.lambert_coeff.y), f2u(a.lambert_coeff.z), f2u(a.metal_n[0].x), f2u(a.metal_n[0].y));
  v[3 * n] = make_uint4(f2u(a.metal_n[0].z), f2u(a.metal_n[1].x), f2u(a.metal_n[1].y), f2u(a.metal_n[1].z));
  v[4 * n] = make_uint4(f2u(a.metal_k[0].x), f2u(a.metal_k[0].y), f2u(a.metal_k[0].z), f2u(a.metal_k[1].x));
  v[5 * n] = make_uint4(f2u(a.metal_k[1].y), f2u(a.metal_k[1].z), f2u(a.ax[0]), f2u(a.ax[1]));
  v[6 * n] = make_uint4(f2u(a.ay[0]), f2u(a.ay[1]), 0u, 0u);
}
__device__ __forceinline__ void load_adjoint(const VertexQueue& X, uint32_t t, AdjCtx& a) {
  static_assert(kGradParams == 4, "one 16-byte word of gradients");
  const size_t n = X.capacity;
  const uint4* v = X.adjoint + t;
  const uint4 g = v[0], b = v[n], c = v[2 * n], d = v[3 * n], e = v[4 * n], f = v[5 * n], h = v[6 * n];
  a.g[0] = u2f(g.x);
  a.g[1] = u2f(g.y);
  a.g[2] = u2f(g.z);
  a.g[3] = u2f(g.w);
  a.weight = vec3(u2f(b.x), u2f(b.y), u2f(b.z));
  a.lambert_coeff = vec3(u2f(b.w), u2f(c.x), u2f(c.y));
  a.metal_n[0] = vec3(u2f(c.z), u2f(c.w), u2f(d.x));
  a.metal_n[1] = vec3(u2f(d.y), u2f(d.z), u2f(d.w));
  a.metal_k[0] = vec3(u2f(e.x), u2f(e.y), u2f(e.z));
  a.metal_k[1] = vec3(u2f(e.w), u2f(f.x), u2f(f.y));
  a.ax[0] = u2f(f.z);
  a.ax[1] = u2f(f.w);
  a.ay[0] = u2f(h.x);
  a.ay[1] = u2f(h.y);
}

template <bool kVol, bool kDefer, bool kAdj, uint32_t kF>
__global__ void __launch_bounds__(shade_threads<kVol, kDefer, kAdj, kF>(), shade_blocks_per_sm<kVol, kDefer, kAdj, kF>()) k_shade(
    PathPool P, const WaveControl* __restrict__ ctl, HitPool H, PathPool Q, const JobDesc* __restrict__ jobs,
    WaveCounters* counters, ShadowQueue shadow_q, float* grads = nullptr, uint32_t grad_materials = 0,
    ShadePhase ph = ShadePhase{}) {
  static_assert(!(kVol && kDefer), "volume transmittance needs the path's sampler: shadow rays are traced inline");
  static_assert(!(kAdj && kDefer), "the adjoint pass traces its shadow rays in turn");
  constexpr bool kSpheres = (kF & kFeatSpheres) != 0;
  constexpr bool kPhased = kAdj;
  const VertexQueue& X = ph.X;
  const bool first = !kPhased || ph.phase == 0, last = !kPhased || ph.phase == ph.passes;
  float* s_grad = nullptr;
  const uint32_t n_slots = min(grad_materials, (uint32_t)kMaxGradMaterials) * kGradParams;
  if constexpr (kAdj) {
    __shared__ float s_grad_buf[kMaxGradMaterials * kGradParams];
    s_grad = s_grad_buf;
    for (uint32_t k = threadIdx.x; k < n_slots; k += blockDim.x) s_grad[k] = 0.0f;
    __syncthreads();
  }
  TraversalStack st;
  if constexpr (!kDefer && !kPhased) {
    YM_TRAVERSAL_SHARED_DYNAMIC(s_stack);
    st.bind(s_stack);
  } else {
    st.sp = 0;
    st.overflow = false;
  }
  const bool listed = H.order != nullptr;
  const uint32_t count = listed ? min(ctl->count, counters->hit_count) : ctl->count;
  uint32_t shadow_rays = 0, tests = 0, nodes = 0;
  uint32_t* errors = &counters->errors;
#pragma unroll 1
  for (uint32_t block_base = blockIdx.x * blockDim.x; block_base < count; block_base += gridDim.x * blockDim.x) {
    // The path slot this lane shades: the t-th listed hit, or (hits not listed
    // by bucket) slot t itself when it holds a live path.
    const uint32_t t_idx = block_base + threadIdx.x;
    bool active = t_idx < count;
    const uint32_t i = active ? (listed ? H.order[t_idx] : t_idx) : 0u;
    const uint2 pf = active ? P.pixel_flags[i] : make_uint2(kEmpty, kFlagDead);
    if (pf.y & kFlagDead) active = false;  // a miss (already accumulated) or an empty slot
    uint32_t flags = 0u;     // (phased) kVertex*
    if (kPhased && !first) {
      flags = active ? X.flags[t_idx] : 0u;
      active = flags != 0u;
      if (!__syncthreads_or(active)) continue;
    }
    bool alive = false;      // continues into Q
    bool ended = false;      // a path whose radiance is complete
    bool surface = false;    // a material vertex: next-event estimation and a BSDF continuation
    bool volume = false;     // a volume vertex: the same with the media's phase functions

    vec3 new_o, new_d, tp, rad, rd;
    uint32_t new_flags = 0, new_last_inst = kEmpty, new_last_tri = kEmpty;
    PathSampler hs{0, 0u, 0u};
    RayTransfer rt;
    rt.record_count = 0;
    rt.max_priority_record_index = -1;
    const uint32_t job = active ? pf.y >> kFlagJobShift : 0u;
    const JobDesc& J = jobs[job];
    const uint32_t slot = J.scene_slot;
    const DeviceScene& S = c_scenes[slot];
    const RenderSetting& rs = J.setting;
    const float inv_spp = 1.0f / gmax(rs.ssp, 1);
    int depth = (int)(pf.y & kFlagDepthMask);
    const uint32_t sample_bits = pf.y & ~(kFlagDepthMask | kFlagNeverScatter | kFlagCameraRay | kFlagDead);  // job
    uint32_t inst_idx = kEmpty, tri = kEmpty, material = 0;
    int hit_back = 0, n_nb = 0;
    NearbyHit nb[kMaxNearby];
    SurfacePoint sp;           // (a volume vertex: its position in sp.p)
    LayeredBsdf B;
    AdjCtx adj_ctx;
    vec3 delta(0.0f), l_total(0.0f);
    // media of a volume vertex
    float vw[kMaxBoundaryRecord], gs[kMaxBoundaryRecord];
    int n_media = 0;

    if (active) {
      const float4 d4 = P.ray_d[i], t4 = P.throughput[i], r4 = P.radiance[i];
      rd = vec3(d4.x, d4.y, d4.z);
      tp = vec3(t4.x, t4.y, t4.z);
      rad = vec3(r4.x, r4.y, r4.z);
      const uint4 s4 = P.sampler[i];
      hs.index = (uint64_t)s4.x | ((uint64_t)s4.y << 32);
      hs.dim = s4.z;
      hs.aux = s4.w;
      const bool never_scatter = (pf.y & kFlagNeverScatter) != 0;
      if (P.transfer_count[i] > 0) rt = P.transfer[i];
      const float4 bt = H.bary_t[i];
      const uint4 ids = H.ids[i];
      const vec3 bary(bt.x, bt.y, bt.z);
      inst_idx = ids.x;
      tri = ids.y;
      hit_back = (int)(ids.z & 1u);
      volume = kVol && (ids.z & 2u);
      if (kPhased && !first) hs.dim = X.dim[t_idx];
      if (kAdj) {
        const float4 dl = J.dloss[pf.x];
        delta = vec3(dl.x, dl.y, dl.z) * inv_spp;  // dLoss/d(this path's radiance)
      }
      if (volume) {
        // Ray_shading_path_tracing volume branch (src/Shading.cu:2066-2126).
        int vidx[kMaxBoundaryRecord];
        n_media = current_volumes(rt, S.volume_count, vidx);
#pragma unroll 1
        for (int k = 0; k < n_media; ++k) {
          gs[k] = S.volumes[vidx[k]].g;
          vw[k] = H.vol_w[(size_t)i * kMaxBoundaryRecord + k];
        }
        sp.p = bary;
        inst_idx = tri = kEmpty;
      } else if (inst_idx == kEmpty) {
        // a miss (Ray_trace_path_tracing, src/Shading.cu:1855-1864): the
        // background when the environment light is on, then the path ends
        if (rs.enable_env_light) rad += indirect_clamp(rs, tp * background(rd), depth);
        ended = true;
      } else {
        n_nb = load_nearby(H, i, ids, bt.w, nb);
        const Instance inst = S.instances[inst_idx];
        material = inst.material_idx;
        if (first) sp = fetch_surface<kF>(S, inst_idx, tri, bary);
        if (kPhased && !first) {
          surface = true;
        } else if (!(material < S.material_count)) {
          ended = true;
        } else {
          const Material& mat = S.materials[material];
          uint32_t prio = 0;
          fetch_ior(mat, &prio);
          if (inst.treat_as_boundary ||
              (rt.record_count != 0 && prio < rt.records[rt.max_priority_record_index].ior_priority)) {
            // a boundary, or a lower-priority one: pass straight through, no depth consumed
            boundary_transition(S, rt, nb, n_nb, errors);
            new_o = offset_ray_origin(sp.p, sp.p_err, rd, sp.ng);
            new_d = normalize(rd);
            new_flags = flags_pack(depth, never_scatter, false, 0) | sample_bits;
            new_last_inst = inst_idx;
            new_last_tri = tri;
            alive = true;
          } else if (mat.material_type == kLightMtl) {
            if (never_scatter) rad += indirect_clamp(rs, tp * mat.light_mtl.light_color * mat.light_mtl.intensity, depth);
            ended = true;
          } else {
            surface = true;
          }
        }
      }
    }

    // The layered BSDF of a material vertex.
    __syncthreads();
    ChosenLight L;
    vec3 direct(0.0f);
    if (kPhased && !first && active) {
      const uint4 m0 = X.state[t_idx], m1 = X.state[X.capacity + t_idx];
      rad = vec3(u2f(m0.x), u2f(m0.y), u2f(m0.z));
      direct = vec3(u2f(m1.x), u2f(m1.y), u2f(m1.z));
      L.index = (int)m0.w;
      L.select_pdf = u2f(m1.w);
      if (surface) load_vertex(X, t_idx, sp, B);
      if constexpr (kAdj) {
        if (surface) load_adjoint(X, t_idx, adj_ctx);
      }
    }
    bool plain = true;
    DefaultMtl mt;
    if constexpr ((kF & kFeatTextures) != 0) {
      if (first) {
        const TexCoord tc{sp.u, sp.v, sp.p_obj};
        const bool textured = surface && material_textured(S.materials[material].default_mtl);
        if (textured) {
          // textured parameters, normal or bump mapping: read at the hit
          mt = S.materials[material].default_mtl;
          init_shading_frame_mapped(B, mt, hit_back, rd, sp, S.i_transforms[S.instances[inst_idx].transform_idx], S, tc,
                                    errors);
          plain = false;
        }
        __syncthreads();
        if (textured) resolve_material_textures(mt, S.textures, tc, errors);
        __syncthreads();
      }
    }
    if (first && surface) {
      const DefaultMtl* mp = plain ? &S.materials[material].default_mtl : &mt;
      if (plain) init_shading_frame(B, hit_back, rd, sp.ng, sp.ns, sp.dpdu, sp.dpdv);
      init_layered_lobes(B, *mp, rd, hit_back, ray_ior(rt), ex_ior(rt, inst_idx));
      if constexpr (kAdj) {
        const float4 lt = J.path_radiance[P.path_id[i]];
        l_total = vec3(lt.x, lt.y, lt.z);
        init_adjoint(adj_ctx, B, *mp);
        adj_ctx.weight = delta * tp;
      }
    }
    if constexpr (kAdj) {
      if (!first && surface) {
        const float4 lt = J.path_radiance[P.path_id[i]];
        l_total = vec3(lt.x, lt.y, lt.z);
      }
    }
    const vec3 wo = surface ? B.to_local(-rd) : vec3(0.0f);

    // Next-event estimation: EvalDistantLight / EvalShapeLight (src/Shading.cu:83-198,
    // 294-417) at material vertices, EvalVolumeDistantLight / EvalVolumeShapeLight
    // (:202-291, 419-513) at volume vertices. Two kinds of light, and for each
    // a direction sampled from the light (pass 0) and one from the BSDF or the
    // phase functions (pass 1).
    // (phased) one pass per launch: its shadow rays are queued and traced by
    // k_occlude and k_transmit, whose answers the next launch takes up here.
    auto kind_of = [&](int pass) { return kPhased ? (ph.kinds == 2u || pass >= 2 ? 1 : 0) : pass >> 1; };
    auto kind_on = [&](bool distant) {
      return (surface || (volume && n_media > 0)) &&
             (distant ? rs.enable_distant_light && S.distant_light_count > 0
                      : rs.enable_shape_light != 0 && S.shape_light_count > 0);
    };
    // a pass's contribution, and after the second of a kind the kind's estimate
    auto finish_kind = [&](bool distant) {
      const vec3 e = distant || (kVol && volume) ? (L.select_pdf > 0.0f ? direct / L.select_pdf : vec3(0.0f))
                                                 : direct * safe_rcp(L.select_pdf);
      rad += indirect_clamp(rs, tp * e, depth);
    };
    if constexpr (kPhased) {
      if (!first && active) {
        const int p = ph.phase - 1;
        const bool distant = kind_of(p) == 0;
        if (flags & kVertexRay) {
          const float4 r = X.result[t_idx];
          if (r.w != 0.0f) {
            const uint4 p0 = X.pass[t_idx], p1 = X.pass[X.capacity + t_idx];
            const vec3 contrib = u2f(p0.x) * vec3(r.x, r.y, r.z) * vec3(u2f(p0.y), u2f(p0.z), u2f(p0.w)) *
                                 vec3(u2f(p1.x), u2f(p1.y), u2f(p1.z));
            direct += contrib;
            if constexpr (kAdj) {
              if (surface) {
                // d(direct)/dp = mis * tr * fc * (df/dp)/f * Lc, scaled like the estimator
                const float mul = distant ? 1.0f : safe_rcp(L.select_pdf), div = distant ? L.select_pdf : 1.0f;
                const uint4 p2 = X.pass[2 * (size_t)X.capacity + t_idx];
                const vec3 dir(u2f(p1.w), u2f(p2.x), u2f(p2.y));
                add_relative_grads(&adj_ctx, B, wo, B.to_local(dir), adj_ctx.weight * (mul / div), contrib);
              }
            }
          }
        }
        if ((p & 1) && kind_on(distant)) finish_kind(distant);
      }
    }
#pragma unroll 1
    for (int p = kPhased ? ph.phase : 0; p < (kPhased ? min(ph.phase + 1, ph.passes) : 4); ++p) {
      const bool distant = kind_of(p) == 0;
      const int pass = p & 1;
      const bool on = kind_on(distant);
      if (!kPhased && pass == 0 && !__syncthreads_or(on)) {
        ++p;  // neither pass of this kind
        continue;
      }
      if (on) {
        if (pass == 0) {
          direct = vec3(0.0f);
        } else if (kPhased) {
          reload_light<kF>(S, distant, L);
        }
      }
      {
        LightSample q{vec3(0.0f), vec3(0.0f), vec3(0.0f), vec3(0.0f), vec3(0.0f), 0.0f};
        vec3 f(0.0f), lwi(0.0f), so(0.0f);
        float spdf = 0.0f, maxd = kTMax;  // spdf: of the BSDF or the phase functions
        bool ok = on, tb = false;
        if (on) {
          // pass 0: the light's choice and a point on it; pass 1: a direction
          const float3 u = sample_next(hs, S, pass == 0 || surface ? 3 : 2);
          if (pass == 0) {
            choose_light<kF>(S, distant, u.x, L);
            ok = sample_chosen_light<kF>(S, L, sp.p, u.y, u.z, q);
            if (ok) {
              if (!kVol || surface) {
                lwi = B.to_local(q.dir);
                f = bsdf_eval(B, wo, lwi, &spdf);
              } else {
                f = vec3(eval_mixed_phases(vw, gs, n_media, -rd, q.dir, &spdf));
              }
              ok = max_component(f) > kMinColorEps;
            }
          } else {
            if (!kVol || surface) {
              ok = bsdf_sample(B, wo, &f, &lwi, &spdf, u.x, u.y, u.z);
              if (ok) q.dir = B.to_world(lwi);
            } else {
              float pw = 0.0f;
              ok = sample_mixed_phases(vw, gs, n_media, u.x, u.y, -rd, &pw, &q.dir, &spdf);
              f = vec3(pw);
            }
            if (ok) {
              eval_chosen_light<kF>(S, L, sp.p, q);
              ok = max_component(q.Li) > kMinColorEps;
            }
          }
          so = sp.p;
          if (ok && surface) {
            tb = dot(-rd, sp.ng) * dot(q.dir, sp.ng) < 0.0f;
            if (same_hemisphere(wo, lwi) ? tb : !tb) ok = false;
            else so = offset_ray_origin(sp.p, sp.p_err, q.dir, sp.ng);
          }
          if (ok && !distant) maxd = length(offset_ray_origin(q.pos, q.err, -q.dir, q.ng) - sp.p) * kShadowRayClamp;
        }
        float mis = 0.0f;
        vec3 fc(0.0f), Lc(0.0f);
        if (ok) {
          ++shadow_rays;
          mis = power_heuristic(pass == 0 ? q.pdf : spdf, pass == 0 ? spdf : q.pdf);
          fc = vmin(f, vec3(kMaxColorClamp));
          Lc = vmin(q.Li, vec3(kMaxColorClamp));
        }
        if constexpr (kDefer) {
          // the light-selection pdf enters as a factor here and as a quotient for distant lights
          if (ok) {
            const ShadowEmit em{shadow_q, &counters->shadow_count[shadow_q.turn], errors, pf.x, job, P.path_id[i], tp * inv_spp};
            const float mul = distant ? 1.0f : safe_rcp(L.select_pdf), div = distant ? L.select_pdf : 1.0f;
            emit_shadow_ray(em, so, normalize(q.dir), maxd, ((mis * vec3(1.0f) * fc * Lc) * mul) / div);
          }
          __syncthreads();
        } else if constexpr (kPhased) {
          // kept for the next launch: the vertex (once), what the pass changes,
          // and the ray
          flags = surface || volume ? (surface ? kVertexSurface : kVertexScatter) | (ok ? kVertexRay : 0u) : 0u;
          if (flags) {
            if (first && surface) {
              store_vertex(X, t_idx, sp, B);
            }
            if constexpr (kAdj) {
              if (surface) store_adjoint(X, t_idx, adj_ctx, !first);
            }
            X.state[t_idx] = make_uint4(f2u(rad.x), f2u(rad.y), f2u(rad.z), (uint32_t)L.index);
            X.state[X.capacity + t_idx] = make_uint4(f2u(direct.x), f2u(direct.y), f2u(direct.z), f2u(L.select_pdf));
            X.dim[t_idx] = hs.dim;
          }
          if (ok) {
            const vec3 dir = normalize(q.dir);
            const bool media = kVol && (volume || rs.enable_volume_scattering);
            X.ray_o[t_idx] = make_float4(so.x, so.y, so.z, maxd);
            X.ray_d[t_idx] = make_float4(dir.x, dir.y, dir.z,
                                         u2f(slot << kRaySlotShift | (tb ? kRayCrosses : 0u) | (media ? kRayMedia : 0u)));
            X.pass[t_idx] = make_uint4(f2u(mis), f2u(fc.x), f2u(fc.y), f2u(fc.z));
            X.pass[X.capacity + t_idx] = make_uint4(f2u(Lc.x), f2u(Lc.y), f2u(Lc.z), f2u(q.dir.x));
            if (kAdj) X.pass[2 * (size_t)X.capacity + t_idx] = make_uint4(f2u(q.dir.y), f2u(q.dir.z), 0u, 0u);
          }
          const uint32_t at = warp_append(&counters->ray_count[p], ok);
          if (ok) X.queue[at] = t_idx;
        } else {
          __syncthreads();
          const vec3 dir = normalize(q.dir);
          if (ok) ok = !trace_occluded_impl<kSpheres>(slot, st, so, dir, maxd, &tests, &nodes);
          if (kVol) __syncthreads();
          if (ok) {
            vec3 tr(1.0f);
            if (kVol && (volume || rs.enable_volume_scattering)) {
              RayTransfer srt = rt;
              if (tb) boundary_transition(S, srt, nb, n_nb, errors);
              tr = trace_tr<kF>(slot, st, so, dir, maxd, inst_idx, tri, srt, hs, errors, &tests, &nodes);
            }
            direct += mis * tr * fc * Lc;
          }
          __syncthreads();
        }
      }
      if (!kPhased && pass == 1 && on) finish_kind(distant);
    }
    if (kPhased && !last) {
      if (first && t_idx < count) X.flags[t_idx] = flags;
      else if (active) X.flags[t_idx] = flags;
    }

    // The continuation: a direction from the BSDF or the phase functions.
    if (last && (surface || (kVol && volume))) {
      const float3 u = sample_next(hs, S, surface ? 3 : 2);
      vec3 w(0.0f), wi(0.0f);
      float pdf = 0.0f;
      bool valid;
      if (!kVol || surface) {
        valid = bsdf_sample(B, wo, &w, &wi, &pdf, u.x, u.y, u.z);
      } else {
        float pw = 0.0f;
        valid = sample_mixed_phases(vw, gs, n_media, u.x, u.y, -rd, &pw, &wi, &pdf);
        w = vec3(pw);
      }
      if constexpr (kAdj) {
        if (surface) {
          // the radiance gathered after this vertex, through the sampled BSDF value
          if (valid) add_relative_grads(&adj_ctx, B, wo, wi, delta, l_total - rad);
          for (int k = 0; k < kGradParams; ++k) {
            if (adj_ctx.g[k] == 0.0f) continue;
            if (material * kGradParams + k < n_slots) atomicAdd(&s_grad[material * kGradParams + k], adj_ctx.g[k]);
            else if (material < grad_materials) atomicAdd(&grads[material * kGradParams + k], adj_ctx.g[k]);
          }
        }
      }
      bool terminate = !valid;
      if (valid) {
        tp *= w;
        float rr = gmax(tp.x, gmax(tp.y, tp.z));
        rr = gmin(rr, 1.0f);
        if (depth + 1 > rs.ray_depth) {
          if (rs.enable_russian_roulette && sample1d(hs, S) < rr) tp /= gmax(rr, kMinColorEps);
          else terminate = true;
        }
      }
      if (!terminate) {
        new_o = sp.p;
        vec3 nd = wi;
        if (!kVol || surface) {
          nd = B.to_world(wi);
          const bool tb = dot(-rd, sp.ng) * dot(nd, sp.ng) < 0.0f;
          if (same_hemisphere(wo, wi) ? tb : !tb) {
            terminate = true;
          } else {
            if (tb) boundary_transition(S, rt, nb, n_nb, errors);
            new_o = offset_ray_origin(sp.p, sp.p_err, nd, sp.ng);
          }
        }
        new_d = normalize(nd);
        depth += 1;
        if (depth > kMaxRayDepth) terminate = true;
        new_flags = flags_pack(depth, false, false, 0) | sample_bits;
        new_last_inst = inst_idx;
        new_last_tri = tri;
        alive = !terminate;
      }
      ended = terminate;
    }
    if (ended) end_path<kAdj>(J, pf.x, P.path_id[i], rad, inv_spp);

    const uint32_t q_slot = warp_append(&counters->next_count, alive);
    if (alive) {
      if (q_slot < Q.capacity) {
        store_path(Q, q_slot, new_o, new_d, tp, rad, pf.x, new_flags, new_last_inst, new_last_tri, hs, P.path_id[i]);
        Q.transfer_count[q_slot] = (uint8_t)rt.record_count;
        if (rt.record_count > 0) Q.transfer[q_slot] = rt;
      } else {
        atomicOr(&counters->errors, (uint32_t)kDevErrQueue);
      }
    }
  }
  if (st.overflow) atomicOr(&counters->errors, (uint32_t)kDevErrStack);
  uint32_t s_sum = shadow_rays, t_sum = tests, n_sum = nodes;
  for (int off = 16; off > 0; off >>= 1) {
    s_sum += __shfl_down_sync(0xFFFFFFFFu, s_sum, off);
    t_sum += __shfl_down_sync(0xFFFFFFFFu, t_sum, off);
    n_sum += __shfl_down_sync(0xFFFFFFFFu, n_sum, off);
  }
  if ((threadIdx.x & 31) == 0) {
    if (s_sum) atomicAdd(&counters->shadow_rays, (unsigned long long)s_sum);
    if (t_sum) atomicAdd(&counters->shadow_tri_tests, (unsigned long long)t_sum);
    if (n_sum) atomicAdd(&counters->shadow_node_visits, (unsigned long long)n_sum);
  }
  if constexpr (kAdj) {
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < n_slots; k += blockDim.x)
      if (s_grad[k] != 0.0f) atomicAdd(&grads[k], s_grad[k]);
  }
}

// Lets a k_shade instantiation that traces its shadow rays inline take its
// block's traversal stacks in dynamic shared memory (more than the default 48 KB).
template <bool kVol, uint32_t kF>
static void allow_shade_shared() {
  cudaFuncSetAttribute(k_shade<kVol, false, false, kF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)traversal_shared_bytes(shade_threads<kVol, false, false, kF>()));
}

// Launches k_shade over the wave (one thread per pool slot): the forward
// pass, with deferred or inline shadow rays.
template <bool kVol, bool kDefer, uint32_t kF>
void launch_shade(const WaveArgs& w, const ShadowQueue& q) {
  constexpr uint32_t threads = shade_threads<kVol, kDefer, false, kF>();
  const uint32_t blocks = (w.blocks * kTraceBlock + threads - 1) / threads;
  const size_t shared = kDefer ? 0 : traversal_shared_bytes(threads);
  k_shade<kVol, kDefer, false, kF><<<blocks, threads, shared, w.stream>>>(w.A, w.ctl, w.H, w.B, w.jobs, w.counters, q);
}

// ------------------------------------------- phased next-event estimation ---
//
// The adjoint pass weighs each shadow ray's gradient terms by what the ray
// finds (and with media its transmittance draws from the path's sampler), so
// a vertex's shadow rays come one after the other. k_shade then runs in
// phases, one per pass (light kind x estimator): it queues the pass's rays and
// keeps the vertices; k_occlude and k_transmit trace the queue with full warps
// over the whole GPU; the next phase takes up the answers. Traced inline, a
// block waited at its barriers for its longest ray with a third of its lanes
// on a ray (backward of 4 views 512x512 16 spp 67.7 -> 61.8 ms, of 4 views
// 256x256 8 spp in fog 36.4 -> 31.4 ms). The forward media pass stays inline:
// it gained nothing (volumetric 1280x720 227 and 227 ms, solid textures 56.8
// inline and 58.2 phased) and would pay the extra launches in small renders.

// Occlusion of a pass's queued rays: persistent, with k_connect's warp-level
// work fetch. An unoccluded ray in media goes on to k_transmit's queue.
template <bool kSpheres>
static __global__ void __launch_bounds__(kTraceBlock, kConnectBlocksPerSm) k_occlude(VertexQueue X, WaveCounters* counters,
                                                                                     int pass) {
  extern __shared__ __align__(16) uint32_t s_occ[];  // occluded_shared_bytes(blockDim.x)
  OccStack st;
  st.bind(s_occ);
  OccWalk w;
  const uint32_t n = min(counters->ray_count[pass], X.capacity);
  const int lane = threadIdx.x & 31;
  uint32_t ray = kEmpty;   // the vertex whose ray this lane traces (kEmpty: idle)
  uint32_t bits = 0;
  bool exhausted = false;  // the queue has been handed out (warp-uniform)
  uint32_t tests = 0, nodes = 0;
  for (;;) {
    if (!exhausted) {
      const uint32_t idle = __ballot_sync(0xFFFFFFFFu, ray == kEmpty);
      if (idle) {
        const int leader = __ffs(idle) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(&counters->ray_cursor[pass], (uint32_t)__popc(idle));
        base = __shfl_sync(0xFFFFFFFFu, base, leader);
        if (base + (uint32_t)__popc(idle) >= n) exhausted = true;
        if (ray == kEmpty) {
          const uint32_t t = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
          if (t < n) {
            ray = X.queue[t];
            const float4 o = X.ray_o[ray], d = X.ray_d[ray];
            bits = __float_as_uint(d.w);
            w.begin(bits >> kRaySlotShift, vec3(o.x, o.y, o.z), vec3(d.x, d.y, d.z), o.w, st);
          }
        }
      }
    }
    if (__ballot_sync(0xFFFFFFFFu, ray != kEmpty) == 0) break;
    if (ray != kEmpty) {
      const int r = occluded_step<kSpheres>(w, st, &tests, &nodes);
      if (r != kWalkGoing) {
        const bool clear = r == kWalkClear;
        if (clear && (bits & kRayMedia)) {
          cg::coalesced_group g = cg::coalesced_threads();
          uint32_t base = 0;
          if (g.thread_rank() == 0) base = atomicAdd(&counters->tr_count[pass], g.size());
          X.queue_tr[g.shfl(base, 0) + g.thread_rank()] = ray;
        } else {
          X.result[ray] = clear ? make_float4(1.0f, 1.0f, 1.0f, 1.0f) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        ray = kEmpty;
      }
    }
  }
  for (int off = 16; off > 0; off >>= 1) {
    tests += __shfl_down_sync(0xFFFFFFFFu, tests, off);
    nodes += __shfl_down_sync(0xFFFFFFFFu, nodes, off);
  }
  if (lane == 0) {
    if (tests) atomicAdd(&counters->shadow_tri_tests, (unsigned long long)tests);
    if (nodes) atomicAdd(&counters->shadow_node_visits, (unsigned long long)nodes);
  }
  if (st.overflow) atomicOr(&counters->errors, (uint32_t)kDevErrStack);
}

// Transmittance of a pass's unoccluded rays, from the state their vertex's
// sampler was left in. With grid_grads, the ray's tracking is replayed with
// the same samples for the density-grid terms, weighted by its share of dLoss.
template <uint32_t kF>
static __global__ void __launch_bounds__(kTraceBlock, 4) k_transmit(VertexQueue X, PathPool P, HitPool H,
                                                                    const JobDesc* __restrict__ jobs,
                                                                    WaveCounters* counters, int pass, bool distant,
                                                                    float* grid_grads, uint32_t grid_tex) {
  YM_TRAVERSAL_SHARED_DYNAMIC(s_stack);
  TraversalStack st;
  st.bind(s_stack);
  const uint32_t n = min(counters->tr_count[pass], X.capacity);
  uint32_t tests = 0, nodes = 0;
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;  // (one thread per pool slot)
  if ((k & ~31u) >= n) return;  // (whole warps)
  if (k < n) {
    const uint32_t t = X.queue_tr[k];
    const uint32_t i = H.order ? H.order[t] : t;
    const float4 o4 = X.ray_o[t], d4 = X.ray_d[t];
    const uint32_t bits = __float_as_uint(d4.w), slot = bits >> kRaySlotShift;
    const vec3 o(o4.x, o4.y, o4.z), d(d4.x, d4.y, d4.z);
    const uint4 ids = H.ids[i];
    const bool volume = (ids.z & 2u) != 0u;
    const uint32_t inst = volume ? kEmpty : ids.x, tri = volume ? kEmpty : ids.y;
    RayTransfer rt;
    rt.record_count = 0;
    rt.max_priority_record_index = -1;
    if (P.transfer_count[i] > 0) rt = P.transfer[i];
    if (bits & kRayCrosses) {
      NearbyHit nb[kMaxNearby];
      const int n_nb = load_nearby(H, i, ids, H.bary_t[i].w, nb);
      boundary_transition(c_scenes[slot], rt, nb, n_nb, &counters->errors);
    }
    const uint4 s4 = P.sampler[i];
    PathSampler hs{(uint64_t)s4.x | ((uint64_t)s4.y << 32), X.dim[t], s4.w};
    RayTransfer rt0;
    const PathSampler hs0 = hs;
    if (grid_grads) rt0 = rt;
    const vec3 tr = trace_tr<kF>(slot, st, o, d, o4.w, inst, tri, rt, hs, &counters->errors, &tests, &nodes);
    X.result[t] = make_float4(tr.x, tr.y, tr.z, 1.0f);
    X.dim[t] = hs.dim;
    if (grid_grads) {
      const uint2 pf = P.pixel_flags[i];
      const JobDesc& J = jobs[pf.y >> kFlagJobShift];
      const float inv_spp = 1.0f / gmax(J.setting.ssp, 1);
      const float4 dl = J.dloss[pf.x], t4 = P.throughput[i];
      const vec3 weight = vec3(dl.x, dl.y, dl.z) * inv_spp * vec3(t4.x, t4.y, t4.z);
      const uint4 p0 = X.pass[t], p1 = X.pass[X.capacity + t];
      const vec3 contrib = u2f(p0.x) * tr * vec3(u2f(p0.y), u2f(p0.z), u2f(p0.w)) *
                           vec3(u2f(p1.x), u2f(p1.y), u2f(p1.z));
      const float select_pdf = u2f(X.state[X.capacity + t].w);
      const float mul = distant ? 1.0f : safe_rcp(select_pdf), div = distant ? select_pdf : 1.0f;
      vec3 scale(0.0f);
      if (!volume) scale = weight * (mul / div) * contrib;
      else if (select_pdf > 0.0f) scale = weight * contrib / select_pdf;
      if (max_component(vabs(scale)) > 0.0f) {
        const MediumAdj am{scale, grid_tex, grid_grads};
        hs = hs0;
        trace_tr<kF, true>(slot, st, o, d, o4.w, inst, tri, rt0, hs, &counters->errors, &tests, &nodes, &am);
      }
    }
  }
  for (int off = 16; off > 0; off >>= 1) {
    tests += __shfl_down_sync(0xFFFFFFFFu, tests, off);
    nodes += __shfl_down_sync(0xFFFFFFFFu, nodes, off);
  }
  if ((threadIdx.x & 31) == 0) {
    if (tests) atomicAdd(&counters->shadow_tri_tests, (unsigned long long)tests);
    if (nodes) atomicAdd(&counters->shadow_node_visits, (unsigned long long)nodes);
  }
  if (st.overflow) atomicOr(&counters->errors, (uint32_t)kDevErrStack);
}

// A wave's adjoint shading in phases: k_shade, k_occlude and k_transmit per
// pass, then k_shade's continuation. Returns the launches.
template <bool kVol, uint32_t kF>
uint32_t launch_shade_phases(const WaveArgs& w, const WaveOptions& opt) {
  constexpr uint32_t threads = shade_threads<kVol, false, true, kF>();
  const uint32_t blocks = (w.blocks * kTraceBlock + threads - 1) / threads;
  ShadePhase ph;
  ph.X = opt.vertices;
  ph.kinds = opt.light_kinds;
  ph.passes = ((opt.light_kinds & 1u) ? 2 : 0) + ((opt.light_kinds & 2u) ? 2 : 0);
  uint32_t launches = 0;
  for (ph.phase = 0; ph.phase <= ph.passes; ++ph.phase) {
    k_shade<kVol, false, true, kF><<<blocks, threads, 0, w.stream>>>(w.A, w.ctl, w.H, w.B, w.jobs, w.counters,
                                                                    ShadowQueue{}, opt.grads, opt.grad_materials, ph);
    ++launches;
    if (ph.phase == ph.passes) break;
    k_occlude<(kF & kFeatSpheres) != 0><<<opt.connect_blocks, kTraceBlock, occluded_shared_bytes(kTraceBlock), w.stream>>>(
        ph.X, w.counters, ph.phase);
    ++launches;
    if constexpr (kVol) {
      const bool distant = ph.kinds != 2u && ph.phase < 2;
      k_transmit<kF><<<w.blocks, kTraceBlock, traversal_shared_bytes(kTraceBlock), w.stream>>>(
          ph.X, w.A, w.H, w.jobs, w.counters, ph.phase, distant, opt.grid_grads, opt.grid_tex);
      ++launches;
    }
  }
  return launches;
}

// ------------------------------------------------------------- connect ---
//
// Traces the wave's queued shadow rays and adds each unoccluded ray's
// contribution to its pixel. Persistent (a GPU-sized grid) with warp-level
// work fetch (Aila & Laine, HPG 2009): a lane whose ray is done takes the next
// queued ray at once, one atomic per warp for all its idle lanes, instead of
// waiting for the warp's slowest ray; each loop iteration advances every busy
// lane by one step of its own walk (occluded_step).
template <uint32_t kF>
__global__ void __launch_bounds__(kMaxTraceBlock, kConnectBlocksPerSm * kTraceBlock / kMaxTraceBlock) k_connect(ShadowQueue Q,
                                                                             const JobDesc* __restrict__ jobs,
                                                                             WaveCounters* counters) {
  extern __shared__ __align__(16) uint32_t s_occ[];  // occluded_shared_bytes(blockDim.x)
  OccStack st;
  st.bind(s_occ);
  OccWalk w;
  const uint32_t n = min(counters->shadow_count[Q.turn], Q.capacity);
  const int lane = threadIdx.x & 31;
  uint32_t ray = kEmpty;   // queue index of this lane's ray (kEmpty: idle)
  bool exhausted = false;  // the queue has been handed out (warp-uniform)
  uint32_t tests = 0, nodes = 0;
  for (;;) {
    if (!exhausted) {
      const uint32_t idle = __ballot_sync(0xFFFFFFFFu, ray == kEmpty);
      if (idle) {
        const int leader = __ffs(idle) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(&counters->shadow_cursor[Q.turn], (uint32_t)__popc(idle));
        base = __shfl_sync(0xFFFFFFFFu, base, leader);
        if (base + (uint32_t)__popc(idle) >= n) exhausted = true;
        if (ray == kEmpty) {
          const uint32_t t = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
          if (t < n) {
            const float4 o = Q.o[t], d = Q.d[t];
            const uint32_t job = __float_as_uint(Q.c[t].w);
            w.begin(jobs[job].scene_slot, vec3(o.x, o.y, o.z), vec3(d.x, d.y, d.z), o.w, st);
            ray = t;
          }
        }
      }
    }
    if (__ballot_sync(0xFFFFFFFFu, ray != kEmpty) == 0) break;
    if (ray != kEmpty) {
      const int r = occluded_step<(kF & kFeatSpheres) != 0>(w, st, &tests, &nodes);
      if (r != kWalkGoing) {
        if (r == kWalkClear) {
          const float4 c = Q.c[ray];
          const JobDesc& J = jobs[__float_as_uint(c.w)];
          atomicAdd(J.image + __float_as_uint(Q.d[ray].w), make_float4(c.x, c.y, c.z, 0.0f));
          if (J.path_radiance) {
            // the record holds radiance, the contribution is weighted by 1/spp
            const float spp = (float)gmax(J.setting.ssp, 1);
            atomicAdd(J.path_radiance + Q.path[ray], make_float4(c.x * spp, c.y * spp, c.z * spp, 0.0f));
          }
        }
        ray = kEmpty;
      }
    }
  }
  for (int off = 16; off > 0; off >>= 1) {
    tests += __shfl_down_sync(0xFFFFFFFFu, tests, off);
    nodes += __shfl_down_sync(0xFFFFFFFFu, nodes, off);
  }
  if (lane == 0) {
    if (tests) atomicAdd(&counters->shadow_tri_tests, (unsigned long long)tests);
    if (nodes) atomicAdd(&counters->shadow_node_visits, (unsigned long long)nodes);
  }
  if (st.overflow) atomicOr(&counters->errors, (uint32_t)kDevErrStack);
}

// Scene features a wave kernel is instantiated on. Surface kernels: the
// sphere and texture bits (grids are media). Media kernels: the sphere bit
// and one bit for the full texture node set (grids or the solid nodes beyond
// fBm switch on both). So each runs one of four instantiations.
constexpr uint32_t surface_features(uint32_t f) { return f & (kFeatSpheres | kFeatTextures); }
constexpr uint32_t media_features(uint32_t f) {
  return (f & (kFeatGrids | kFeatTextures)) ? (f | kFeatGrids | kFeatTextures) : (f & kFeatSpheres);
}

// Lets a k_extend instantiation take the dynamic shared memory of a
// kMaxTraceBlock-thread block (more than the default 48 KB).
template <typename K>
static void allow_trace_shared(K kernel) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)traversal_shared_bytes(kMaxTraceBlock));
}

// Writes scenes[k] into this translation unit's constant slot slots[k]
// (k < n; slots == nullptr: slot k).
static cudaError_t upload_slots_here(const DeviceScene* scenes, const uint32_t* slots, uint32_t n,
                                     cudaStream_t stream) {
  if (n > (uint32_t)kMaxBatchScenes) return cudaErrorInvalidValue;
  cudaError_t e = cudaSuccess;
  uint32_t k = 0;
  while (k < n && e == cudaSuccess) {
    // one copy per run of consecutive slots
    const uint32_t first = slots ? slots[k] : k;
    if (first >= (uint32_t)kMaxBatchScenes) return cudaErrorInvalidValue;
    uint32_t run = 1;
    while (k + run < n && (slots ? slots[k + run] : k + run) == first + run) ++run;
    e = cudaMemcpyToSymbolAsync(c_scenes, scenes + k, sizeof(DeviceScene) * run, sizeof(DeviceScene) * first,
                                cudaMemcpyHostToDevice, stream);
    k += run;
  }
  return e;
}

// This translation unit's bound record (dev_bound.cuh), optionally cleared.
static cudaError_t read_bound_here(BoundRecord* out, bool clear, cudaStream_t stream) {
  cudaError_t e = cudaMemcpyFromSymbolAsync(out, g_bound, sizeof(BoundRecord), 0, cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e == cudaSuccess && clear) {
    const BoundRecord zero{};
    e = cudaMemcpyToSymbolAsync(g_bound, &zero, sizeof(zero), 0, cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  }
  return e;
}

}  // namespace ym
