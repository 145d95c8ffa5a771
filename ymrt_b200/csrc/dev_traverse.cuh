// Two-level ray traversal over compressed 8-wide BVHs (sm_100a).
//
// Semantics follow the reference's TraceRay / IntersectMeshObject /
// IntersectTri / IntersectSphereObject / BVHTraverseShadow
// (src/ShadingUtilities.cuh:54-276, 310-431, 563-635): world rays are carried into each instance with the
// instance's inverse transform (glm mat4*vec4 order), triangles are tested
// with the watertight test in the reference's exact float order (so t and the
// barycentrics are bit-identical), a hit is kept when TMIN <= t <= current t
// (a later hit at an equal t replaces the earlier one), and the "nearby hits"
// list for nested media records every instance whose hit lies within two
// ulps of the final t.
//
// The acceleration structure is this project's: each node holds 8 child boxes
// quantised to bytes on a per-node power-of-two grid (80-byte nodes, five
// 128-bit read-only loads), leaves hold up to three triangles stored as three
// float4 vertices (no index indirection), and the traversal stack lives in
// shared memory (spilling to a short local-memory tail). Box tests use fused
// multiply-adds and are widened by a few ulps so that they are conservative:
// they only decide which triangles are tested, never the hit itself.
#pragma once

#include "dev_constants.cuh"
#include "sphere.h"
#include "ymrt_scene.h"

namespace ym {

// Entries per thread in shared memory: what the stacks leave is L1 (the
// instanced 1080p 64-spp frame 188.5 ms at 32, 187.4 at 16; the volumetric
// 1280x720 16-spp one 267 and 263 ms), and few walks go deeper than 16.
constexpr int kStackShared = 16;
constexpr int kStackLocal = 80;   // further entries per thread in local memory
constexpr int kTraceBlock = 128;  // threads per block of the traversal kernels (default)
constexpr int kMaxTraceBlock = 256;  // largest block k_extend and k_connect are launched with

// Stack entries carry the entry distance of the box that produced them, so a
// pop can drop entries that lie beyond the current closest hit. An entry is a
// node index, or (kInstanceEntry set) a group of the one to seven instances of
// a top-level leaf (a node's meta byte has three bits for them): their count
// in bits 28-30 and the first one's leaf slot.
constexpr uint32_t kInstanceEntry = 0x80000000u;
constexpr uint32_t kEntryCountShift = 28, kEntrySlotMask = (1u << kEntryCountShift) - 1u;
static_assert(kMaxInstanceSlots == kEntrySlotMask + 1u, "an entry holds any slot that a scene may have");

struct TraversalStack {
  uint2* sh;  // shared-memory column of this thread: entry, entry distance (stride: the block's threads)
  uint2 loc[kStackLocal];
  int sp;
  int stride;
  bool overflow;
  __device__ __forceinline__ void bind(uint2* shared) {
    sh = shared + threadIdx.x;
    stride = (int)blockDim.x;
    sp = 0;
    overflow = false;
  }
  __device__ __forceinline__ void push(uint32_t v, float t = 0.0f) {
    if (sp < kStackShared) {
      sh[sp * stride] = make_uint2(v, __float_as_uint(t));
    } else if (sp < kStackShared + kStackLocal) {
      loc[sp - kStackShared] = make_uint2(v, __float_as_uint(t));
    } else {
      overflow = true;
      return;
    }
    ++sp;
  }
  __device__ __forceinline__ uint32_t pop(float* t) {
    --sp;
    const uint2 e = sp < kStackShared ? sh[sp * stride] : loc[sp - kStackShared];
    *t = __uint_as_float(e.y);
    return e.x;
  }
  __device__ __forceinline__ uint32_t pop() {
    float t;
    return pop(&t);
  }
};

// Shared-memory backing of the traversal stacks of one kTraceBlock block.
#define YM_TRAVERSAL_SHARED(name) __shared__ uint2 name[kStackShared * kTraceBlock]
// The same, in the dynamic shared memory of a kernel launched with any block
// size (traversal_shared_bytes of it).
#define YM_TRAVERSAL_SHARED_DYNAMIC(name) extern __shared__ __align__(16) uint2 name[]
constexpr size_t traversal_shared_bytes(uint32_t block) { return (size_t)kStackShared * block * 8u; }

// The far end of the box-test interval for a ray whose closest hit so far is
// at t: boxes are widened by 1e-6 relative, and so is this bound, so a box
// entered beyond it cannot hold a hit at or near t.
__device__ __forceinline__ float widened_tmax(float t) { return __fmaf_rn(fabsf(t), 1e-6f, t); }

// Ray set-up shared by every triangle test of one object-space ray: the
// reference recomputes these in each IntersectTri call; they are the same
// numbers each time.
struct TriRay {
  vec3 o, d;
  int kx, ky, kz;
  float sx, sy, sz;
};
__device__ __forceinline__ TriRay make_tri_ray(vec3 o, vec3 d) {
  TriRay r;
  r.o = o;
  r.d = d;
  r.kz = max_dimension(vabs(d));
  r.kx = r.kz + 1; if (r.kx == 3) r.kx = 0;
  r.ky = r.kx + 1; if (r.ky == 3) r.ky = 0;
  const vec3 dd(d[r.kx], d[r.ky], d[r.kz]);
  r.sx = -dd.x / dd.z;
  r.sy = -dd.y / dd.z;
  r.sz = 1.f / dd.z;
  return r;
}

// Watertight ray/triangle test, IntersectTri (src/ShadingUtilities.cuh:54-134).
// Returns false when the edge tests fail; otherwise t (may be outside range)
// and the three unnormalised edge values with 1/den.
__device__ __forceinline__ bool tri_test(const TriRay& R, vec3 p0, vec3 p1, vec3 p2, float* t_out, float* e_out,
                                         float* inv_den_out) {
  p0 = p0 - R.o;
  p1 = p1 - R.o;
  p2 = p2 - R.o;
  p0 = vec3(p0[R.kx], p0[R.ky], p0[R.kz]);
  p1 = vec3(p1[R.kx], p1[R.ky], p1[R.kz]);
  p2 = vec3(p2[R.kx], p2[R.ky], p2[R.kz]);
  p0.x += R.sx * p0.z;
  p0.y += R.sy * p0.z;
  p1.x += R.sx * p1.z;
  p1.y += R.sy * p1.z;
  p2.x += R.sx * p2.z;
  p2.y += R.sy * p2.z;
  const float e0 = p1.x * p2.y - p1.y * p2.x;
  const float e1 = p2.x * p0.y - p2.y * p0.x;
  const float e2 = p0.x * p1.y - p0.y * p1.x;
  if ((e0 < 0 || e1 < 0 || e2 < 0) && (e0 > 0 || e1 > 0 || e2 > 0)) return false;
  const float den = e0 + e1 + e2;
  if (den == 0) return false;
  p0.z *= R.sz;
  p1.z *= R.sz;
  p2.z *= R.sz;
  const float inv = 1.0f / den;
  float t = e0 * p0.z + e1 * p1.z + e2 * p2.z;
  t *= inv;
  *t_out = t;
  e_out[0] = e0;
  e_out[1] = e1;
  e_out[2] = e2;
  *inv_den_out = inv;
  return true;
}

__device__ __forceinline__ void load_tri(const float4* __restrict__ wtris, uint32_t i, vec3* p0, vec3* p1, vec3* p2,
                                         uint32_t* id) {
  const float4 a = __ldg(wtris + 3 * (size_t)i);
  const float4 b = __ldg(wtris + 3 * (size_t)i + 1);
  const float4 c = __ldg(wtris + 3 * (size_t)i + 2);
  *p0 = vec3(a.x, a.y, a.z);
  *p1 = vec3(b.x, b.y, b.z);
  *p2 = vec3(c.x, c.y, c.z);
  *id = __float_as_uint(a.w);
}

// Per-ray constants for box tests.
struct BoxRay {
  float ox, oy, oz, ix, iy, iz;
};
__device__ __forceinline__ BoxRay make_box_ray(vec3 o, vec3 d) {
  BoxRay b;
  b.ox = o.x; b.oy = o.y; b.oz = o.z;
  b.ix = 1.0f / d.x; b.iy = 1.0f / d.y; b.iz = 1.0f / d.z;
  return b;
}

// Byte k of a word as a float.
__device__ __forceinline__ float byte_of(uint32_t w, int k) { return (float)((w >> (8 * k)) & 0xFFu); }

// The low bits of the four bytes' "is not zero", in bits 0-3.
__device__ __forceinline__ uint32_t nonzero_bytes(uint32_t w) {
  const uint32_t high = (((w & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | w) & 0x80808080u;  // the high bit of each nonzero byte
  return ((high >> 7) * 0x10204080u) >> 28;
}

__device__ __forceinline__ uint32_t child_meta(const uint32_t meta[2], int c) {
  return __byte_perm(meta[0], meta[1], (uint32_t)c) & 0xFFu;
}

// Tests the 8 child boxes of a node. Returns a mask of hit children; tnear
// receives each hit child's entry distance. The near and far bounds of an
// axis are chosen for four children at a time, on the words that hold them.
__device__ __forceinline__ uint32_t intersect_children(const uint4* __restrict__ nodes_u4, uint32_t node, const BoxRay& r,
                                                       float tmax, float tnear_out[8], uint32_t* imask,
                                                       uint32_t* child_base, uint32_t* prim_base, uint32_t meta[2]) {
  const uint4* p = nodes_u4 + 5 * (size_t)node;
  const uint4 w0 = __ldg(p), w1 = __ldg(p + 1), w2 = __ldg(p + 2), w3 = __ldg(p + 3), w4 = __ldg(p + 4);
  const float nox = __uint_as_float(w0.x), noy = __uint_as_float(w0.y), noz = __uint_as_float(w0.z);
  const float sx = __uint_as_float((w0.w & 0xFFu) << 23);
  const float sy = __uint_as_float((w0.w << 15) & 0x7F800000u);
  const float sz = __uint_as_float((w0.w << 7) & 0x7F800000u);
  *imask = w0.w >> 24;
  *child_base = w1.x;
  *prim_base = w1.y;
  meta[0] = w1.z;
  meta[1] = w1.w;
  // t = (origin + q * scale - o) * inv = q * (scale * inv) + (origin - o) * inv
  const float ax = sx * r.ix, bx = (nox - r.ox) * r.ix;
  const float ay = sy * r.iy, by = (noy - r.oy) * r.iy;
  const float az = sz * r.iz, bz = (noz - r.oz) * r.iz;
  // byte planes: w2 = qlo_x[0..7], qlo_y[0..7]; w3 = qlo_z, qhi_x; w4 = qhi_y, qhi_z
  const bool negx = r.ix < 0.0f, negy = r.iy < 0.0f, negz = r.iz < 0.0f;
  const uint32_t nx[2] = {negx ? w3.z : w2.x, negx ? w3.w : w2.y}, fx[2] = {negx ? w2.x : w3.z, negx ? w2.y : w3.w};
  const uint32_t ny[2] = {negy ? w4.x : w2.z, negy ? w4.y : w2.w}, fy[2] = {negy ? w2.z : w4.x, negy ? w2.w : w4.y};
  const uint32_t nz[2] = {negz ? w4.z : w3.x, negz ? w4.w : w3.y}, fz[2] = {negz ? w3.x : w4.z, negz ? w3.y : w4.w};
  uint32_t hits = 0;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int k = c & 3, h = c >> 2;
    const float t0x = __fmaf_rn(byte_of(nx[h], k), ax, bx), t1x = __fmaf_rn(byte_of(fx[h], k), ax, bx);
    const float t0y = __fmaf_rn(byte_of(ny[h], k), ay, by), t1y = __fmaf_rn(byte_of(fy[h], k), ay, by);
    const float t0z = __fmaf_rn(byte_of(nz[h], k), az, bz), t1z = __fmaf_rn(byte_of(fz[h], k), az, bz);
    float tn = fmaxf(fmaxf(t0x, t0y), fmaxf(t0z, 0.0f));
    float tf = fminf(fminf(t1x, t1y), fminf(t1z, tmax));
    tn = __fmaf_rn(-fabsf(tn), 1e-6f, tn);
    tf = __fmaf_rn(fabsf(tf), 1e-6f, tf);
    if (tn <= tf) hits |= 1u << c;
    tnear_out[c] = tn;
  }
  return hits & (*imask | nonzero_bytes(meta[0]) | (nonzero_bytes(meta[1]) << 4));
}

// The stack entry of child c of a node: its node, or (a top-level leaf) its
// group of instances.
__device__ __forceinline__ uint32_t child_entry(int c, uint32_t imask, const uint32_t meta[2], uint32_t child_base,
                                                uint32_t prim_base) {
  const uint32_t m = child_meta(meta, c);
  return ((imask >> c) & 1u) ? child_base + m
                             : (kInstanceEntry | ((m >> 5) << kEntryCountShift) | (prim_base + (m & 31u)));
}

// Sends the walk on to the children in `mask` near to far: the nearest
// becomes the entry to visit next (kEmpty: none), the others go on the stack,
// the farthest first, each with its entry distance. Children are ordered by
// keys that hold the entry distance (non-negative, so its bits order like the
// float) with the child slot in the low three bits, plus one; misses are 0.
// Taking the greatest key again and again is a short loop with one copy of
// the push: with the register-held next entry it replaced a 19-comparator
// network with ten inlined pushes (the walk's code 53 -> 24 KB; closest hits
// of the instanced 1080p 64-spp frame 116 -> 100 ms, shading of the volumetric
// 1280x720 16-spp frame, which traces inline, 222 -> 199 ms).
__device__ __forceinline__ uint32_t push_children(TraversalStack& st, uint32_t mask, const float tnear[8],
                                                  uint32_t imask, const uint32_t meta[2], uint32_t child_base,
                                                  uint32_t prim_base, float* next_t) {
  if (mask == 0) return kEmpty;
  uint32_t key[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) key[c] = ((mask >> c) & 1u) ? ((__float_as_uint(tnear[c]) & ~7u) | (uint32_t)c) + 1u : 0u;
#pragma unroll 1
  for (int left = __popc(mask);; --left) {
    uint32_t hi = key[0];
#pragma unroll
    for (int c = 1; c < 8; ++c) hi = max(hi, key[c]);
    const uint32_t e = child_entry((int)((hi - 1u) & 7u), imask, meta, child_base, prim_base);
    const float t = __uint_as_float((hi - 1u) & ~7u);
    if (left == 1) {
      *next_t = t;
      return e;
    }
    st.push(e, t);
#pragma unroll
    for (int c = 0; c < 8; ++c) key[c] = key[c] == hi ? 0u : key[c];
  }
}

// An instance slot as the traversal reads it, and the object-space ray (one
// record instead of the instance -> transform -> geometry chain: closest hits
// of the instanced 1080p 64-spp frame 100.0 -> 98.6 ms, of Cornell 256x256 16
// spp 1.107 -> 1.070 ms, shadow rays of the former 28.2 -> 27.2 ms).
struct EnteredInstance {
  uint32_t inst, node_offset, wtri_offset, flags;
  vec3 o, d;
};
__device__ __forceinline__ EnteredInstance enter_instance(const InstanceSlot* __restrict__ slots, uint32_t slot, vec3 wo,
                                                          vec3 wd) {
  const float4* p = reinterpret_cast<const float4*>(slots + slot);
  const uint4 w = __ldg(reinterpret_cast<const uint4*>(p + 3));
  EnteredInstance e;
  e.inst = w.x;
  e.node_offset = w.y;
  e.wtri_offset = w.z;
  e.flags = w.w;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    // glm mat4 * vec4 (xform_point_glm, xform_dir_glm)
    const float4 m = __ldg(p + r);
    e.o[r] = (m.x * wo.x + m.y * wo.y) + (m.z * wo.z + m.w * 1.0f);
    e.d[r] = (m.x * wd.x + m.y * wd.y) + (m.z * wd.z + m.w * 0.0f);
  }
  return e;
}

// Sphere tests of the traversals, kept out of line so that their registers do
// not weigh on the triangle loop that surrounds them.
struct SphereTest {
  float t, px, py, pz;  // the hit, when hit != 0
  float xt;             // the extra crossing, when xhit != 0
  int hit, back, xhit, xback;
};
static __device__ __noinline__ SphereTest sphere_instance_test(float radius, vec3 o, vec3 d, float t_max) {
  SphereHit h{0.0f, vec3(0.0f), 0};
  SphereExtra x{false, kTMax, 0};
  SphereTest r;
  r.hit = sphere_intersect(radius, o, d, t_max, &h, &x);
  r.t = h.t;
  r.px = h.p.x;
  r.py = h.p.y;
  r.pz = h.p.z;
  r.back = h.back;
  r.xhit = x.hit;
  r.xt = x.t;
  r.xback = x.back;
  return r;
}
static __device__ __noinline__ bool sphere_occludes(float radius, vec3 o, vec3 d, float t_max) {
  SphereHit h;
  SphereExtra x;
  return sphere_intersect(radius, o, d, t_max, &h, &x);
}

// Results of one step of a resumable walk (ClosestWalk, occluded_step).
constexpr int kWalkGoing = 0, kWalkOccluded = 1, kWalkClear = 2;

struct NearbyHit {
  uint32_t prim;
  float t;
  int back;
};

struct ClosestHit {
  float t;
  float b0, b1, b2;
  uint32_t inst, tri;
  int back;
  int nearby_count;
  NearbyHit nearby[kMaxNearby];
};

// Closest hit of one world-space ray (TraceRay, src/ShadingUtilities.cuh:310-431)
// in the scene of constant-memory slot `scene`, as a resumable walk: one
// step() visits one node or enters one instance, so a persistent kernel can
// advance the lanes of a warp on different rays (k_extend); trace_closest_impl
// runs the steps to the end.
// kVolumeOnly: traverse only treat_as_boundary instances (TraceVolume, :434-561).
//
// One loop serves both levels: each step takes one entry -- a top-level node,
// an instance to enter, or a bottom-level node of the current instance -- so
// the lanes of a warp run the same node code whatever level they are in.
// Instance leaves are ordered by distance with the internal nodes,
// bottom-level leaves are tested at once, and entries whose box begins beyond
// the closest hit so far are dropped when taken.
//
// kSpheres: the scene holds sphere geometry. The walk without sphere code is a
// separate instantiation, so scenes of meshes alone keep its register
// allocation (the sphere branch costs the triangle loop about 5%).
template <bool kSpheres, bool kVolumeOnly>
struct ClosestWalk {
  uint32_t slot;
  vec3 wo, wd;
  BoxRay wray;
  uint32_t last_inst, last_tri;
  bool skip_enabled, hit;
  float t_ray, t_upper, t_lower;
  int n_nearby;
  uint32_t next;  // the entry to visit before the stack's (kEmpty: none), its entry distance
  float next_t;
  // the instance being traversed (inst_base < 0: none)
  int inst_base;
  uint32_t inst_idx, wtri_offset;
  vec3 od;
  TriRay tr;
  BoxRay br;
  bool skip_here, inst_hit, inst_sphere;
  float inst_t, hb0, hb1, hb2, extra_t;
  // hit_w / extra_w: the wide-BVH slot of the hit / extra triangle, or for a
  // sphere (inst_sphere) the back-face flag of its hit / extra crossing
  uint32_t hit_tri, hit_w, extra_w;

  __device__ __forceinline__ void begin(uint32_t scene, TraversalStack& st, vec3 o, vec3 d, float tmax,
                                        uint32_t li, uint32_t lt) {
    slot = scene;
    wo = o;
    wd = d;
    wray = make_box_ray(o, d);
    last_inst = li;
    last_tri = lt;
    skip_enabled = li != kEmpty && lt != kEmpty;
    hit = false;
    t_ray = tmax;
    t_upper = t_lower = 0.0f;
    n_nearby = 0;
    inst_base = -1;
    inst_idx = wtri_offset = 0;
    od = vec3(0.0f);
    br = wray;
    skip_here = inst_hit = inst_sphere = false;
    inst_t = hb0 = hb1 = hb2 = 0.0f;
    extra_t = kTMax;
    hit_tri = kEmpty;
    hit_w = 0;
    extra_w = kEmpty;
    st.sp = 0;
    next = 0;
    next_t = 0.0f;
  }

  // Leaving the instance: its hit (and the nearby-hit list) into `out`.
  __device__ __forceinline__ void leave_instance(const DeviceScene& S, ClosestHit* out) {
    NearbyHit* nb = out->nearby;
    if (inst_hit) {
      int back;
      if (kSpheres && inst_sphere) {
        back = (int)hit_w;
      } else {
        vec3 p0, p1, p2;
        uint32_t tid;
        load_tri(S.wtris, hit_w, &p0, &p1, &p2, &tid);
        const vec3 ng = normalize(cross(p1 - p0, p2 - p0));
        back = dot(ng, od) > 0.0f;
      }
      out->t = inst_t;
      out->b0 = hb0;
      out->b1 = hb1;
      out->b2 = hb2;
      out->inst = inst_idx;
      out->tri = hit_tri;
      out->back = back;
      hit = true;
      t_upper = next_float_up(next_float_up(t_ray));
      t_lower = next_float_down(next_float_down(t_ray));
      int head = 0, tail = n_nearby - 1;
      while (head <= tail) {
        if (nb[head].t > t_lower && nb[head].t < t_upper) ++head;
        else {
          const NearbyHit tmp = nb[head];
          nb[head] = nb[tail];
          nb[tail] = tmp;
          --tail;
        }
      }
      n_nearby = head;
      if (n_nearby < kMaxNearby) nb[n_nearby++] = NearbyHit{inst_idx, inst_t, back};
    } else if (hit && extra_w != kEmpty && extra_t > t_lower && extra_t < t_upper) {
      int back;
      if (kSpheres && inst_sphere) {
        back = (int)extra_w;
      } else {
        vec3 p0, p1, p2;
        uint32_t tid;
        load_tri(S.wtris, extra_w, &p0, &p1, &p2, &tid);
        const vec3 ng = normalize(cross(p1 - p0, p2 - p0));
        back = dot(ng, od) > 0.0f;
      }
      if (n_nearby < kMaxNearby) nb[n_nearby++] = NearbyHit{inst_idx, extra_t, back};
    }
    inst_base = -1;
  }

  // One step; kWalkGoing while entries remain, else kWalkClear (the walk is
  // over: `hit` says whether `out` holds a hit; out->nearby_count is set).
  __device__ __forceinline__ int step(TraversalStack& st, ClosestHit* out, uint32_t* tri_tests,
                                      uint32_t* node_visits) {
    const DeviceScene& S = c_scenes[slot];
    uint32_t e = next;
    float etn = next_t;
    next = kEmpty;
    if (e == kEmpty) {
      if (inst_base >= 0 && st.sp == inst_base) leave_instance(S, out);
      if (st.sp == 0) {
        out->nearby_count = n_nearby;
        return kWalkClear;
      }
      e = st.pop(&etn);
    }
    if (etn > widened_tmax(t_ray)) return kWalkGoing;
    if (e & kInstanceEntry) {
      // the group's last instance now, the others after it
      const uint32_t count = (e >> kEntryCountShift) & 7u, at = e & kEntrySlotMask;
      if (count > 1) st.push(e - (1u << kEntryCountShift), etn);
      const EnteredInstance in = enter_instance(S.inst_slots, at + count - 1, wo, wd);
      if (kVolumeOnly && !(in.flags & kSlotBoundary)) return kWalkGoing;
      inst_idx = in.inst;
      const vec3 oo = in.o;
      od = in.d;
      if (kSpheres && (in.flags & kSlotSphere)) {
        // a sphere is tested at once and left at the next step; its hit
        // point travels in the barycentric slots and its triangle is EMPTY
        ++*tri_tests;
        const SphereTest q = sphere_instance_test(u2f(in.wtri_offset), oo, od, t_ray);
        inst_sphere = true;
        inst_hit = q.hit != 0;
        if (inst_hit) {
          t_ray = q.t;
          inst_t = q.t;
          hb0 = q.px;
          hb1 = q.py;
          hb2 = q.pz;
          hit_tri = kEmpty;
          hit_w = (uint32_t)q.back;
        }
        extra_t = q.xhit ? q.xt : kTMax;
        extra_w = q.xhit ? (uint32_t)q.xback : kEmpty;
        inst_base = st.sp;
        return kWalkGoing;
      }
      inst_sphere = false;
      tr = make_tri_ray(oo, od);
      br = make_box_ray(oo, od);
      wtri_offset = in.wtri_offset;
      skip_here = skip_enabled && inst_idx == last_inst;
      inst_hit = false;
      extra_t = kTMax;
      extra_w = kEmpty;
      inst_base = st.sp;
      e = in.node_offset;  // continue with the instance's root in this step
    }
    const bool in_blas = inst_base >= 0;
    const uint32_t node = e;
    ++*node_visits;
    float tn[8];
    uint32_t imask, cbase, pbase, meta[2];
    const uint32_t hits = intersect_children(reinterpret_cast<const uint4*>(in_blas ? S.blas_nodes : S.tlas_nodes), e,
                                             in_blas ? br : wray, t_ray, tn, &imask, &cbase, &pbase, meta);
    uint32_t leaves = hits & ~imask;
    if (in_blas) {
      while (leaves) {
        const int c = __ffs(leaves) - 1;
        leaves &= leaves - 1;
        const uint32_t m = child_meta(meta, c);
        const uint32_t cnt = m >> 5, off = m & 31u;
        for (uint32_t q = 0; q < cnt; ++q) {
          const uint32_t wi = wtri_offset + pbase + off + q;
          vec3 p0, p1, p2;
          uint32_t tid;
          load_tri(S.wtris, wi, &p0, &p1, &p2, &tid);
          if (skip_here && tid == last_tri) continue;
          float t, ev[3], inv;
          ++*tri_tests;
          if (!tri_test(tr, p0, p1, p2, &t, ev, &inv)) continue;
          if (t >= kTMin && t < extra_t) {
            extra_t = t;
            extra_w = wi;
          }
          if (t < kTMin || t > t_ray) continue;
          t_ray = t;
          inst_hit = true;
          inst_t = t;
          hb0 = ev[0] * inv;
          hb1 = ev[1] * inv;
          hb2 = ev[2] * inv;
          hit_tri = tid;
          hit_w = wi;
        }
      }
    }
    uint32_t go = in_blas ? hits & imask : hits;
    if (kVolumeOnly && !in_blas) go &= __ldg(S.tlas_kinds + node);
    next = push_children(st, go, tn, imask, meta, cbase, pbase, &next_t);
    return kWalkGoing;
  }
};

// The whole walk of one ray (see ClosestWalk).
template <bool kSpheres, bool kVolumeOnly>
static __device__ __noinline__ bool trace_closest_impl(uint32_t scene, TraversalStack& st, vec3 wo, vec3 wd,
                                                       float tmax, uint32_t last_inst, uint32_t last_tri,
                                                       ClosestHit* out, uint32_t* tri_tests, uint32_t* node_visits) {
  ClosestWalk<kSpheres, kVolumeOnly> w;
  w.begin(scene, st, wo, wd, tmax, last_inst, last_tri);
  while (w.step(st, out, tri_tests, node_visits) == kWalkGoing) {
  }
  return w.hit;
}

// Closest hit of one world-space ray in the scene of constant-memory slot
// `scene` (see trace_closest_impl). Out of line, so that its callers keep one
// call site whichever instantiation runs.
static __device__ __noinline__ bool trace_closest(uint32_t scene, TraversalStack& st, vec3 wo, vec3 wd, float tmax,
                                              uint32_t last_inst, uint32_t last_tri, ClosestHit* out,
                                              uint32_t* tri_tests, uint32_t* node_visits) {
  if (c_scenes[scene].sphere_count != 0)
    return trace_closest_impl<true, false>(scene, st, wo, wd, tmax, last_inst, last_tri, out, tri_tests, node_visits);
  return trace_closest_impl<false, false>(scene, st, wo, wd, tmax, last_inst, last_tri, out, tri_tests, node_visits);
}

// ------------------------------------------------ resumable occlusion walk ---
//
// Any hit within (TMIN, tmax] ignoring boundary-only instances
// (BVHTraverseShadow, src/ShadingUtilities.cuh:563-635), cut into steps, so
// that a persistent kernel can advance the lanes of a warp on different rays
// and hand a finished lane its next ray at once (k_connect). One step enters
// an instance and visits its root, or visits one node: its child boxes are
// tested, the triangles of its leaf children tested, one other child kept to
// visit next and the rest pushed (unordered: any hit ends the query). Stack
// entries need no entry distance here, so k_connect's stack is entries only.
constexpr int kOccStackShared = 32;  // entries per thread in shared memory
constexpr int kConnectBlocksPerSm = 8;  // at kTraceBlock threads (the register budget of the launch bounds)
constexpr size_t occluded_shared_bytes(uint32_t block) { return (size_t)kOccStackShared * block * 4u; }

struct OccStack {
  uint32_t* sh;  // shared-memory column of this thread (stride: the block's threads)
  uint32_t loc[kStackLocal];
  int sp;
  int stride;
  bool overflow;
  __device__ __forceinline__ void bind(uint32_t* shared_entries) {
    sh = shared_entries + threadIdx.x;
    stride = (int)blockDim.x;
    sp = 0;
    overflow = false;
  }
  __device__ __forceinline__ void push(uint32_t v) {
    if (sp < kOccStackShared) sh[sp * stride] = v;
    else if (sp < kOccStackShared + kStackLocal) loc[sp - kOccStackShared] = v;
    else {
      overflow = true;
      return;
    }
    ++sp;
  }
  __device__ __forceinline__ uint32_t pop() {
    --sp;
    return sp < kOccStackShared ? sh[sp * stride] : loc[sp - kOccStackShared];
  }
};

struct OccWalk {
  uint32_t slot;       // scene slot
  vec3 wo, wd;         // world ray
  float tmax;
  BoxRay wray;
  uint32_t next;       // the entry to visit before the stack's (kEmpty: none)
  int inst_base;       // stack depth below the current instance's entries (-1: top level)
  uint32_t wtri_offset;
  TriRay tr;           // the current instance's object-space ray
  BoxRay br;
  template <typename Stack>
  __device__ __forceinline__ void begin(uint32_t scene, vec3 o, vec3 d, float t_max, Stack& st) {
    slot = scene;
    wo = o;
    wd = d;
    tmax = t_max;
    wray = make_box_ray(o, d);
    inst_base = -1;
    st.sp = 0;
    next = 0;
  }
};

template <bool kSpheres, typename Stack>
__device__ __forceinline__ int occluded_step(OccWalk& w, Stack& st, uint32_t* tri_tests, uint32_t* node_visits) {
  const DeviceScene& S = c_scenes[w.slot];
  uint32_t e = w.next;
  w.next = kEmpty;
  if (e == kEmpty) {
    if (w.inst_base >= 0 && st.sp == w.inst_base) w.inst_base = -1;
    if (st.sp == 0) return kWalkClear;
    e = st.pop();
  }
  if (e & kInstanceEntry) {
    const uint32_t count = (e >> kEntryCountShift) & 7u, at = e & kEntrySlotMask;
    if (count > 1) st.push(e - (1u << kEntryCountShift));
    const EnteredInstance in = enter_instance(S.inst_slots, at + count - 1, w.wo, w.wd);
    if (in.flags & kSlotBoundary) return kWalkGoing;
    if (kSpheres && (in.flags & kSlotSphere)) {
      ++*tri_tests;
      return sphere_occludes(u2f(in.wtri_offset), in.o, in.d, w.tmax) ? kWalkOccluded : kWalkGoing;
    }
    w.tr = make_tri_ray(in.o, in.d);
    w.br = make_box_ray(in.o, in.d);
    w.wtri_offset = in.wtri_offset;
    w.inst_base = st.sp;
    e = in.node_offset;
  }
  const bool in_blas = w.inst_base >= 0;
  ++*node_visits;
  float tn[8];
  uint32_t imask, cbase, pbase, meta[2];
  const uint32_t hits = intersect_children(reinterpret_cast<const uint4*>(in_blas ? S.blas_nodes : S.tlas_nodes), e,
                                           in_blas ? w.br : w.wray, w.tmax, tn, &imask, &cbase, &pbase, meta);
  if (in_blas) {
    uint32_t leaves = hits & ~imask;
    while (leaves) {
      const int c = __ffs(leaves) - 1;
      leaves &= leaves - 1;
      const uint32_t m = child_meta(meta, c);
      const uint32_t cnt = m >> 5, off = m & 31u;
      for (uint32_t q = 0; q < cnt; ++q) {
        vec3 p0, p1, p2;
        uint32_t tid;
        load_tri(S.wtris, w.wtri_offset + pbase + off + q, &p0, &p1, &p2, &tid);
        float t, ev[3], inv;
        ++*tri_tests;
        if (!tri_test(w.tr, p0, p1, p2, &t, ev, &inv)) continue;
        if (t < kTMin || t > w.tmax) continue;
        return kWalkOccluded;
      }
    }
  }
  uint32_t go = in_blas ? hits & imask : hits;
  if (!in_blas && S.boundary_count != 0) go &= __ldg(S.tlas_kinds + e) >> 8;
  while (go) {
    const int c = __ffs(go) - 1;
    go &= go - 1;
    if (w.next != kEmpty) st.push(w.next);
    w.next = child_entry(c, imask, meta, cbase, pbase);
  }
  return kWalkGoing;
}

// The whole occlusion query of one ray.
template <bool kSpheres>
__device__ __noinline__ bool trace_occluded_impl(uint32_t scene, TraversalStack& st, vec3 wo, vec3 wd, float tmax,
                                                 uint32_t* tri_tests, uint32_t* node_visits) {
  OccWalk w;
  w.begin(scene, wo, wd, tmax, st);
  int r;
  do r = occluded_step<kSpheres>(w, st, tri_tests, node_visits);
  while (r == kWalkGoing);
  st.sp = 0;
  return r == kWalkOccluded;
}

static __device__ __noinline__ bool trace_occluded(uint32_t scene, TraversalStack& st, vec3 wo, vec3 wd, float tmax,
                                               uint32_t* tri_tests, uint32_t* node_visits) {
  if (c_scenes[scene].sphere_count != 0) return trace_occluded_impl<true>(scene, st, wo, wd, tmax, tri_tests, node_visits);
  return trace_occluded_impl<false>(scene, st, wo, wd, tmax, tri_tests, node_visits);
}

}  // namespace ym
