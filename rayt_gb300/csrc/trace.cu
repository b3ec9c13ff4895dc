// Tracing passes, the hot path: traversal of the rays of one or many views
// against the block cache, plus the reference's debug depth view.
//
// Per ray this fuses what the reference runs as separate full-frame kernels
// with a 48-byte TracingState round trip through memory:
//   ray setup       InitTracingFrame   (rayt/GPU_renderer/kernels/init_tracing_frame.cl:11-45)
//   traversal       CastRay            (rayt/GPU_renderer/kernels/raycast.cl:33-256)
//   pass logic      RaytracingPass     (rayt/GPU_renderer/kernels/raytracing_pass.cl:4-61)
//   shading         ProcessHit         (rayt/GPU_renderer/kernels/shading.cl:4-33)
//   final colour    FinishTracingFrame (rayt/GPU_renderer/kernels/finish_tracing_frame.cl:3-24)
//   block words     NodeToBlockKernel  (rayt/GPU_renderer/kernels/feedback_compression.cl:4-13)
//
// Kernels:
//   trace_kernel             one ray per lane: first passes over the 32-pixel
//                            tiles of all views of the launch (4x8 by default;
//                            lane i of a tile = pixel (i % tile_w, i / tile_w)),
//                            later passes over the compacted list of rays that
//                            faulted; small launches give a warp fewer rays
//   trace_persistent_kernel  first pass with work stealing: warps stop their
//                            rays every step_budget iterations and refill idle
//                            lanes (an autotuner candidate; slower on the
//                            measured workloads, see the design notes)
//   finish_kernel            FinishTracingFrame for rays still faulted
//   depth_view_kernel        raytracer.cl, the reference's debug depth view
//   unique_from_bits_kernel  the feedback bitmaps as the reference's sorted
//                            unique array
// A ray that ends (hit, miss, iteration limit) writes its final RGBA8 pixel;
// a ray that faults on a missing block is appended with its state (advanced
// origin, direction, parent node, pixel) to the next pass's list.  Feedback
// goes into two bitmaps (fault blocks; hit cache blocks with the duplicate
// flag).
//
// FP32 arithmetic follows the reference's operation order exactly; the file is
// compiled with --fmad=false and IEEE division/sqrt so no operation is fused or
// approximated, which keeps hit node IDs identical to the CPU oracle.
#include <algorithm>

#include "internal.h"

namespace rayt {
namespace {

constexpr int kSMax = 23;
constexpr float kEps = 0.00000011920928955078125f;  // exp2(-S_MAX)
constexpr int kIterLimit = 300;
constexpr int kBlockThreads = 128;
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ float dot4(float ax, float ay, float az, float aw, float bx, float by, float bz, float bw) {
  float r = ax * bx;
  r = r + ay * by;
  r = r + az * bz;
  r = r + aw * bw;
  return r;
}

// 0 / d as an IEEE division gives it: a zero with d's sign, NaN for a zero
// or NaN d.
__device__ __forceinline__ float zero_over(float d) {
  return (d == 0.0f || d != d) ? __int_as_float(0x7fffffff) : copysignf(0.0f, d);
}

// mul(float16, float3) of init_tracing_frame.cl:3-9
__device__ __forceinline__ void mul_point(const float* m, float x, float y, float z, float* o) {
  float d = dot4(x, y, z, 1.0f, m[12], m[13], m[14], m[15]);
  o[0] = __fdiv_rn(dot4(x, y, z, 1.0f, m[0], m[1], m[2], m[3]), d);
  o[1] = __fdiv_rn(dot4(x, y, z, 1.0f, m[4], m[5], m[6], m[7]), d);
  o[2] = __fdiv_rn(dot4(x, y, z, 1.0f, m[8], m[9], m[10], m[11]), d);
  o[3] = zero_over(d);
}

// InitTracingFrame for pixel (x, y) of view v.  The view's origin and its
// normalised pixel coordinates come precomputed (the same IEEE operations,
// done once per view and per column/row instead of per ray).
__device__ __forceinline__ void init_direction(const ViewDesc& v, int x, int y, float4& o, float4& d) {
  const float* m = v.m;
  const int W = v.width;
  const float* cx = v.coords;          // (x + 0.5) / W * 2 - 1
  const float* cy = cx + W + W + 1;    // (y + 0.5) / H * 2 - 1
  const float ox = v.origin[0], oy = v.origin[1], oz = v.origin[2], ow = v.origin[3];
  float q[4];
  mul_point(m, __ldg(cx + x), __ldg(cy + y), 0.0f, q);
  float dx = q[0] - ox, dy = q[1] - oy, dz = q[2] - oz, dw = q[3] - ow;
  float len = __fsqrt_rn(dot4(dx, dy, dz, dw, dx, dy, dz, dw));
  dx = __fdiv_rn(dx, len);
  dy = __fdiv_rn(dy, len);
  dz = __fdiv_rn(dz, len);
  o = make_float4(ox, oy, oz, 0.0f);
  d = make_float4(dx, dy, dz, 0.0f);
}
// The direction's fourth component: the voxel size that counts as one pixel,
// per unit of distance.
__device__ __forceinline__ float init_coef(const ViewDesc& v, int x, int y) {
  const float* m = v.m;
  const int W = v.width, H = v.height;
  const float* ax = v.coords + W;      // x / W * 2 - 1, x in [0, W]
  const float* ay = ax + W + 1 + H;    // y / H * 2 - 1, y in [0, H]
  const float ox = v.origin[0], oy = v.origin[1], oz = v.origin[2], ow = v.origin[3];
  float p1[4], p2[4];
  mul_point(m, __ldg(ax + x), __ldg(ay + y), 0.0f, p1);
  mul_point(m, __ldg(ax + x + 1), __ldg(ay + y + 1), 0.0f, p2);
  float bx = p1[0] - p2[0], by = p1[1] - p2[1], bz = p1[2] - p2[2], bw = p1[3] - p2[3];
  float ex = ox - p1[0], ey = oy - p1[1], ez = oz - p1[2], ew = ow - p1[3];
  float dist12 = __fsqrt_rn(dot4(bx, by, bz, bw, bx, by, bz, bw));
  float dist01 = __fsqrt_rn(dot4(ex, ey, ez, ew, ex, ey, ez, ew));
  return __fdiv_rn(v.lod * dist12, dist01);
}
__device__ __forceinline__ void init_ray(const ViewDesc& v, int x, int y, float4& o, float4& d) {
  init_direction(v, x, y, o, d);
  d.w = init_coef(v, x, y);
}

// CastRay (raycast.cl:33-256) split into cast_begin() (everything before its
// while loop) and cast_run() (the loop, for a bounded number of iterations),
// so a warp can stop its rays at a common point and hand idle lanes new rays.
// The state is the reference's loop state; the outcome is encoded in it
// (see Outcome) instead of extra result registers.
struct Cast {
  float tx_coef, ty_coef, tz_coef, tx_bias, ty_bias, tz_bias;
  float t_min, t_max, h, px, py, pz, scale_exp2, coef, bias;
  uint32_t parent, desc;
  int idx, scale, octant, iter;
};

// How cast_run left a ray.  kHit: node = parent, duplicate flag = bit 9 of
// desc.  kFault: node = parent, t = t_min, block = desc >> 11.
enum Outcome : int { kRunning = 0, kHit = 1, kFault = 2, kMiss = 3, kError = 4 };

__device__ __forceinline__ void cast_begin(Cast& c, uint32_t root, float4 o, float4 d) {
  float px0 = o.x + 1.0f, py0 = o.y + 1.0f, pz0 = o.z + 1.0f;
  float dx = d.x, dy = d.y, dz = d.z;
  c.coef = d.w;
  c.bias = o.w;
  if (fabsf(dx) < kEps) dx = copysignf(kEps, dx);
  if (fabsf(dy) < kEps) dy = copysignf(kEps, dy);
  if (fabsf(dz) < kEps) dz = copysignf(kEps, dz);
  c.tx_coef = __fdiv_rn(1.0f, -fabsf(dx));
  c.ty_coef = __fdiv_rn(1.0f, -fabsf(dy));
  c.tz_coef = __fdiv_rn(1.0f, -fabsf(dz));
  c.tx_bias = c.tx_coef * px0;
  c.ty_bias = c.ty_coef * py0;
  c.tz_bias = c.tz_coef * pz0;
  c.octant = 0;
  if (dx > 0.0f) c.octant ^= 1, c.tx_bias = 3.0f * c.tx_coef - c.tx_bias;
  if (dy > 0.0f) c.octant ^= 2, c.ty_bias = 3.0f * c.ty_coef - c.ty_bias;
  if (dz > 0.0f) c.octant ^= 4, c.tz_bias = 3.0f * c.tz_coef - c.tz_bias;
  c.t_min = fmaxf(fmaxf(2.0f * c.tx_coef - c.tx_bias, 2.0f * c.ty_coef - c.ty_bias), 2.0f * c.tz_coef - c.tz_bias);
  c.t_max = fminf(fminf(c.tx_coef - c.tx_bias, c.ty_coef - c.ty_bias), c.tz_coef - c.tz_bias);
  c.h = c.t_max;
  c.t_min = fmaxf(c.t_min, 0.0f);
  c.parent = root;
  c.desc = 0;
  c.idx = 0;
  c.px = 1.0f;
  c.py = 1.0f;
  c.pz = 1.0f;
  c.scale = kSMax - 1;
  c.scale_exp2 = 0.5f;
  if (1.5f * c.tx_coef - c.tx_bias > c.t_min) c.idx ^= 1, c.px = 1.5f;
  if (1.5f * c.ty_coef - c.ty_bias > c.t_min) c.idx ^= 2, c.py = 1.5f;
  if (1.5f * c.tz_coef - c.tz_bias > c.t_min) c.idx ^= 4, c.pz = 1.5f;
  c.iter = 0;
}

// How a ray ended.  error: iteration limit or a corrupt cache; fault_block
// != -1: the children of `node` are not loaded (t = where the ray stopped);
// node == -1: miss; else a hit on `node` with the duplicate flag `dup`.
struct RayEnd {
  float t;
  int node, fault_block, dup, error;
  int iter;
};

// CastRay as one function over local state, for rays that run to their end
// in one go (the one-thread-per-ray kernel).  The arithmetic and stack rules
// are cast_begin + cast_run's; kept as a single loop with the reference's
// shape because that form compiles to about 5% fewer warp instructions on
// sm_103a than the resumable one.
// kBias: the ray may have an LOD bias (origins that were advanced, the depth
// view); first-pass rays start with a bias of zero.
//
// kLazy: the direction comes without its fourth component, a quarter of what a
// first-pass ray takes to set up, and the ray asks `late_coef` for it before it
// first enters a child.  The rays that leave through empty children of the
// root never do (all the rays of half the warps of a frame that looks past
// the scene's edge: 1919x1079 pixels with nothing in sight 42.5 -> 28.2 us,
// 512x512 60.6 -> 58.9, a frame full of the scene 321.4 -> 324.2).
//
// The lanes meet again where they have found their child of the root: left to
// the compiler, those that found it after as many steps stayed together, and
// a warp went through the traversal in such parts.  That hardly cost cameras
// whose root children are met in the same step (512x512 59.0 us, 59.1 with the
// meeting; the most it costs one is 2%, or 1 us of a 128x96 frame's 11 with little
// in sight), and others a quarter (512x512 85.5 and 69.2 us, 1919x1079 199 and
// 175, 500 views of 32x32 203 and 156).
template <bool kCount, bool kBias, bool kLazy, class F>
__device__ __forceinline__ RayEnd cast_ray(const TraceCore& p, float4 o, float4& d, uint32_t& fetches,
                                           uint32_t& far_fetches, const F& late_coef) {
  RayEnd r;
  r.fault_block = -1;
  r.error = 0;
  r.dup = 0;
  const float px0 = o.x + 1.0f, py0 = o.y + 1.0f, pz0 = o.z + 1.0f;
  float dx = d.x, dy = d.y, dz = d.z;
  float coef = d.w;
  const float bias = o.w;
  // (parent, t_max, the parent's descriptor): a pop needs no reload of the
  // descriptor, which no pass changes (1.7% off the first pass)
  uint4 stack[kSMax + 1];
  if (fabsf(dx) < kEps) dx = copysignf(kEps, dx);
  if (fabsf(dy) < kEps) dy = copysignf(kEps, dy);
  if (fabsf(dz) < kEps) dz = copysignf(kEps, dz);
  const float tx_coef = __fdiv_rn(1.0f, -fabsf(dx));
  const float ty_coef = __fdiv_rn(1.0f, -fabsf(dy));
  const float tz_coef = __fdiv_rn(1.0f, -fabsf(dz));
  float tx_bias = tx_coef * px0, ty_bias = ty_coef * py0, tz_bias = tz_coef * pz0;
  int octant = 0;
  if (dx > 0.0f) octant ^= 1, tx_bias = 3.0f * tx_coef - tx_bias;
  if (dy > 0.0f) octant ^= 2, ty_bias = 3.0f * ty_coef - ty_bias;
  if (dz > 0.0f) octant ^= 4, tz_bias = 3.0f * tz_coef - tz_bias;
  float t_min = fmaxf(fmaxf(2.0f * tx_coef - tx_bias, 2.0f * ty_coef - ty_bias), 2.0f * tz_coef - tz_bias);
  float t_max = fminf(fminf(tx_coef - tx_bias, ty_coef - ty_bias), tz_coef - tz_bias);
  float h = t_max;
  t_min = fmaxf(t_min, 0.0f);
  uint32_t parent = (uint32_t)p.root, desc = 0;
  int idx = 0;
  float px = 1.0f, py = 1.0f, pz = 1.0f;
  int scale = kSMax - 1;
  float scale_exp2 = 0.5f;
  if (1.5f * tx_coef - tx_bias > t_min) idx ^= 1, px = 1.5f;
  if (1.5f * ty_coef - ty_bias > t_min) idx ^= 2, py = 1.5f;
  if (1.5f * tz_coef - tz_bias > t_min) idx ^= 4, pz = 1.5f;
  int iter = 0;
  // Every parent is the root or a child index clamped below node_limit, so
  // only the root needs a check (a root outside the cache ends the ray as an
  // error, like the iteration limit).
  if (p.root >= p.node_limit) {
    r.error = 1;
    r.node = -1;
    r.t = 0.0f;
    r.iter = 0;
    return r;
  }
  // The parent's descriptor is in hand where the reference's loop will need
  // it: fetched here for the root, and taken from the stack entry at each pop
  // (raycast.cl fetches it at the top of the next iteration, which always
  // follows a pop; same value, one fewer test per iteration).  The counting
  // form keeps the reference's fetch points so its counts equal the oracle's.
  if (!kCount) desc = __ldg(p.links + parent);
  // `child` holds 31 minus the mirrored child index (the reference's
  // idx ^ octant, the child's flag in the descriptor): shifted left by it, a
  // descriptor has that child's flag on top and only the flags below it under
  // it, so one shift serves the test and the count of the children before it
  // (1.5-2% off the first pass against a mask for each).
  const int mirror = 31 ^ octant;
  int child = mirror ^ idx;
  if (kLazy) {  // the loop below, as long as no child of the root is entered
    const unsigned here = __activemask();
    bool missed = false;
    while (!((int)(desc << child) < 0 && t_min <= t_max)) {
      const float tx_corner = px * tx_coef - tx_bias;
      const float ty_corner = py * ty_coef - ty_bias;
      const float tz_corner = pz * tz_coef - tz_bias;
      const float tc_max = fminf(fminf(tx_corner, ty_corner), tz_corner);
      const int before = child;
      if (tx_corner <= tc_max) child ^= 1, px = px - 0.5f;
      if (ty_corner <= tc_max) child ^= 2, py = py - 0.5f;
      if (tz_corner <= tc_max) child ^= 4, pz = pz - 0.5f;
      t_min = tc_max;
      ++iter;
      // Every step turns an axis over, and one that turned over before leaves the
      // octree, so this ends within four steps.  A ray all of whose corner
      // distances are NaN (a NaN in its matrix, or an origin at infinity, m[14] =
      // 0) steps along no axis: it ends at the limit of the loop below, as an
      // error.  (That test here instead: a full frame 324 us, so 331.)
      if (child == before) break;
      if (((child ^ mirror) & (child ^ before)) != 0) {  // out of the octree: a miss
        missed = true;
        break;
      }
    }
    __syncwarp(here);
    if (missed) {
      r.node = -1;
      r.iter = iter;
      return r;
    }
    d.w = coef = late_coef();
  }
  for (;;) {  // left by a hit, a fault, the iteration limit or a pop past the root
    if (++iter > kIterLimit) {
      r.error = 1;
      break;
    }
    if (kCount && desc == 0) {
      desc = __ldg(p.links + parent);
      ++fetches;
    }
    const float tx_corner = px * tx_coef - tx_bias;
    const float ty_corner = py * ty_coef - ty_bias;
    const float tz_corner = pz * tz_coef - tz_bias;
    const float tc_max = fminf(fminf(tx_corner, ty_corner), tz_corner);
    const uint32_t flags = desc << child;
    if ((int)flags < 0 && t_min <= t_max) {
      if (desc & (1u << 8)) {  // children not loaded: fault
        r.node = (int)parent;
        r.t = t_min;
        r.fault_block = (int)(desc >> 11);
        break;
      }
      // Both indices below are clamped into their buffers instead of tested
      // (a test ends the ray as an error, a branch out of the loop that costs
      // 9% of the first pass).  On a cache this library filled neither clamp
      // ever acts: child links are checked to stay inside their block before
      // upload, and far pointers are written by the cache itself.
      const uint32_t pdesc = desc;
      uint32_t ofs;
      if (desc & (1u << 10)) {
        ofs = __ldg(p.far_ptrs + min(desc >> 11, p.far_limit - 1u));
        if (kCount) ++far_fetches;
      } else {
        ofs = (desc >> 11) + parent - (1u << 20);
      }
      ofs = min(ofs + __popc(flags) - 1u, p.node_limit - 1u);
      desc = __ldg(p.links + ofs);
      if (kCount) ++fetches;
      // without a bias the sum differs from the product in a zero's sign only
      const float voxel = kBias ? tc_max * coef + bias : tc_max * coef;
      if (!(desc & 255u) || scale == 0 || voxel >= scale_exp2) {
        r.t = t_min;
        r.node = (int)ofs;
        r.dup = (int)((desc >> 9) & 1u);
        break;
      }
      // half is a power of two (at least 2^-24) and |coef| is about 1 or
      // more, so half * coef is exact and the fused sum rounds as the
      // reference's multiply and add do
      const float half = scale_exp2 * 0.5f;
      const float tx_center = fmaf(half, tx_coef, tx_corner);
      const float ty_center = fmaf(half, ty_coef, ty_corner);
      const float tz_center = fmaf(half, tz_coef, tz_corner);
      if (tc_max < h) stack[scale] = make_uint4(parent, __float_as_uint(t_max), pdesc, 0u);
      h = tc_max;
      parent = ofs;
      --scale;
      scale_exp2 = half;
      child = mirror;
      if (tx_center > t_min) child ^= 1, px = px + half;
      if (ty_center > t_min) child ^= 2, py = py + half;
      if (tz_center > t_min) child ^= 4, pz = pz + half;
      t_max = tc_max;
      continue;
    }
    const bool sx = tx_corner <= tc_max, sy = ty_corner <= tc_max, sz = tz_corner <= tc_max;
    const int before = child;
    if (sx) child ^= 1, px = px - scale_exp2;
    if (sy) child ^= 2, py = py - scale_exp2;
    if (sz) child ^= 4, pz = pz - scale_exp2;
    t_min = tc_max;
    if (((child ^ mirror) & (child ^ before)) != 0) {  // idx & step: out of the parent
      uint32_t diff = 0;
      if (sx) diff |= (uint32_t)(__float_as_int(px) ^ __float_as_int(px + scale_exp2));
      if (sy) diff |= (uint32_t)(__float_as_int(py) ^ __float_as_int(py + scale_exp2));
      if (sz) diff |= (uint32_t)(__float_as_int(pz) ^ __float_as_int(pz + scale_exp2));
      scale = 31 - __clz((int)diff);  // the highest bit that changed
      if (scale >= kSMax) {           // left the octree: a miss
        r.node = -1;
        break;
      }
      scale_exp2 = __int_as_float((scale - kSMax + 127) << 23);
      const uint4 e = stack[scale];
      parent = e.x;
      t_max = __uint_as_float(e.y);
      desc = kCount ? 0u : e.z;  // the parent's descriptor, needed next iteration
      const uint32_t shx = __float_as_uint(px) >> scale;
      const uint32_t shy = __float_as_uint(py) >> scale;
      const uint32_t shz = __float_as_uint(pz) >> scale;
      px = __uint_as_float(shx << scale);
      py = __uint_as_float(shy << scale);
      pz = __uint_as_float(shz << scale);
      child = mirror ^ (int)((shx & 1u) | ((shy & 1u) << 1) | ((shz & 1u) << 2));
      h = 0.0f;
    }
  }
  r.iter = iter;
  return r;
}

// CastRay's loop until the ray ends or (kBudget) its iteration count reaches
// `stop` <= kIterLimit (kRunning: the ray continues from there on the next
// call).  The loop runs on local copies of the state, written back once at
// the end, and leaves through one exit.
// A node at scale 0 ends the ray like a leaf: its children would lie below
// float resolution and below the stack, which only a tree deeper than 23
// levels reaches (the reference reads and writes past its stack there).  So
// every stack index stays in [0, 22].
template <bool kCount, bool kBudget>
__device__ __forceinline__ int cast_run(Cast& c, int stop, uint2* stack, const TraceCore& p, uint32_t& fetches,
                                        uint32_t& far_fetches) {
  const float tx_coef = c.tx_coef, ty_coef = c.ty_coef, tz_coef = c.tz_coef;
  const float tx_bias = c.tx_bias, ty_bias = c.ty_bias, tz_bias = c.tz_bias;
  const float coef = c.coef, bias = c.bias;
  const int octant = c.octant;
  float t_min = c.t_min, t_max = c.t_max, h = c.h, px = c.px, py = c.py, pz = c.pz, scale_exp2 = c.scale_exp2;
  uint32_t parent = c.parent, desc = c.desc;
  int idx = c.idx, scale = c.scale, iter = c.iter;
  int outcome = kMiss;
  while (scale < kSMax) {
    if (++iter > (kBudget ? stop : kIterLimit)) {
      if (!kBudget || iter > kIterLimit) {
        outcome = kError;
      } else {
        --iter;
        outcome = kRunning;
      }
      break;
    }
    if (desc == 0) {
      if (parent >= p.node_limit) {  // only reachable from a corrupt cache
        outcome = kError;
        break;
      }
      desc = __ldg(p.links + parent);
      if (kCount) ++fetches;
    }
    const float tx_corner = px * tx_coef - tx_bias;
    const float ty_corner = py * ty_coef - ty_bias;
    const float tz_corner = pz * tz_coef - tz_bias;
    const float tc_max = fminf(fminf(tx_corner, ty_corner), tz_corner);
    const uint32_t bit = 1u << (idx ^ octant);
    if ((desc & bit) != 0 && t_min <= t_max) {
      if (desc & (1u << 8)) {  // children not loaded
        outcome = kFault;
        break;
      }
      uint32_t ofs;  // indices clamped into their buffers, as in cast_ray
      if (desc & (1u << 10)) {
        ofs = __ldg(p.far_ptrs + min(desc >> 11, p.far_limit - 1u));
        if (kCount) ++far_fetches;
      } else {
        ofs = (desc >> 11) + parent - (1u << 20);
      }
      ofs = min(ofs + __popc(desc & (bit - 1) & 255u), p.node_limit - 1u);
      desc = __ldg(p.links + ofs);
      if (kCount) ++fetches;
      if (!(desc & 255u) || scale == 0 || tc_max * coef + bias >= scale_exp2) {
        parent = ofs;
        outcome = kHit;
        break;
      }
      const float half = scale_exp2 * 0.5f;
      const float tx_center = half * tx_coef + tx_corner;
      const float ty_center = half * ty_coef + ty_corner;
      const float tz_center = half * tz_coef + tz_corner;
      if (tc_max < h) stack[scale] = make_uint2(parent, __float_as_uint(t_max));
      h = tc_max;
      parent = ofs;
      idx = 0;
      --scale;
      scale_exp2 = half;
      if (tx_center > t_min) idx ^= 1, px = px + scale_exp2;
      if (ty_center > t_min) idx ^= 2, py = py + scale_exp2;
      if (tz_center > t_min) idx ^= 4, pz = pz + scale_exp2;
      t_max = tc_max;
      continue;
    }
    int step = 0;
    if (tx_corner <= tc_max) step ^= 1, px = px - scale_exp2;
    if (ty_corner <= tc_max) step ^= 2, py = py - scale_exp2;
    if (tz_corner <= tc_max) step ^= 4, pz = pz - scale_exp2;
    t_min = tc_max;
    idx ^= step;
    if ((idx & step) != 0) {
      uint32_t diff = 0;
      if (step & 1) diff |= (uint32_t)(__float_as_int(px) ^ __float_as_int(px + scale_exp2));
      if (step & 2) diff |= (uint32_t)(__float_as_int(py) ^ __float_as_int(py + scale_exp2));
      if (step & 4) diff |= (uint32_t)(__float_as_int(pz) ^ __float_as_int(pz + scale_exp2));
      // (float)diff is exact (diff < 2^23), so its exponent is the top bit
      scale = (__float_as_int((float)diff) >> 23) - 127;
      // popping past the root ends the loop (the reference reads one more
      // stack entry first, whose value it never uses)
      if (scale >= kSMax) break;
      scale_exp2 = __int_as_float((scale - kSMax + 127) << 23);
      const uint2 e = stack[scale];
      parent = e.x;
      t_max = __uint_as_float(e.y);
      const uint32_t shx = __float_as_uint(px) >> scale;
      const uint32_t shy = __float_as_uint(py) >> scale;
      const uint32_t shz = __float_as_uint(pz) >> scale;
      px = __uint_as_float(shx << scale);
      py = __uint_as_float(shy << scale);
      pz = __uint_as_float(shz << scale);
      idx = (int)((shx & 1u) | ((shy & 1u) << 1) | ((shz & 1u) << 2));
      h = 0.0f;
      desc = 0;
    }
  }
  c.t_min = t_min;
  c.t_max = t_max;
  c.h = h;
  c.px = px;
  c.py = py;
  c.pz = pz;
  c.scale_exp2 = scale_exp2;
  c.parent = parent;
  c.desc = desc;
  c.idx = idx;
  c.scale = scale;
  c.iter = iter;
  return outcome;
}

// x / 127 correctly rounded for an integer x in [-128, 127] (a char normal
// component): the product with the rounded reciprocal, then one FMA-exact
// residual correction.  Equal to the IEEE quotient for all 256 inputs (a CPU
// test checks every one); a fifth of a full-range division's instructions.
__device__ __forceinline__ float div127(float x) {
  const float r = 1.0f / 127.0f;
  const float q0 = x * r;
  const float e = fmaf(-q0, 127.0f, x);
  return fmaf(e, r, q0);
}

// ProcessHit: fixed ambient + three directional lights; returns RGBA8 (A=255).
__device__ __forceinline__ uchar4 shade(const TraceCore& p, uint32_t node) {
  const char4 cn = p.normals[node];
  // the reference's w component is 0 / 127 = +0
  const float nx = div127((float)cn.x), ny = div127((float)cn.y), nz = div127((float)cn.z), nw = 0.0f;
  // The light directions (shading.cl:7-32): normalize(v) * w for v, w =
  // (2,-2,3), .6; (-3,-3,-2), .5; (1,2.5,-1), .3, each as the reference
  // computes it per call in IEEE float (dot left to right, correctly rounded
  // sqrt and divisions, then the product).  Constants, so no ray pays for 3
  // square roots and 9 divisions; a CPU test recomputes them.
  const float l[3][3] = {{0x1.2a071ep-2f, -0x1.2a071ep-2f, 0x1.bf0aacp-2f},
                         {-0x1.4779eep-2f, -0x1.4779eep-2f, -0x1.b4a294p-3f},
                         {0x1.abd032p-4f, 0x1.0b6220p-2f, -0x1.abd032p-4f}};
  float a[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float dd = dot4(-nx, -ny, -nz, -nw, l[k][0], l[k][1], l[k][2], 0.0f);
    a[k] = 0.f < dd ? dd : 0.f;
  }
  const float light = ((.1f + a[0] * 1.f) + a[1] * 1.f) + a[2] * 1.f;
  const uchar4 cc = p.colors[node];
  float c0 = (float)cc.x * light, c1 = (float)cc.y * light, c2 = (float)cc.z * light;
  c0 = c0 < 255.f ? c0 : 255.f;
  c1 = c1 < 255.f ? c1 : 255.f;
  c2 = c2 < 255.f ? c2 : 255.f;
  return make_uchar4((unsigned char)c0, (unsigned char)c1, (unsigned char)c2, 255);
}

// FinishTracingFrame's blend of the accumulated colour over the background,
// for a pixel nothing was accumulated in (alpha 0): the same for every such
// pixel, so the host computes it (finish_empty).  An opaque pixel (hits,
// errors) is left as it is: w = 255 - 255 = 0 adds a zero, and c + .5 truncates
// to c.
__device__ __forceinline__ uchar4 shaded(const TraceCore& p, uint32_t node) {
  return p.normals && p.colors ? shade(p, node) : p.empty_pixel;
}

// Appends `pred` lanes of the active warp to a global list: returns this
// lane's slot (or -1).
__device__ __forceinline__ int warp_append(int* counter, bool pred) {
  const unsigned active = __activemask();
  const unsigned mask = __ballot_sync(active, pred);
  if (!mask) return -1;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(mask) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(counter, __popc(mask));
  base = __shfl_sync(active, base, leader);
  return pred ? base + __popc(mask & ((1u << lane) - 1)) : -1;
}

// Sets bit `bit` (>= 0) of a bitmap, one atomic per distinct word in the warp:
// the lanes of a word OR their bits in one reduction, word by word (a tile's
// hits lie in one or two words), then each word's first lane looks whether
// they are all set already, all words at once.
__device__ __forceinline__ void warp_set_bit(uint32_t* bits, int bit) {
  const unsigned active = __activemask();
  const int lane = threadIdx.x & 31;
  const int word = bit >> 5;  // negative: no bit
  const unsigned m = 1u << (bit & 31);
  unsigned todo = __ballot_sync(active, bit >= 0);
  unsigned mine = 0;
  while (todo) {
    const int leader = __ffs(todo) - 1;
    const bool same = word == __shfl_sync(active, word, leader);
    const unsigned acc = __reduce_or_sync(active, same ? m : 0u);
    if (lane == leader) mine = acc;
    todo &= ~__ballot_sync(active, same);
  }
  if (mine && (__ldcg(bits + word) & mine) != mine) atomicOr(bits + word, mine);
}

// Notes that the lanes `none` of the warp ended without a feedback word (the unique array
// then ends with NO_HIT).  Only warps with such a ray touch a flag, and only
// the first of them write it: a count of the words was one atomic per warp on
// one address.
__device__ __forceinline__ void mark_no_word(const TraceCore& p, unsigned none) {
  int* flag = p.words->no_word + (blockIdx.x % kNoWordFlags) * kNoWordStride;
  if (none && (int)(threadIdx.x & 31) == __ffs(none) - 1 && __ldcg(flag) == 0) *flag = 1;
}

// View of the launch holding tile `tile` (tile_base is ascending).
template <class P>
__device__ __forceinline__ int view_of_tile(const P& p, int tile) {
  int lo = 0, hi = p.n_views - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (p.views[mid].tile_base <= tile) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Served mode: the client slot owning pixel `ray` (client_base ascending).
__device__ __forceinline__ int slot_of(const TraceCore& p, uint32_t ray) {
  int lo = 0, hi = p.n_clients - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((uint32_t)p.client_base[mid] <= ray) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Pixel (x, y) and view of first-pass ray r (tile r / 32, lane r % 32);
// false for the lanes of a partial tile that fall outside the view.
// kOneTile: the warp's rays lie in one tile, and so in one view; the reduction's
// result is one for the warp, so that the view is read through uniform loads
// (12 views 2% faster).  Work stealing hands a warp rays from any offset on,
// of two tiles and two views.
template <bool kOneTile, class P>
__device__ __forceinline__ bool first_pass_pixel(const P& p, int r, int& v, int& x, int& y) {
  const int tile = (int)(r >> 5), k = (int)(r & 31);
  if (sizeof(P) == sizeof(TraceParams1)) v = 0;
  else if (kOneTile) v = (int)__reduce_max_sync(__activemask(), (unsigned)view_of_tile(p, tile));
  else v = view_of_tile(p, tile);
  const ViewDesc& vd = p.views[v];
  const int t = tile - vd.tile_base;
  // t / tiles_x: the product with the reciprocal rounded up is the quotient or
  // one more (its excess over t / tiles_x is below t / 2^32), with the largest
  // word for 1 / 1 one less
  int row = (int)__umulhi((uint32_t)t, vd.tiles_x_inv), col = t - row * vd.tiles_x;
  if (col < 0) --row, col += vd.tiles_x;
  if (col >= vd.tiles_x) ++row, col -= vd.tiles_x;
  x = (col << p.tile_w_log2) + (k & ((1 << p.tile_w_log2) - 1));
  y = row * (32 >> p.tile_w_log2) + (k >> p.tile_w_log2);
  return x < vd.width && y < vd.height;
}

// kBudget: warps stop their rays every step_budget iterations and refill idle
// lanes once `refill` of them are idle; otherwise a warp takes new rays once
// all 32 ended.
// Ray r of the launch (first pass: tile r / 32 of the views; later passes:
// record r of the input list): its pixel, origin, direction and (depth
// output) the distance it advanced in earlier passes; false for the lanes of
// a partial tile that fall outside their view.
template <bool kFirst, bool kLazy, bool kOneTile, class P>
__device__ __forceinline__ bool ray_at(const P& p, int r, uint32_t& ray, float4& o, float4& d,
                                       float& adv, int& v, int& x, int& y) {
  adv = 0.0f;
  if (kFirst) {
    if (!first_pass_pixel<kOneTile>(p, r, v, x, y)) return false;
    const ViewDesc& vd = p.views[v];
    if (kLazy) init_direction(vd, x, y, o, d);
    else init_ray(vd, x, y, o, d);
    ray = (uint32_t)(vd.pix_base + y * vd.width + x);
  } else {
    o = p.in_origin[r];
    d = p.in_dir[r];
    ray = p.in_ray[r];
    if (p.in_adv) adv = p.in_adv[r];
  }
  return true;
}

// Depth output of a pixel whose ray ended: the distance along the ray to what
// the pixel shows (earlier passes' advances plus this pass's t, in float, in
// pass order) and the cache node that shaded it.  Miss: +inf and -1; error
// (iteration limit, corrupt cache): NaN and -2.
__device__ __forceinline__ void write_depth(const TraceCore& p, uint32_t ray, float depth, int node) {
  p.depth[ray] = depth;
  p.hit_node[ray] = node;
}
constexpr uint32_t kDepthNaN = 0x7fffffffu;
constexpr uint32_t kDepthInf = 0x7f800000u;

// A final pixel: into the image, and into the caller's host image when the
// renderer delivers one (later passes and the finish; the first pass's pixels
// reach it by one copy).
__device__ __forceinline__ void put_pixel(const TraceCore& p, uint32_t ray, uchar4 px) {
  p.image[ray] = px;
  if (p.host_image) p.host_image[ray] = px;
}

// RaytracingPass's handling of an ended ray (raytracing_pass.cl:20-58) plus
// FinishTracingFrame for rays that end here: the final pixel, the next pass's
// record of a faulted ray, the feedback bitmaps and counters.  Called by the
// lanes whose rays ended, together.
template <bool kCount>
__device__ __forceinline__ void end_ray(const TraceCore& p, const RayEnd& e, uint32_t ray, float4 o, const float4 d,
                                        float adv, uint32_t fetches, uint32_t far_fetches) {
  const int lane = threadIdx.x & 31;
  const bool faulted = !e.error && e.fault_block != -1;
  const bool hit = !e.error && e.fault_block == -1 && e.node != -1;
  const int node = e.node, dup = e.dup, fault_block = e.fault_block;
  int32_t word = kNoHit;
  if (e.error) {
    put_pixel(p, ray, make_uchar4(255, 0, 0, 255));
    if (p.depth) write_depth(p, ray, __uint_as_float(kDepthNaN), -2);
  } else if (faulted) {
    word = -fault_block - 1;
  } else if (!hit) {
    put_pixel(p, ray, p.empty_pixel);
    if (p.depth) write_depth(p, ray, __uint_as_float(kDepthInf), -1);
  } else {
    put_pixel(p, ray, shaded(p, (uint32_t)node));
    word = (int32_t)(((uint32_t)(node + 1) << 1) | (uint32_t)dup);
    if (p.depth) write_depth(p, ray, adv + e.t, node);
  }
  if (p.words_dense) p.words_dense[ray] = word;
  // what no ray of the warp needs is passed over together
  const unsigned here = __activemask();
  const unsigned faults = __ballot_sync(here, faulted), hits = __ballot_sync(here, hit);
  if (faults) {
    const int slot = warp_append(&p.words->rays, faulted);
    if (faulted) {
      if (!p.restart) {  // origin moved to the fault (raytracing_pass.cl:37-41)
        o.x = o.x + d.x * e.t;
        o.y = o.y + d.y * e.t;
        o.z = o.z + d.z * e.t;
        o.w = o.w + d.w * e.t;
      }
      if (p.client_faults) atomicAdd(p.client_faults + slot_of(p, ray), 1);
      p.out_origin[slot] = o;
      p.out_dir[slot] = d;
      p.out_parent[slot] = node;
      p.out_ray[slot] = ray;
      if (p.out_adv) p.out_adv[slot] = p.restart ? adv : adv + e.t;
    }
    warp_set_bit(p.fault_bits, faulted && fault_block < p.fault_bit_limit ? fault_block : -1);
  }
  if (hits) {
    const uint32_t block =
        p.block_shift >= 0 ? (uint32_t)node >> p.block_shift : (uint32_t)node / (uint32_t)p.nodes_in_block;
    warp_set_bit(p.hit_bits, hit ? (int)(2 * block) + dup : -1);
  }
  mark_no_word(p, here & ~(faults | hits));
  if (kCount) {
    const unsigned v[6] = {1u, fetches, far_fetches, (unsigned)e.iter, hit ? 1u : 0u, faulted ? 1u : 0u};
    const unsigned active = __activemask();
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const unsigned sum = __reduce_add_sync(active, v[k]);
      if (lane == __ffs(active) - 1) atomicAdd(p.counters + k, (unsigned long long)sum);
    }
  }
}

// One ray per lane, p.lanes of them per warp, over a grid that covers the
// launch's rays: the first pass's 32-ray tiles, or (kFirst false) the rays
// that faulted in the pass before.
// 10 CTAs per SM: at 48 registers; 9 at the 52 it would take are 3% slower on
// 1919x1079 frames.
template <bool kFirst, bool kCount, class P>
__global__ void __launch_bounds__(kBlockThreads, 10) trace_kernel(const __grid_constant__ P p) {
  if (p.stamp && blockIdx.x == 0 && threadIdx.x == 0) p.words->start_ns = global_ns();
  const int total = kFirst ? p.total_tiles * 32 : *p.n_in;
  const int lane = threadIdx.x & 31;
  const int r = (blockIdx.x * (kBlockThreads / 32) + (threadIdx.x >> 5)) * p.lanes + lane;
  if (lane >= p.lanes || r >= total) return;
  uint32_t ray;
  float4 o, d;
  float adv;
  int v = 0, x = 0, y = 0;
  constexpr bool kLazy = kFirst && !kCount;
  if (!ray_at<kFirst, kLazy, true>(p, r, ray, o, d, adv, v, x, y)) return;
  if (!kFirst && p.finish_mask && ((p.finish_mask >> slot_of(p, ray)) & 1ull)) {
    // served mode: the request stops here; FinishTracingFrame's shading with
    // the fault's parent node
    put_pixel(p, ray, shaded(p, (uint32_t)p.in_parent[r]));
    if (p.depth) write_depth(p, ray, adv, p.in_parent[r]);
    mark_no_word(p, __activemask());
    return;
  }
  uint32_t fetches = 0, far_fetches = 0;
  const RayEnd e = cast_ray<kCount, !kFirst, kLazy>(p, o, d, fetches, far_fetches, [&] {
    return init_coef(p.views[v], x, y);
  });
  end_ray<kCount>(p, e, ray, o, d, adv, fetches, far_fetches);
}

// Persistent form: one CTA per SM slot; every warp takes rays from the
// launch's work counter.  A warp runs its rays for step_budget iterations at a
// time and, once at least `refill` of its lanes sit idle (refill = 32: all of
// them), hands those lanes the next rays, so lanes do not idle through the
// warp's longest ray.  Once the counter is exhausted the rays run to the end.
template <bool kFirst, bool kCount>
__global__ void __launch_bounds__(kBlockThreads) trace_persistent_kernel(const __grid_constant__ TraceParams p) {
  if (p.stamp && blockIdx.x == 0 && threadIdx.x == 0) p.words->start_ns = global_ns();
  __shared__ float4 s_origin[kBlockThreads], s_dir[kBlockThreads];
  const int lane = threadIdx.x & 31;
  const int total = kFirst ? p.total_tiles * 32 : *p.n_in;  // below 2^31: at most 2^30 pixels
  uint2 stack[kSMax + 1];
  Cast c;
  int outcome = kRunning;
  uint32_t ray = 0;
  float adv = 0.0f;
  bool have = false, exhausted = false;
  uint32_t fetches = 0, far_fetches = 0;

  for (;;) {
    const unsigned idle = __ballot_sync(kFull, !have);
    if (!exhausted && __popc(idle) >= p.refill) {
      const int want = __popc(idle);
      const int leader = __ffs(idle) - 1;
      int base = 0;
      if (lane == leader) base = atomicAdd(p.work, want);
      base = __shfl_sync(kFull, base, leader);
      if (base + want >= total) exhausted = true;
      if (!have) {
        const int r = base + __popc(idle & ((1u << lane) - 1));
        float4 o, d;
        int v, x, y;
        if (r < total && ray_at<kFirst, false, false>(p, r, ray, o, d, adv, v, x, y)) {
          s_origin[threadIdx.x] = o;  // kept for the ray's fault record
          s_dir[threadIdx.x] = d;
          cast_begin(c, p.root, o, d);
          have = true;
          fetches = far_fetches = 0;
        }
      }
    }
    if (!__ballot_sync(kFull, have)) {
      if (exhausted) break;
      continue;
    }
    if (have && outcome == kRunning) {
      const int stop = exhausted ? kIterLimit : min(c.iter + p.step_budget, kIterLimit);
      outcome = cast_run<kCount, true>(c, stop, stack, p, fetches, far_fetches);
    }
    if (outcome != kRunning) {
      RayEnd e;
      e.t = c.t_min;
      e.node = outcome == kMiss ? -1 : (int)c.parent;
      e.fault_block = outcome == kFault ? (int)(c.desc >> 11) : -1;
      e.dup = (int)((c.desc >> 9) & 1u);
      e.error = outcome == kError;
      e.iter = c.iter;
      end_ray<kCount>(p, e, ray, s_origin[threadIdx.x], s_dir[threadIdx.x], adv, fetches, far_fetches);
      have = false;
      outcome = kRunning;
    }
  }
}

// FinishTracingFrame for rays still faulted at the end of the frame: shade
// with the fault's parent node as the cache holds it now.  Depth output: the
// distance at which the ray stopped and that parent node.
__global__ void __launch_bounds__(kBlockThreads) finish_kernel(const __grid_constant__ TraceCore p) {
  const int i = blockIdx.x * kBlockThreads + threadIdx.x;
  if (i >= *p.n_in) return;
  put_pixel(p, p.in_ray[i], shaded(p, (uint32_t)p.in_parent[i]));
  if (p.depth) write_depth(p, p.in_ray[i], p.in_adv[i], p.in_parent[i]);
}

// Copies finished frames to host memory beside the traversal of the clients
// after them.  Eight CTAs already fill the host link (187 of 189 GB/s), and
// leave the SMs to the traversal.
constexpr int kDeliverCtas = 8, kDeliverThreads = 512;
__global__ void __launch_bounds__(kDeliverThreads) deliver_kernel(const __grid_constant__ DeliverParams p) {
  for (int k = 0; k < p.images; ++k) {
    if (p.faults[p.at[k].slot] != 0) continue;
    const int64_t units = p.at[k].pixels / 4;  // 16 bytes; both addresses are 256-byte aligned
    const uint4* a = reinterpret_cast<const uint4*>(p.at[k].image);
    uint4* b = reinterpret_cast<uint4*>(p.at[k].host);
    for (int64_t i = blockIdx.x * kDeliverThreads + threadIdx.x; i < units; i += kDeliverCtas * kDeliverThreads)
      b[i] = a[i];
    const int64_t i = units * 4 + threadIdx.x;
    if (blockIdx.x == 0 && i < p.at[k].pixels) p.at[k].host[i] = p.at[k].image[i];
  }
}

// raytracer.cl:18-71 (RaytraceKernel, the reference's debug depth view) for
// view 0 of the parameters: rays from the near plane, one pass over the cache
// as it is, no feedback.  Red for a fault or an error, black for a miss, else
// grey = 255 * (1 - log-depth in [0.01, 5]) clamped to [0, 255] (the
// reference's float-to-uchar conversion is undefined outside that range).
__global__ void __launch_bounds__(kBlockThreads) depth_view_kernel(const __grid_constant__ TraceParams1 p) {
  const ViewDesc& v = p.views[0];
  const int W = v.width, H = v.height;
  const int i = blockIdx.x * kBlockThreads + threadIdx.x;
  if (i >= W * H) return;
  const int x = i % W, y = i / W;
  const float cx = __fdiv_rn(x + 0.5f, (float)W) * 2 - 1, cy = __fdiv_rn(y + 0.5f, (float)H) * 2 - 1;
  float o[4], q[4], p1n[4], p1f[4], p2n[4], p2f[4];
  mul_point(v.m, cx, cy, -1.0f, o);
  mul_point(v.m, cx, cy, 0.0f, q);
  float dx = q[0] - o[0], dy = q[1] - o[1], dz = q[2] - o[2], dw = q[3] - o[3];
  const float len = __fsqrt_rn(dot4(dx, dy, dz, dw, dx, dy, dz, dw));
  dx = __fdiv_rn(dx, len);
  dy = __fdiv_rn(dy, len);
  dz = __fdiv_rn(dz, len);
  const float ax = __fdiv_rn((float)x, (float)W) * 2 - 1, ay = __fdiv_rn((float)y, (float)H) * 2 - 1;
  const float bx = __fdiv_rn((float)(x + 1), (float)W) * 2 - 1, by = __fdiv_rn((float)(y + 1), (float)H) * 2 - 1;
  mul_point(v.m, ax, ay, -1.0f, p1n);
  mul_point(v.m, ax, ay, 0.0f, p1f);
  mul_point(v.m, bx, by, -1.0f, p2n);
  mul_point(v.m, bx, by, 0.0f, p2f);
  auto dist = [](const float* a, const float* b) {
    const float ex = a[0] - b[0], ey = a[1] - b[1], ez = a[2] - b[2], ew = a[3] - b[3];
    return __fsqrt_rn(dot4(ex, ey, ez, ew, ex, ey, ez, ew));
  };
  const float bias = v.lod * dist(p1n, p2n);
  const float coef = bias < 1e-10f ? 0.0f : __fdiv_rn(v.lod * (dist(p1f, p2f) - dist(p1n, p2n)), dist(p1n, p1f));
  uint32_t fetches = 0, far_fetches = 0;
  float4 dir = make_float4(dx, dy, dz, coef);
  const RayEnd e = cast_ray<false, true, false>(p, make_float4(o[0], o[1], o[2], bias), dir, fetches, far_fetches,
                                                [] { return 0.0f; });
  uchar4 c;
  if (e.error || e.fault_block != -1) {
    c = make_uchar4(255, 0, 0, 255);
  } else if (e.node == -1) {
    c = make_uchar4(0, 0, 0, 255);
  } else {
    const float near_ = 0.01f, far_ = 5.0f;
    float d = __fdiv_rn(logf(e.t) - logf(near_), logf(far_) - logf(near_));
    d = (1 - d) * 255;
    d = fminf(255.0f, fmaxf(0.0f, d));
    const unsigned char g = (unsigned char)d;
    c = make_uchar4(g, g, g, 255);
  }
  p.image[i] = c;
}

__global__ void fill_kernel(int* p, int32_t v, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}

// Bitmaps -> [faults by descending block][hits ascending][NO_HIT], the order
// of the reference's sorted unique array.  One CTA; each thread owns a run of
// bitmap words in output order, reads them once (up to kUniqKeep of them are
// kept) and leaves them zero.  It also takes the pass's counters, clears those
// of the pass before and publishes the result to the host, which is what lets
// a pass do without a memset before it and event records and a stream
// synchronisation after it: those took 16 us of a frame's 27 us outside its
// kernels.
constexpr int kUniqThreads = 1024;
constexpr int kUniqKeep = 8;
__global__ void __launch_bounds__(kUniqThreads) unique_from_bits_kernel(const UniqueFromBitsParams q) {
  __shared__ int warp_sums[32];
  __shared__ int fsum;
  const unsigned long long begin_ns = global_ns();
  const int total = q.fault_words + q.hit_words;
  const int per = (total + kUniqThreads - 1) / kUniqThreads;
  const int begin = min(total, (int)threadIdx.x * per), end = min(total, begin + per);
  auto word_ptr = [&](int k) -> uint32_t* {
    return k < q.fault_words ? q.fault_bits + (q.fault_words - 1 - k) : q.hit_bits + (k - q.fault_words);
  };
  uint32_t kept[kUniqKeep];
#pragma unroll
  for (int i = 0; i < kUniqKeep; ++i) kept[i] = begin + i < end ? *word_ptr(begin + i) : 0u;
  bool none = threadIdx.x < kNoWordFlags && q.words->no_word[threadIdx.x * kNoWordStride] != 0;
  if (q.later && threadIdx.x == 0) none = none || q.previous->rays < q.total_pixels;
  int cnt = 0, fcnt = 0;
#pragma unroll
  for (int i = 0; i < kUniqKeep; ++i) {
    const int n = __popc(kept[i]);
    cnt += n;
    if (begin + i < q.fault_words) fcnt += n;
  }
  for (int k = begin + kUniqKeep; k < end; ++k) {
    const int n = __popc(*word_ptr(k));
    cnt += n;
    if (k < q.fault_words) fcnt += n;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = cnt;
  for (int off = 1; off < 32; off <<= 1) {
    int v = __shfl_up_sync(kFull, incl, off);
    if (lane >= off) incl += v;
  }
  if (lane == 31) warp_sums[warp] = incl;
  if (threadIdx.x == 0) fsum = 0;
  const bool no_word = __syncthreads_or(none);
  const int sums = warp_sums[lane];
  int pos = __reduce_add_sync(kFull, lane < warp ? sums : 0) + incl - cnt;
  const int all = __reduce_add_sync(kFull, sums);
  auto emit = [&](int k, uint32_t w) {
    if (k < q.fault_words) {
      const int wi = q.fault_words - 1 - k;
      while (w) {  // descending bits
        const int b = 31 - __clz(w);
        w &= ~(1u << b);
        q.unique_out[pos++] = -(wi * 32 + b) - 1;
      }
    } else {
      const int wi = k - q.fault_words;
      while (w) {  // ascending bits: value = bit index + 2
        const int b = __ffs(w) - 1;
        w &= w - 1;
        q.unique_out[pos++] = wi * 32 + b + 2;
      }
    }
  };
#pragma unroll
  for (int i = 0; i < kUniqKeep; ++i)
    if (kept[i]) {
      emit(begin + i, kept[i]);
      *word_ptr(begin + i) = 0u;
    }
  for (int k = begin + kUniqKeep; k < end; ++k) {
    uint32_t* w = word_ptr(k);
    if (*w) {
      emit(k, *w);
      *w = 0u;
    }
  }
  fcnt = __reduce_add_sync(kFull, fcnt);
  if (lane == 0 && fcnt) atomicAdd(&fsum, fcnt);
  if (q.client_faults && threadIdx.x < kMaxClients) {
    q.result->client_faults[threadIdx.x] = q.client_faults[threadIdx.x];
    q.next_client_faults[threadIdx.x] = 0;
  }
  // the other pass's words; every read of them came before the barrier above
  for (int i = threadIdx.x; i < kPassInts; i += kUniqThreads) reinterpret_cast<int*>(q.previous)[i] = 0;
  __threadfence_system();  // the values reach the host before the pass's number
  __syncthreads();
  if (threadIdx.x == 0) {
    int n = all;
    if (no_word) q.unique_out[n++] = kNoHit;
    q.result->unique = n;
    q.result->faults = fsum;
    q.result->rays = q.words->rays;
    q.result->trace_ms = (float)(long long)(begin_ns - q.words->start_ns) * 1e-6f;
    q.result->unique_ms = (float)(long long)(global_ns() - begin_ns) * 1e-6f;
    const unsigned int pass = *q.passes + 1;
    *q.passes = pass;
    __threadfence_system();
    *(volatile unsigned int*)&q.result->pass = pass;
  }
}

template <typename Kernel>
int resident_grid(Kernel kernel) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBlockThreads, 0);
  return sms * (per_sm > 0 ? per_sm : 1);
}

template <bool kCount>
int persistent_grid() {
  static const int grid = resident_grid(trace_persistent_kernel<true, kCount>);
  return grid;
}

// The traversal launch for pass kind (first, count): function, grid and
// parameters.
template <bool kFirst, bool kCount>
void trace_launch_shape(const TraceParams* p, int rays, int grid, TraceLaunch* l) {
  if (kFirst && p->refill < 32) {
    l->kp.func = reinterpret_cast<void*>(trace_persistent_kernel<true, kCount>);
    l->kp.gridDim = dim3(grid > 0 ? grid : persistent_grid<kCount>());
    l->args[0] = const_cast<TraceParams*>(p);
    return;
  }
  const int per = kBlockThreads / 32 * p->lanes;
  l->kp.gridDim = dim3(std::max(1, (rays + per - 1) / per));
  if (kFirst && p->n_views > 1) {
    l->kp.func = reinterpret_cast<void*>(trace_kernel<true, kCount, TraceParams>);
    l->args[0] = const_cast<TraceParams*>(p);
    return;
  }
  l->kp.func = reinterpret_cast<void*>(trace_kernel<kFirst, kCount, TraceParams1>);
  static_cast<TraceCore&>(l->one) = *p;
  l->one.views[0] = p->views[0];
  l->args[0] = &l->one;
}

}  // namespace

// A warp of 32 rays runs both sides of most iterations (descents and
// advances mix) and takes about 600 cycles for one; with 1 to 4 rays it is
// 350 to 450.  That is what a launch waits for when its warps do not fill the
// GPU and the longest ray decides, so such launches spread their rays over
// more warps: first passes up to 48 warps per SM (one resident wave holds 40;
// 128x96: 31.7 us with 32 rays per warp, 24.7 with 2; 200x150: 40.7 and 37.6
// with 4; 400x300 the same with 32 and 16, slower with 8), later passes, whose
// warps also end with a list append and feedback atomics each, up to 16
// (1280x720 stream, 12 thousand rays per later pass: 0.199 ms of traversal per
// frame with 32, 0.191 with 8 or 4, 0.196 with 2; 1919x1079, 27 thousand:
// best with 32 or 16).  Larger launches are bound by instruction issue, where
// half-empty warps cost 1.5 times the instructions.
int trace_lanes(bool first, int rays) {
  static const int sms = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
  }();
  const int warps = sms * (first ? 48 : 16);
  int lanes = 32;
  while (lanes > 1 && rays / (lanes / 2) <= warps) lanes /= 2;
  return lanes;
}

int trace_persistent_grid(bool count) { return count ? persistent_grid<true>() : persistent_grid<false>(); }

void trace_node_params(const TraceParams* p, bool first, bool count, int rays, int grid, TraceLaunch* l) {
  l->kp = cudaKernelNodeParams{};
  if (first) {
    if (count) trace_launch_shape<true, true>(p, rays, grid, l);
    else trace_launch_shape<true, false>(p, rays, grid, l);
  } else {
    if (count) trace_launch_shape<false, true>(p, rays, grid, l);
    else trace_launch_shape<false, false>(p, rays, grid, l);
  }
  l->kp.blockDim = dim3(kBlockThreads);
  l->kp.kernelParams = l->args;
}

cudaError_t launch_trace(const TraceParams& p, bool first, bool count, int rays, int grid, cudaStream_t s) {
  TraceLaunch l;
  trace_node_params(&p, first, count, rays, grid, &l);
  return cudaLaunchKernel(l.kp.func, l.kp.gridDim, l.kp.blockDim, l.kp.kernelParams, 0, s);
}

cudaError_t unique_node_params(const UniqueFromBitsParams* q, void** args, cudaKernelNodeParams* kp) {
  args[0] = const_cast<UniqueFromBitsParams*>(q);
  *kp = cudaKernelNodeParams{};
  kp->func = reinterpret_cast<void*>(unique_from_bits_kernel);
  kp->gridDim = dim3(1);
  kp->blockDim = dim3(kUniqThreads);
  kp->kernelParams = args;
  return cudaSuccess;
}

uchar4 finish_empty(const float* bg) {
  unsigned char o[4];
  for (int k = 0; k < 4; ++k) {
    const volatile float scaled = bg[k] * 255.f;  // each operation rounds by itself, as on the device
    const volatile float sum = 0.f + scaled;
    float v = sum + .5f;
    v = v < 255.f ? v : 255.f;
    v = 0.f < v ? v : 0.f;
    o[k] = (unsigned char)v;
  }
  return make_uchar4(o[0], o[1], o[2], o[3]);
}

cudaError_t launch_finish(const TraceCore& p, int max_rays, cudaStream_t s) {
  if (max_rays <= 0) return cudaSuccess;
  finish_kernel<<<(max_rays + kBlockThreads - 1) / kBlockThreads, kBlockThreads, 0, s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_deliver(const DeliverParams& p, cudaStream_t s) {
  if (p.images <= 0) return cudaSuccess;
  deliver_kernel<<<kDeliverCtas, kDeliverThreads, 0, s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_depth_view(const TraceParams1& p, cudaStream_t s) {
  const long long n = (long long)p.views[0].width * p.views[0].height;
  if (n <= 0) return cudaSuccess;
  depth_view_kernel<<<(unsigned)((n + kBlockThreads - 1) / kBlockThreads), kBlockThreads, 0, s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_fill_i32(int* ptr, int32_t v, size_t n, cudaStream_t s) {
  if (!n) return cudaSuccess;
  int grid = (int)((n + 255) / 256);
  if (grid > 4096) grid = 4096;
  fill_kernel<<<grid, 256, 0, s>>>(ptr, v, n);
  return cudaGetLastError();
}

cudaError_t launch_unique_from_bits(const UniqueFromBitsParams& q, cudaStream_t s) {
  unique_from_bits_kernel<<<1, kUniqThreads, 0, s>>>(q);
  return cudaGetLastError();
}

}  // namespace rayt
