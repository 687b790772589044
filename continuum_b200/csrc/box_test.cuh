// A cone against an axis-aligned box: the reference's test and its short form.
// Included by cone_device.cuh inside namespace cc; uses nothing of CUDA beyond
// the two approximations defined there, so that the two forms can be compared
// on the host (tests/test_box_test_cpu.py).
#pragma once

__device__ __forceinline__ bool in_bound(const Cone& c, f3 p, float r) {  // :159-168
  if (c.bcos < -1.0f) return true;
  f3 d = p - c.apex;
  float l = len(d);
  if (l <= r) return true;
  float s = r / l;
  float limit = c.bcos * sqrtf(1.0f - s * s) - c.bsin * s;
  return dot(c.baxis, d) >= limit * l;
}

// may_touch_box (:234-255), which is node_cone_test (:519-574) for exact cones.
// kHorizon: sky cones, whose horizon `horizon` (the receiver's normal, in the
// cone's space) also culls a box wholly below it (:245); a light cone's
// horizon is zero (:146-147), which culls nothing, so light cones skip it.
// One corner at a time, in a fifth of the unrolled code: it runs where
// box_verdict leaves a box open.
template <bool kHorizon = false>
__device__ __forceinline__ bool may_touch_box(const Cone& c, f3 lo, f3 hi, f3 horizon = f3{0.f, 0.f, 0.f}) {
  bool far_out = true, near_out = true, out_u0 = true, out_u1 = true, out_v0 = true, out_v1 = true, below = kHorizon;
#pragma unroll 1
  for (int k = 0; k < 8; ++k) {
    f3 corner = mk((k & 1) ? hi.x : lo.x, (k & 2) ? hi.y : lo.y, (k & 4) ? hi.z : lo.z);
    if (c.far_offset - dot(c.fwd, corner) >= 0.0f) far_out = false;
    if constexpr (kHorizon) {
      if (dot(horizon, corner - c.apex) >= 0.0f) below = false;
    }
    f3 p = to_local(c, corner);
    if (p.z >= kNear) near_out = false;
    if (p.x - c.u0 * p.z >= 0.0f) out_u0 = false;
    if (c.u1 * p.z - p.x >= 0.0f) out_u1 = false;
    if (p.y - c.v0 * p.z >= 0.0f) out_v0 = false;
    if (c.v1 * p.z - p.y >= 0.0f) out_v1 = false;
  }
  if (far_out || near_out || out_u0 || out_u1 || out_v0 || out_v1 || below) return false;
  return in_bound(c, (lo + hi) * 0.5f, 0.5f * len(hi - lo));
}

// may_touch_box decided from a box's centre and half extents. Its exact form
// asks, plane by plane, whether some corner of eight passes; the plane's
// largest value over the box is its value at the centre plus |normal| x half
// extents, a quarter of the work. Both are f32 evaluations of one real
// number with errors below 16 units in the last place of the terms they sum
// (coordinates from the apex, of size `reach`, times 1 + the window's largest
// side; for the far plane and the bounding cone, world coordinates; all times
// the axes' largest component, where an object's matrix made it exceed 1), so
// a value farther from zero than 33 of them decides as the exact form would,
// and any other (not-a-numbers among them) leaves the question to it. All sums
// here are doubled: centre x 2 and the whole extents are one subtraction each.
constexpr float kBoxSlack = 2e-6f;  // 33 x 2^-24
struct BoxTest {
  f3 nu0, nu1, nv0, nv1;  // the window's planes: right - u0 fwd, u1 fwd - right, up - v0 fwd, v1 fwd - up
  float side;             // 1 + the window's largest side
  float world;            // the world coordinates' size at the apex, times `axes`
  float axes;             // 1, or the axes' largest component
  float far_rel;          // the far plane's distance along fwd from the apex, doubled
};
__device__ __forceinline__ f3 fma3(f3 a, float s, f3 b) {
  return {__fmaf_rn(a.x, s, b.x), __fmaf_rn(a.y, s, b.y), __fmaf_rn(a.z, s, b.z)};
}
__device__ __forceinline__ float fdot(f3 a, f3 b, float s) {
  return __fmaf_rn(a.x, b.x, __fmaf_rn(a.y, b.y, __fmaf_rn(a.z, b.z, s)));
}
__device__ __forceinline__ float fdot_abs(f3 a, f3 h, float s) {  // |a| . h + s
  return __fmaf_rn(fabsf(a.x), h.x, __fmaf_rn(fabsf(a.y), h.y, __fmaf_rn(fabsf(a.z), h.z, s)));
}
// kPlaced: the cone may be in the space of a placed object, whose matrix need
// not be a rotation (cc_scene_move and cc_scene_upload take any); else its axes
// are unit vectors.
template <bool kPlaced>
__device__ __forceinline__ BoxTest box_test(const Cone& c) {
  BoxTest t;
  t.nu0 = fma3(c.fwd, -c.u0, c.right);
  t.nu1 = fma3(c.fwd, c.u1, -c.right);
  t.nv0 = fma3(c.fwd, -c.v0, c.up);
  t.nv1 = fma3(c.fwd, c.v1, -c.up);
  t.side = 1.0f + fmaxf(fmaxf(fabsf(c.u0), fabsf(c.u1)), fmaxf(fabsf(c.v0), fabsf(c.v1)));
  t.axes = 1.0f;
  if constexpr (kPlaced) {
    auto size = [](f3 a) { return fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fabsf(a.z)); };
    t.axes = fmaxf(fmaxf(fmaxf(size(c.right), size(c.up)), fmaxf(size(c.fwd), size(c.baxis))), 1.0f);
  }
  t.world = t.axes * (fabsf(c.apex.x) + fabsf(c.apex.y) + fabsf(c.apex.z));
  t.far_rel = 2.0f * (c.far_offset - fdot(c.fwd, c.apex, 0.0f));
  return t;
}
// A sky cone's horizon as the tests take it. The caller's normal may have any
// length, and the plane's error has its size: scaled by a power of two to a
// largest component in [1/2, 1), which changes no sign of the exact form, it
// has the slack of the other planes. One of zero (CC_SKY_NO_HORIZON_CULL) culls
// nothing and gets a value far above the slack, as zero would leave every box
// that touches to the exact form.
struct Horizon {
  f3 normal;
  float lift;
};
__device__ __forceinline__ Horizon scaled_horizon(f3 n) {
  const float size = fmaxf(fmaxf(fabsf(n.x), fabsf(n.y)), fabsf(n.z));
  const uint32_t e = __float_as_uint(size) >> 23;  // 2^(e - 127) <= size, but for subnormal sizes
  const float scale = e < 253u ? __uint_as_float((253u - e) << 23) : 2.9387359e-39f;  // 2^-128
  return {n * scale, size == 0.0f ? 1e30f : 0.0f};
}
// 0: the cone cannot touch the box, 1: it may, 2: ask may_touch_box.
template <bool kHorizon>
__device__ __forceinline__ int box_verdict(const Cone& c, const BoxTest& t, f3 lo, f3 hi, const Horizon& h) {
  const f3 a = lo - c.apex, b = hi - c.apex;
  // Doubled centre (from the apex) and half extents; an uploaded box's corners
  // may be swapped, which the exact form does not see.
  const f3 m = a + b, e = mk(fabsf(b.x - a.x), fabsf(b.y - a.y), fabsf(b.z - a.z));
  const float reach = (fabsf(m.x) + e.x) + (fabsf(m.y) + e.y) + (fabsf(m.z) + e.z);
  const float s_near = kBoxSlack * t.axes * reach, s_side = s_near * t.side;
  const float s_world = __fmaf_rn(kBoxSlack, t.world, s_near);  // half the doubled sums' world coordinates
  const float fm = fdot(c.fwd, m, 0.0f), fe = fdot_abs(c.fwd, e, 0.0f);
  float v = min_nan(min_nan(fdot(t.nu0, m, fdot_abs(t.nu0, e, 0.0f)), fdot(t.nu1, m, fdot_abs(t.nu1, e, 0.0f))),
                    min_nan(fdot(t.nv0, m, fdot_abs(t.nv0, e, 0.0f)), fdot(t.nv1, m, fdot_abs(t.nv1, e, 0.0f))));
  float n = fm + fe - 2.0f * kNear;
  if constexpr (kHorizon) n = min_nan(n, fdot(h.normal, m, fdot_abs(h.normal, e, h.lift)));
  const float f = t.far_rel - fm + fe;
  const float s_far = 2.0f * s_world + kBoxSlack * fabsf(c.far_offset);
  // The bounding cone: axis . d >= bcos sqrt(d.d - r r) - bsin r once outside
  // the sphere of radius r.
  const float l2 = fdot(m, m, 0.0f), r2 = fdot(e, e, 0.0f);
  const float q = l2 - r2, s_q = 4.0f * s_world * reach;
  const float rs = rsqrt_approx(q);
  const float g = fdot(c.baxis, m, __fmaf_rn(-c.bcos, q * rs, c.bsin * (r2 * rsqrt_approx(r2))));
  const float s_g = __fmaf_rn(s_q, rs, 4.0f * s_world);
  const bool sphere = q < -s_q;  // the apex lies inside the box's sphere
  const bool apart = q > 64.0f * s_q;
  if (reach < 1e15f) {
    if (v < -s_side || n < -s_near || f < -s_far || (apart && g < -s_g)) return 0;
    if (v >= s_side && n >= s_near && f >= s_far && (sphere || (apart && g >= s_g))) return 1;
  }
  return 2;
}
// may_touch_box's answer.
template <bool kHorizon>
__device__ __forceinline__ bool touches_box(const Cone& c, const BoxTest& t, f3 lo, f3 hi, const Horizon& h) {
  int v = box_verdict<kHorizon>(c, t, lo, hi, h);
  if (v == 2) v = may_touch_box<kHorizon>(c, lo, hi, h.normal) ? 1 : 0;
  return v == 1;
}
