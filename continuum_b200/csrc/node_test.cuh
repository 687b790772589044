// The decision of a prefiltering cone at a hierarchy node: the reference's and
// its short form. Included by splat_device.cuh inside namespace cc, after
// box_test.cuh; the two forms are compared on the host
// (tests/test_box_test_cpu.py).
#pragma once

// node_cone_test (:519-574) up to the opacity: 0 if the box cannot touch the
// cone, 3 if the cone must descend, 1 if it splats the box, whose projected
// corners (in bins) are then in pts and their bounds in bins (lowest x and y,
// highest x and y).
template <bool kHorizon>
__device__ __forceinline__ int project_node(const Cone& c, f3 horizon, f3 lo, f3 hi, float prefilter, float2* pts,
                                            float4& bins) {
  const float g = float(kGrid);
  float mnx = 3.4e38f, mny = 3.4e38f, mxx = -3.4e38f, mxy = -3.4e38f;
  bool far_out = true, near_out = true, out_u0 = true, out_u1 = true, out_v0 = true, out_v1 = true;
  bool below = kHorizon;
  bool inside = prefilter > 0.0f;  // splattable: every corner between the near and far planes
#pragma unroll 1
  for (int k = 0; k < 8; ++k) {
    const f3 corner = mk((k & 1) ? hi.x : lo.x, (k & 2) ? hi.y : lo.y, (k & 4) ? hi.z : lo.z);
    if constexpr (kHorizon) {
      if (dot(horizon, corner - c.apex) >= 0.0f) below = false;
    }
    const bool in_far = c.far_offset - dot(c.fwd, corner) >= 0.0f;
    if (in_far) far_out = false; else inside = false;
    const f3 p = to_local(c, corner);
    if (p.z >= kNear) near_out = false; else inside = false;
    if (p.x - c.u0 * p.z >= 0.0f) out_u0 = false;
    if (c.u1 * p.z - p.x >= 0.0f) out_u1 = false;
    if (p.y - c.v0 * p.z >= 0.0f) out_v0 = false;
    if (c.v1 * p.z - p.y >= 0.0f) out_v1 = false;
    if (inside) {
      const float qx = (p.x / p.z - c.u0) / (c.u1 - c.u0) * g;
      const float qy = (p.y / p.z - c.v0) / (c.v1 - c.v0) * g;
      pts[k] = make_float2(qx, qy);
      mnx = fminf(mnx, qx);
      mny = fminf(mny, qy);
      mxx = fmaxf(mxx, qx);
      mxy = fmaxf(mxy, qy);
    }
  }
  if (far_out || near_out || out_u0 || out_u1 || out_v0 || out_v1 || below) return 0;
  if (!in_bound(c, (lo + hi) * 0.5f, 0.5f * len(hi - lo))) return 0;
  bins = make_float4(mnx, mny, mxx, mxy);
  return !inside || fmaxf(mxx - mnx, mxy - mny) > prefilter ? 3 : 1;
}

// node_cone_test's first answer from box_verdict and two opposite corners:
// 0 (cannot touch), 3 (descend), or 4: ask node_cone_test. A node that
// touches is descended into when some corner lies before the apex or past the
// far plane, or when the box is wider in the cone than `prefilter` bins; of
// the corners farthest apart along the window's right (and up) axis, the
// projections' distance is a lower bound of that width. Every comparison
// leaves box_verdict's slack, so the answer is node_cone_test's.
template <bool kHorizon>
__device__ __forceinline__ int quick_node_test(const Cone& c, const BoxTest& t, f3 lo, f3 hi, const Horizon& h,
                                               float prefilter) {
  const int v = box_verdict<kHorizon>(c, t, lo, hi, h);
  if (v != 1) return v == 0 ? 0 : 4;
  const f3 a = lo - c.apex, b = hi - c.apex;
  const f3 m = a + b, e = mk(fabsf(b.x - a.x), fabsf(b.y - a.y), fabsf(b.z - a.z));
  const float reach = (fabsf(m.x) + e.x) + (fabsf(m.y) + e.y) + (fabsf(m.z) + e.z);
  const float slack = kBoxSlack * t.axes * reach;
  const float fm = fdot(c.fwd, m, 0.0f), fe = fdot_abs(c.fwd, e, 0.0f);
  if (fm - fe < -slack) return 3;
  if (t.far_rel - fm - fe < -(2.0f * __fmaf_rn(kBoxSlack, t.world, slack) + kBoxSlack * fabsf(c.far_offset))) return 3;
  bool wide = false;
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    const f3 axis = k ? c.up : c.right;
    const float x = fdot(axis, m, 0.0f), w = fdot_abs(axis, e, 0.0f);
    const float z = fdot(c.fwd, mk(copysignf(e.x, axis.x), copysignf(e.y, axis.y), copysignf(e.z, axis.z)), 0.0f);
    const float z0 = fm - z, z1 = fm + z, least = fminf(z0, z1);
    if (!(least > 64.0f * slack)) continue;
    const float q0 = __fdividef(x - w, z0), q1 = __fdividef(x + w, z1);
    const float side = k ? c.v1 - c.v0 : c.u1 - c.u0;
    if (fabsf(q1 - q0) - __fdividef(4.0f * slack * (1.0f + fabsf(q0) + fabsf(q1)), least) >
        1.001f * prefilter * side * (1.0f / float(kGrid)))
      wide = true;
  }
  return wide ? 3 : 4;
}
