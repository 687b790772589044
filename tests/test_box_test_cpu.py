"""The short box and node tests against the exact ones, on the host.

box_test.cuh's box_verdict must never contradict may_touch_box: it answers
only where f32 rounding cannot change the answer, and leaves the rest to it.
The header is compiled with the host compiler (no contraction, as the walk's
units) over random cones and boxes of every size, boxes with a corner on a
window plane, flat boxes, sky faces, and values that are not finite.
"""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

HARNESS = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include <string>
#define __device__
#define __forceinline__ inline
#include <cstdint>
#include <cstring>
#define __fmaf_rn fmaf
static uint32_t __float_as_uint(float x) { uint32_t u; memcpy(&u, &x, 4); return u; }
static float __uint_as_float(uint32_t u) { float x; memcpy(&x, &u, 4); return x; }
namespace cc {
struct f3 { float x, y, z; };
static f3 mk(float x, float y, float z) { return {x, y, z}; }
static f3 operator+(f3 a, f3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
static f3 operator-(f3 a, f3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
static f3 operator-(f3 a) { return {-a.x, -a.y, -a.z}; }
static f3 operator*(f3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
static float dot(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
static f3 cross(f3 a, f3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
static float len(f3 a) { return sqrtf(dot(a, a)); }
static f3 normalize(f3 a) { const float l = len(a); return {a.x / l, a.y / l, a.z / l}; }
constexpr float kNear = 1e-4f;
struct Cone { f3 apex, right, up, fwd; float u0, v0, u1, v1, far_offset; f3 baxis; float bcos, bsin; };
static f3 direction(const Cone& c, float s, float t) {
  return c.fwd + c.right * (c.u0 + s * (c.u1 - c.u0)) + c.up * (c.v0 + t * (c.v1 - c.v0));
}
static f3 to_local(const Cone& c, f3 p) { const f3 d = p - c.apex; return {dot(c.right, d), dot(c.up, d), dot(c.fwd, d)}; }
static float min_nan(float a, float b) { return std::isnan(a) || std::isnan(b) ? NAN : fminf(a, b); }
static float rsqrt_approx(float x) { return (float)(1.0 / std::sqrt((double)x)) * (1.0f + 2e-7f); }
#include "box_test.cuh"
constexpr int kGrid = 8;
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
static float2 make_float2(float x, float y) { return {x, y}; }
static float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
static float __fdividef(float a, float b) {  // within 2 units in the last place, either way
  static int n;
  return a / b * (n++ & 1 ? 1.0f + 2.4e-7f : 1.0f - 2.4e-7f);
}
#include "node_test.cuh"
}  // namespace cc
using namespace cc;
"""

BOX_MAIN = r"""
int main(int, char** argv) {
  std::mt19937_64 g(atoi(argv[1]));
  const std::string form = argv[2];
  auto u = [&] { return (double)(g() >> 11) / 9007199254740992.0; };
  auto U = [&](double a, double b) { return (float)(a + (b - a) * u()); };
  auto L = [&](double a, double b) { return (float)std::exp(std::log(a) + (std::log(b) - std::log(a)) * u()); };
  long asked = 0, open = 0, wrong = 0, touching = 0, touching_open = 0;
  for (long it = 0; it < 60000; ++it) {
    const float world = L(0.5, 3000);
    Cone c{};
    c.apex = mk(U(-world, world), U(0, world * 0.1), U(-world, world));
    const f3 f = normalize(mk(U(-1, 1), U(-1, 1), U(-1, 1)));
    c.fwd = f;
    c.right = normalize(cross(std::fabs(f.x) > 0.9f ? mk(0, 1, 0) : mk(1, 0, 0), f));
    c.up = cross(f, c.right);
    const bool sky = it % 11 == 0;
    if (it % 7 == 0 || sky) {
      c.fwd = mk(0, it % 2 ? 1.f : -1.f, 0);
      c.right = mk(0, 0, 1);
      c.up = cross(c.fwd, c.right);
    }
    const float ext = L(0.003, 12);
    c.u0 = U(-3, 3);
    c.v0 = U(-3, 3);
    c.u1 = c.u0 + ext;
    c.v1 = c.v0 + ext * U(0.3, 1);
    if (sky) { c.u0 = c.v0 = -1; c.u1 = c.v1 = 1; }
    const float dist = L(0.01, world * 1.5);
    c.far_offset = dot(c.fwd, c.apex) + (sky ? 1e7f : dist * (1 - 1e-5f));
    c.baxis = normalize(direction(c, 0.5f, 0.5f));
    float ch = 1;
    for (int k = 0; k < 4; ++k) ch = fminf(ch, dot(c.baxis, normalize(direction(c, float(k & 1), float(k >> 1)))));
    c.bcos = fminf(fmaxf(ch - 1e-5f, -1.f), 1.f);
    c.bsin = sqrtf(fmaxf(1.f - c.bcos * c.bcos, 0.f));
    f3 hz = normalize(mk(U(-1, 1), U(-1, 1), U(-1, 1)));
    if (form == "no horizon") hz = mk(0, 0, 0);
    if (form == "any normal") hz = hz * (it % 9 ? L(1e-4, 1e4) : L(1e-30, 1e30));
    if (it % 5003 == 1) c.right.x = NAN;
    if (it % 5003 == 2) c.baxis.y = NAN;
    if (it % 5003 == 3) c.apex.z = INFINITY;
    if (form == "any axes") {
      const float grow = L(1, 1e4);
      f3 row[3] = {normalize(mk(U(-1, 1), U(-1, 1), U(-1, 1))), normalize(mk(U(-1, 1), U(-1, 1), U(-1, 1)))};
      row[2] = normalize(cross(row[0], row[1]));
      row[1] = cross(row[2], row[0]);
      if (it % 3 == 0) row[1] = row[1] * U(0.1, 1);
      for (f3& r : row) r = r * grow;
      for (f3* a : {&c.right, &c.up, &c.fwd, &c.baxis}) *a = row[0] * a->x + row[1] * a->y + row[2] * a->z;
      c.far_offset = dot(c.fwd, c.apex) + dist * dot(c.fwd, c.fwd);
    }
    const BoxTest t = form == "any axes" ? box_test<true>(c) : box_test<false>(c);
    for (int k = 0; k < 24; ++k) {
      const float size = L(0.001, world);
      f3 e = mk(L(0.01, 1) * size, L(0.01, 1) * size, L(0.01, 1) * size);
      if (k % 5 == 0) e.y = 0;
      const float z = L(1e-4, dist * 2), uu = c.u0 + (c.u1 - c.u0) * U(-0.3, 1.3), vv = c.v0 + (c.v1 - c.v0) * U(-0.3, 1.3);
      f3 at = c.apex + (c.fwd + c.right * uu + c.up * vv) * z;
      if (k % 4 == 0) at = mk(U(-world, world), U(-world, world), U(-world, world));
      f3 lo = at - e * 0.5f, hi = at + e * 0.5f;
      if (k % 6 == 1) {  // a corner on the window's first side
        const f3 p = c.apex + (c.fwd + c.right * c.u0 + c.up * vv) * z;
        const f3 q = mk(c.right.x > 0 ? p.x - e.x : p.x + e.x, c.right.y > 0 ? p.y - e.y : p.y + e.y,
                        c.right.z > 0 ? p.z - e.z : p.z + e.z);
        lo = mk(fminf(p.x, q.x), fminf(p.y, q.y), fminf(p.z, q.z));
        hi = mk(fmaxf(p.x, q.x), fmaxf(p.y, q.y), fmaxf(p.z, q.z));
      }
      if (form == "any normal" && k % 3 == 1) {  // the corner farthest along the normal on the horizon
        const f3 top = mk(hz.x > 0 ? hi.x : lo.x, hz.y > 0 ? hi.y : lo.y, hz.z > 0 ? hi.z : lo.z) - c.apex;
        const f3 down = hz * (dot(hz, top) / dot(hz, hz));
        lo = lo - down;
        hi = hi - down;
      }
      if (form == "corners swapped") {
        if (k & 1) std::swap(lo.x, hi.x);
        if (k & 2) std::swap(lo.y, hi.y);
        if (k & 4) std::swap(lo.z, hi.z);
        if (k == 8) lo = mk(3.4e38f, 3.4e38f, 3.4e38f), hi = -lo;  // an empty box as some builders write it
      }
      if (it % 5003 == 4) hi.x = INFINITY;
      for (int h = 0; h < 2; ++h) {
        const bool exact = h ? may_touch_box<true>(c, lo, hi, hz) : may_touch_box<false>(c, lo, hi, hz);
        const int v = h ? box_verdict<true>(c, t, lo, hi, scaled_horizon(hz)) : box_verdict<false>(c, t, lo, hi, {});
        if (h && exact != may_touch_box<true>(c, lo, hi, scaled_horizon(hz).normal)) ++wrong;
        ++asked;
        if (exact) ++touching;
        if (exact && v == 2) ++touching_open;
        if (v == 2) ++open;
        else if ((v == 1) != exact) ++wrong;
      }
    }
  }
  std::printf("%ld %ld %ld %ld %ld\n", asked, open, wrong, touching, touching_open);
}
"""

NODE_MAIN = r"""
int main(int, char** argv) {
  std::mt19937_64 g(atoi(argv[1]));
  auto u = [&] { return (double)(g() >> 11) / 9007199254740992.0; };
  auto U = [&](double a, double b) { return (float)(a + (b - a) * u()); };
  auto L = [&](double a, double b) { return (float)std::exp(std::log(a) + (std::log(b) - std::log(a)) * u()); };
  long asked = 0, quick = 0, wrong = 0, splats = 0;
  for (long it = 0; it < 60000; ++it) {
    const float world = L(0.5, 3000);
    Cone c{};
    c.apex = mk(U(-world, world), U(0, world * 0.1), U(-world, world));
    c.fwd = normalize(mk(U(-1, 1), U(-1, 1), U(-1, 1)));
    c.right = normalize(cross(std::fabs(c.fwd.x) > 0.9f ? mk(0, 1, 0) : mk(1, 0, 0), c.fwd));
    c.up = cross(c.fwd, c.right);
    const bool narrow = it % 3 == 0;  // a small light far to the side
    const float ext = narrow ? L(1e-4, 0.01) : L(0.003, 12);
    c.u0 = narrow ? U(-40, 40) : U(-3, 3);
    c.v0 = narrow ? U(-40, 40) : U(-3, 3);
    c.u1 = c.u0 + ext;
    c.v1 = c.v0 + ext * U(0.3, 1);
    const float dist = L(0.01, world * 1.5);
    c.far_offset = dot(c.fwd, c.apex) + dist * (1 - 1e-5f);
    c.baxis = normalize(direction(c, 0.5f, 0.5f));
    float ch = 1;
    for (int k = 0; k < 4; ++k) ch = fminf(ch, dot(c.baxis, normalize(direction(c, float(k & 1), float(k >> 1)))));
    c.bcos = fminf(fmaxf(ch - 1e-5f, -1.f), 1.f);
    c.bsin = sqrtf(fmaxf(1.f - c.bcos * c.bcos, 0.f));
    const f3 hz = normalize(mk(U(-1, 1), U(-1, 1), U(-1, 1)));
    const BoxTest t = box_test<false>(c);
    for (int k = 0; k < 24; ++k) {
      const float z = L(1e-4, dist * 1.2);
      const float uu = c.u0 + (c.u1 - c.u0) * U(-0.1, 1.1), vv = c.v0 + (c.v1 - c.v0) * U(-0.1, 1.1);
      f3 at = c.apex + (c.fwd + c.right * uu + c.up * vv) * z;
      const float size = ext * z * L(0.01, 30);
      const f3 e = mk(L(0.01, 1) * size, L(0.01, 1) * size, L(0.01, 1) * size);
      if (k % 4 == 1) {  // its first or last corner along the cone's axis at a plane
        const float low = std::fabs(c.fwd.x) * e.x + std::fabs(c.fwd.y) * e.y + std::fabs(c.fwd.z) * e.z;
        const float planes[3] = {0.0f, kNear, dist * (1 - 1e-5f)};
        const int p = (k / 4) % 3;
        at = at + c.fwd * (planes[p] * (1 + U(-1e-6, 1e-6)) + (p == 2 ? -0.5f : 0.5f) * low - dot(c.fwd, at - c.apex));
      }
      const f3 lo = at - e * 0.5f, hi = at + e * 0.5f;
      float2 pts[8];
      float4 bins{};
      project_node<false>(c, hz, lo, hi, 3.4e38f, pts, bins);
      const float width = fmaxf(bins.z - bins.x, bins.w - bins.y);  // of the corners before the first one outside
      for (int h = 0; h < 4; ++h) {
        const float prefilter = h < 2 && width > 0 && width < 1e9f ? width * (1 + U(-1, 1) * L(1e-7, 1e-2)) : L(0.1, 8);
        const int exact = h & 1 ? project_node<true>(c, hz, lo, hi, prefilter, pts, bins)
                                : project_node<false>(c, hz, lo, hi, prefilter, pts, bins);
        const int v = h & 1 ? quick_node_test<true>(c, t, lo, hi, scaled_horizon(hz), prefilter)
                            : quick_node_test<false>(c, t, lo, hi, {}, prefilter);
        ++asked;
        if (exact == 1) ++splats;
        if (v == 4) continue;
        ++quick;
        if (v != exact) ++wrong;
      }
    }
  }
  std::printf("%ld %ld %ld %ld\n", asked, quick, wrong, splats);
}
"""


def built(tmp_path_factory, name, main):
    folder = tmp_path_factory.mktemp(name)
    (folder / "main.cpp").write_text(HARNESS + main)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-Wno-unknown-pragmas", "-I",
                    str(ROOT / "continuum_b200" / "csrc"), "-o", str(folder / name), str(folder / "main.cpp")],
                   check=True)

    def run(*args):
        out = subprocess.run([str(folder / name), *map(str, args)], check=True, capture_output=True, text=True).stdout
        return map(int, out.split())

    return run


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    return built(tmp_path_factory, "box", BOX_MAIN)


@pytest.fixture(scope="module")
def node_harness(tmp_path_factory):
    return built(tmp_path_factory, "node", NODE_MAIN)


@pytest.mark.parametrize("form", ["unit", "no horizon", "any normal", "corners swapped", "any axes"])
@pytest.mark.parametrize("seed", [1, 2])
def test_box_verdict_never_contradicts_the_exact_test(harness, seed, form):
    """`no horizon`: horizons of zero, which cull nothing (CC_SKY_NO_HORIZON_CULL);
    `any normal`: horizons of any length, and boxes with a corner on theirs;
    `corners swapped`: boxes whose low corner is the higher along some axes;
    `any axes`: cones in the space of an object whose matrix is no rotation."""
    asked, left, wrong, touching, touching_left = harness(seed, form)
    assert wrong == 0
    # A sixth of the boxes are put on a plane; most others are decided, and of
    # those that touch as many.
    assert left < 0.25 * asked
    assert touching_left < 0.5 * touching


@pytest.mark.parametrize("seed", [1, 2])
def test_quick_node_test_never_contradicts_the_exact_one(node_harness, seed):
    """Prefiltering cones at nodes as wide as the prefilter (and a little more
    or less), with corners at the apex's, the near and the far plane, and in
    narrow windows far from the axis: where the quick test answers, the exact
    one agrees; both answers and splats occur."""
    asked, quick, wrong, splats = node_harness(seed)
    assert wrong == 0
    assert quick > 0.4 * asked and splats > 0.05 * asked
