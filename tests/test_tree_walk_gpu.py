"""The tree walk (pairs of a cone and a node) against the oracle's walk, where
it can go wrong: packets of every size, meshes at the edges of the leaves'
size, hierarchies of one node, caps that end inside a mesh (which is then
walked in order), windows wide and narrow, and the work counters, which count
every visited node and tested triangle."""
import numpy as np
import pytest

from continuum_b200 import scenes
from continuum_b200.kernel import Light, RectLight, SphereLight, light_gpu
from oracle.oracle import OracleScene

pytestmark = pytest.mark.gpu
ALL = ("full", "any", "partial", "irradiance", "fraction", "work")


def sliced_scene(counts, seed=1):
    """Meshes of `counts` triangles each, cut from displaced icospheres over a
    ground quad, receivers on the ground and on the shapes, two lights."""
    rng = np.random.default_rng(seed)
    meshes = [scenes.ground_quad(30.0)]
    for k, n in enumerate(counts):
        shape = scenes.displaced_icosphere((rng.uniform(-4, 4), 1.5, rng.uniform(-4, 4)), 1.2, seed=40 + k,
                                           subdivisions=3)
        meshes.append(np.ascontiguousarray(shape[:n]))
    lights = np.stack([light_gpu(Light.rect(RectLight((-1.0, 6.0, -1.0), (2.0, 0.0, 0.0), (0.0, 0.0, 2.0), True))),
                       light_gpu(Light(SphereLight((1.0, 5.0, 0.5), 0.8)))])
    n = 21
    x, z = np.meshgrid(np.linspace(-5, 5, n), np.linspace(-5, 5, n))
    rec = np.zeros((n * n, 8), np.float32)
    rec[:, 0], rec[:, 2], rec[:, 5] = x.ravel(), z.ravel(), 1.0
    # Some on a shape, lifted along the normal: cones that graze their own mesh.
    big = meshes[int(np.argmax([len(m) for m in meshes]))][::7]
    nrm = np.cross(big[:, 1] - big[:, 0], big[:, 2] - big[:, 0])
    nrm /= np.maximum(np.linalg.norm(nrm, axis=1, keepdims=True), 1e-12)
    own = np.zeros((len(big), 8), np.float32)
    own[:, 0:3] = big.mean(axis=1) + 1e-4 * nrm
    own[:, 4:7] = nrm
    return meshes, lights, np.concatenate([rec, own]).astype(np.float32)


def same(kernel, meshes, lights, rec, cap=4096, wide_cap=512, wide_extent=8.0, pw=32):
    osc = OracleScene(meshes)
    o = osc.visibility(rec, lights, accumulate=1, light_cone_cap=cap, wide_cone_cap=wide_cap, wide_extent=wide_extent)
    osc.close()
    scene = kernel.scene(meshes)
    kernel.light_cone_cap, kernel.wide_cone_cap, kernel.wide_extent = cap, wide_cap, wide_extent
    try:
        g = kernel.visibility(scene, rec, lights, outputs=ALL, points_per_warp=pw)
    finally:
        kernel.light_cone_cap, kernel.wide_cone_cap, kernel.wide_extent = 4096, 512, 8.0
        scene.close()
    assert np.array_equal(g.full.reshape(-1), o["full"]) and np.array_equal(g.any.reshape(-1), o["any"])
    assert np.array_equal(g.partial.reshape(-1, 64), o["partial"])
    work = g.work.reshape(-1, 4)
    assert np.array_equal(work[:, :3], o["work"][:, :3])
    assert np.array_equal(work[:, 3] & 1, o["work"][:, 3] & 1)  # CC_CONE_CAPPED
    # Light and fraction: the same mask integrated in f32 on both sides.
    assert np.abs(g.fraction.reshape(-1) - o["fraction"]).max() <= 1e-3
    return work


@pytest.mark.parametrize("pw", [1, 5, 16, 32])
def test_packets_of_every_size(kernel, pw):
    same(kernel, *sliced_scene([1280, 1280, 300]), pw=pw)


@pytest.mark.parametrize("counts", [[1], [7, 8, 9], [15, 16, 17], [31, 33, 64, 65], []])
def test_meshes_at_the_leaves_edges(kernel, counts):
    same(kernel, *sliced_scene(counts))


@pytest.mark.parametrize("cap,wide_cap", [(1, 1), (9, 9), (40, 20), (150, 100), (1000, 60)])
def test_caps_inside_a_mesh(kernel, cap, wide_cap):
    work = same(kernel, *sliced_scene([1280, 640], seed=3), cap=cap, wide_cap=wide_cap, wide_extent=0.5)
    assert (work[:, 3] & 1).any()


def test_few_cones(kernel):
    meshes, lights, rec = sliced_scene([1280])
    same(kernel, meshes, lights[:1], rec[:1])
    same(kernel, meshes, lights, rec[:33])


@pytest.mark.parametrize("n", [1, 65, 4735, 4737, 37889])
def test_small_calls_packets_change_no_result(kernel, n):
    """Small calls walk and integrate in smaller pieces; calls that count work
    keep the packets, so they give the other side."""
    meshes, lights, rec = sliced_scene([300, 40])
    rec = np.ascontiguousarray(np.tile(rec, (n // len(rec) + 1, 1))[:n])
    scene = kernel.scene(meshes)
    a = kernel.visibility(scene, rec, lights)
    b = kernel.visibility(scene, rec, lights, outputs=ALL)
    scene.close()
    for k in ("full", "any", "irradiance", "fraction"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k


@pytest.mark.parametrize("squeeze", [(1, 1, 1), (1, 0, 1), (0, 1, 0), (1e-3, 1, 40)])
def test_walk_order_over_any_bounds(kernel, squeeze):
    """The walk order's grid over flat and long scenes, receivers outside their
    bounds and receivers that are no numbers: the order changes no result."""
    from continuum_b200 import _lib

    meshes, lights, rec = sliced_scene([200, 64])
    meshes = [np.ascontiguousarray(m * np.asarray(squeeze, np.float32)) for m in meshes]
    rec[::50, 0:3] *= 1e3
    rec[7::100, 1] = np.nan
    scene = kernel.scene(meshes)
    a = kernel.visibility(scene, rec, lights)
    b = kernel.visibility(scene, rec, lights, flags=_lib.CC_KEEP_ORDER)
    scene.close()
    for k in ("full", "any", "irradiance", "fraction"):
        assert np.array_equal(getattr(a, k), getattr(b, k), equal_nan=k in ("irradiance", "fraction")), k
