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


def same(kernel, meshes, lights, rec, cap=4096, wide_cap=512, wide_extent=8.0, pw=32, prefilter=0.0):
    osc = OracleScene(meshes)
    o = osc.visibility(rec, lights, accumulate=1, light_cone_cap=cap, wide_cone_cap=wide_cap, wide_extent=wide_extent,
                       prefilter=prefilter)
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


def flat_copy(kernel, meshes, flip=False):
    """The scene of `meshes` uploaded as flat arrays; `flip`: with the corners
    of its hierarchies' boxes swapped along some axes."""
    built = kernel.scene(meshes)
    a = built.arrays()
    built.close()
    counts = [len(m) for m in meshes]
    tris = np.zeros((sum(counts), 3, 4), np.float32)
    tris[:, :, 0:3] = np.concatenate(meshes)
    blas, nodes = a["blas"].copy(), a["nodes"].copy()
    if flip:
        rng = np.random.default_rng(7)
        for n in (blas, nodes):
            swap = rng.random((len(n), 3)) < 0.5
            lo, hi = n["lo"][:, :3].copy(), n["hi"][:, :3].copy()
            n["lo"][:, :3], n["hi"][:, :3] = np.where(swap, hi, lo), np.where(swap, lo, hi)
    return kernel.scene_from_flat(tris, a["ranges"], blas, a["blas_items"], nodes, a["items"])


def test_swapped_box_corners_change_no_result(kernel):
    meshes, lights, rec = sliced_scene([1280, 300])
    out = []
    for flip in (False, True):
        scene = flat_copy(kernel, meshes, flip)
        out.append(kernel.visibility(scene, rec, lights))
        scene.close()
    for k in ("full", "any", "irradiance", "fraction"):
        assert np.array_equal(getattr(out[0], k), getattr(out[1], k)), k


def fullest_stack(cones, depth, room):
    """The most pairs waiting in a walk of a complete tree, every node touched:
    32 at a time, or one once `room` are waiting."""
    stack, most = [0] * cones, 0
    while stack:
        n = min(len(stack), 32, max(room - len(stack), 1))
        taken = stack[-n:]
        del stack[-n:]
        for d in taken:
            if d + 1 < depth:
                stack += [d + 1, d + 1]
        most = max(most, len(stack))
    return most


@pytest.mark.parametrize("cap", [1 << 20, 4096])
@pytest.mark.parametrize("prefilter", [0.0, 1e-3])
def test_full_pair_stack(kernel, prefilter, cap):
    """A sheet of 8,192 triangles wholly inside every cone: the pairs waiting
    fill the stack to where they are taken one by one (192 of 256; prefiltering
    cones 256 of 384), and with the smaller cap the cones are walked again in
    order from there."""
    n = 64
    g = np.linspace(-0.4, 0.4, n + 1)
    x, z = (a.astype(np.float32) for a in np.meshgrid(g, g, indexing="ij"))
    at = np.stack([x, np.full_like(x, 2.0), z], axis=-1)
    p00, p10, p01, p11 = at[:-1, :-1], at[1:, :-1], at[:-1, 1:], at[1:, 1:]
    sheet = np.concatenate([np.stack([p00, p10, p11], axis=2).reshape(-1, 3, 3),
                            np.stack([p00, p11, p01], axis=2).reshape(-1, 3, 3)])
    depth = 10  # 1,024 leaves of eight triangles, or fewer in each
    assert fullest_stack(16, depth, 192) > 192 and fullest_stack(16, depth, 256) > 256
    lights = np.stack([light_gpu(Light.rect(RectLight((-2.0, 4.0, -2.0), (4.0, 0.0, 0.0), (0.0, 0.0, 4.0), True)))])
    rec = np.zeros((64, 8), np.float32)
    rec[:, 0], rec[:, 2] = np.tile(np.linspace(-0.1, 0.1, 8), 8), np.repeat(np.linspace(-0.1, 0.1, 8), 8)
    rec[:, 5] = 1.0
    meshes = [np.ascontiguousarray(sheet, np.float32)]
    kernel.prefilter = prefilter
    try:
        work = same(kernel, meshes, lights, rec, cap=cap, prefilter=prefilter)
    finally:
        kernel.prefilter = 0.0
    assert (work[:, 3] & 1).all() == (cap == 4096)


@pytest.mark.parametrize("cap,wide_cap", [(9, 9), (40, 20)])
@pytest.mark.parametrize("prefilter", [0.25, 1.0])
def test_prefiltered_caps_inside_a_mesh(kernel, cap, wide_cap, prefilter):
    kernel.prefilter = prefilter
    try:
        work = same(kernel, *sliced_scene([1280, 640], seed=3), cap=cap, wide_cap=wide_cap, wide_extent=0.5,
                    prefilter=prefilter)
    finally:
        kernel.prefilter = 0.0
    assert (work[:, 3] & 1).any()
