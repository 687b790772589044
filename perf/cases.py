"""Cases that time the visibility library through its public entry points.

Each case is one call (or one frame's calls) that a program holding resident
scenes makes: plain solves from host and device buffers, sky cones, prefiltered
cones, a batch of uneven jobs, served requests, and instanced worlds with and
without moving objects. Scenes are the package's kinds: a ground with boxes
under a rect light, fields of displaced icospheres under rect and disk lights,
and boulders placed as instances. Everything is made from a case and a seed.
"""
import math
from functools import lru_cache

import numpy as np
import torch

from continuum_b200 import _lib, scenes
from continuum_b200.kernel import Batch, Light, MaskConeKernel, RectLight, Server, light_gpu

PLAIN = ("full", "any", "irradiance", "fraction")


def listed():
    return [
        # A tool that asks for a patch of texels at a time, from host arrays:
        # the smallest call, where the launches and copies count.
        dict(name="host_patch", kind="room", entry="host", boxes=64, grid=64),
        # The drop-in call of the reference's kernel, which takes meshes and
        # receivers and tests every triangle: 34 boxes, 65,536 receivers.
        dict(name="drop_in_every_triangle", kind="room", entry="irradiance", boxes=34, grid=256),
        # The small plain workload, resident: 770 triangles, 65,536 cones.
        dict(name="room_resident", kind="room", entry="device", boxes=64, grid=256),
        # A mid-sized view with odd sizes and per-bin coverages kept.
        dict(name="field_ragged", kind="field", entry="device", spheres=61, lights=3, width=317, height=241,
             partial=True),
        # The plain workload at scale: 3.07 M triangles, four lights, 1280 x 720.
        dict(name="field_large", kind="field", entry="device", spheres=150, lights=4, width=1280, height=720,
             partial=False),
        # Ambient light of a bake: exact sky cones of the small scene.
        dict(name="sky_exact", kind="room", entry="sky", boxes=64, grid=256),
        # Ambient light over dense geometry: sky cones prefiltered to one bin.
        dict(name="sky_prefiltered", kind="field", entry="sky", spheres=50, lights=1, width=320, height=180,
             partial=False, prefilter=1.0),
        # Light cones prefiltered, the interactive setting over dense geometry.
        dict(name="lights_prefiltered", kind="field", entry="device", spheres=100, lights=4, width=480, height=270,
             partial=False, prefilter=1.0),
        # Many uneven jobs in one submission (graph replay).
        dict(name="batch_uneven", kind="batch", jobs=24, most_spheres=40, least_points=4000, most_points=160000,
             most_lights=8),
        # Requests of different sizes in flight together, host to host.
        dict(name="served_mix", kind="served", requests=12, spheres=40, least_points=8000, most_points=200000,
             most_lights=6),
        # A large instanced world, every cone.
        dict(name="instanced_full", kind="instanced", objects=60000, lights=4, width=640, height=360, moved=0),
        # A frame of that world with one object in a hundred moved: only the
        # cones the movers may touch are solved again.
        dict(name="instanced_moving", kind="instanced", objects=60000, lights=4, width=800, height=450, moved=600),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("host", "irradiance", "room", "field", "field", "back", "sky", "sky_splat", "splat", "batch",
                       "served", "instanced", "moving"))
    if kind == "host":
        return dict(kind="room", entry="host", boxes=_log(rng, 8, 128), grid=_log(rng, 24, 320))
    if kind == "irradiance":
        return dict(kind="room", entry="irradiance", boxes=_log(rng, 8, 64), grid=_log(rng, 48, 256))
    if kind == "room":
        return dict(kind="room", entry=rng.choice(("device", "static")), boxes=_log(rng, 8, 256),
                    grid=_log(rng, 24, 360))
    if kind in ("field", "back"):
        w = _log(rng, 64, 900)
        return dict(kind="field", entry="back" if kind == "back" else "device", spheres=_log(rng, 3, 150),
                    lights=rng.randint(1, 4), width=w, height=max(8, w * 9 // 16 + rng.randint(-3, 3)),
                    partial=rng.random() < 0.3)
    if kind == "sky":
        return dict(kind="room", entry="sky", boxes=_log(rng, 8, 128), grid=_log(rng, 24, 300))
    if kind == "sky_splat":
        w = _log(rng, 48, 320)
        return dict(kind="field", entry="sky", spheres=_log(rng, 3, 50), lights=1, width=w, height=max(8, w * 9 // 16),
                    partial=False, prefilter=rng.choice((1.0, 2.0)))
    if kind == "splat":
        w = _log(rng, 64, 480)
        return dict(kind="field", entry="device", spheres=_log(rng, 3, 100), lights=rng.randint(1, 4), width=w,
                    height=max(8, w * 9 // 16), partial=False, prefilter=rng.choice((1.0, 2.0, 8.0)))
    if kind == "batch":
        return dict(kind="batch", jobs=_log(rng, 4, 24), most_spheres=_log(rng, 10, 40), least_points=4000,
                    most_points=_log(rng, 20000, 160000), most_lights=rng.randint(1, 8))
    if kind == "served":
        return dict(kind="served", requests=_log(rng, 3, 12), spheres=_log(rng, 5, 40), least_points=4000,
                    most_points=_log(rng, 20000, 200000), most_lights=rng.randint(1, 6))
    w = _log(rng, 96, 640)
    n = _log(rng, 2000, 60000)
    return dict(kind="instanced", objects=n, lights=rng.randint(1, 4), width=w, height=max(8, w * 9 // 16),
                moved=n // 100 if kind == "moving" else 0)


# ---- scenes ---------------------------------------------------------------------


@lru_cache(maxsize=None)
def _shapes(subdivisions):
    """Unit displaced icospheres, the asset library the fields place."""
    return [scenes.displaced_icosphere((0.0, 0.0, 0.0), 1.0, seed=700 + 10 * subdivisions + k,
                                       subdivisions=subdivisions) for k in range(4)]


@lru_cache(maxsize=None)
def _boulders():
    return [scenes.displaced_uv_sphere(900 + k) for k in range(4)]


@lru_cache(maxsize=None)
def _kernel():
    k = MaskConeKernel.new(0)
    if k is None:
        raise RuntimeError("no CUDA device")
    return k


def _room(case, rng):
    """A ground quad with boxes resting on it under a 1 x 1 m light, and a
    grid of receivers on the ground."""
    half = 8.0 * math.sqrt(case["boxes"] / 64.0)
    meshes = [scenes.ground_quad(max(20.0, 2.0 * half))]
    for _ in range(case["boxes"]):
        e = rng.uniform(0.2, 1.0, 3)
        cx, cz = rng.uniform(-half, half, 2)
        meshes.append(scenes.box_mesh([cx - e[0] / 2, 0.0, cz - e[2] / 2], [cx + e[0] / 2, e[1], cz + e[2] / 2]))
    n = case["grid"]
    at = rng.uniform(-0.5, 0.5, 2)
    light = RectLight((float(at[0]) - 0.5, 4.0, float(at[1]) - 0.5), (1.0, 0.0, 0.0), (0.0, 0.0, 1.0), True)
    lin = -10.0 + 20.0 * (np.arange(n) + 0.5) / n
    zz, xx = np.meshgrid(lin, lin, indexing="ij")
    rec = np.zeros((n * n, 8), np.float32)
    rec[:, 0], rec[:, 2], rec[:, 5] = xx.reshape(-1), zz.reshape(-1), 1.0
    return meshes, light, rec


def _light(rng, half):
    """A rect or disk light of size U[0.25, 4] m, 8-20 m up, tilted up to 30
    degrees from straight down (a disk: a sphere light with a 90-degree spot)."""
    tilt, az = math.radians(30.0) * rng.random(), 2.0 * math.pi * rng.random()
    n = np.array([math.sin(tilt) * math.cos(az), -math.cos(tilt), math.sin(tilt) * math.sin(az)])
    u = np.cross([1.0, 0.0, 0.0], n)
    u /= np.linalg.norm(u)
    v = np.cross(n, u)
    x, z = rng.uniform(-0.8 * half, 0.8 * half, 2)
    centre = np.array([x, rng.uniform(8.0, 20.0), z])
    if rng.random() < 0.5:
        eu, ev = u * rng.uniform(0.25, 4.0), v * rng.uniform(0.25, 4.0)
        return light_gpu(Light.rect(RectLight(tuple(centre - 0.5 * (eu + ev)), tuple(eu), tuple(ev), True)))
    out = np.zeros(16, np.float32)
    scale = 1.0 / max(math.cos(math.radians(89.0)) - math.cos(math.radians(90.0)), 1e-3)
    out[0:3], out[3] = centre, 2.0
    out[4:7] = (0.5 * rng.uniform(0.25, 4.0), scale, -math.cos(math.radians(90.0)) * scale)
    out[8:11], out[11] = n, 1.0
    out[12:15] = 1.0
    return out


def _field(rng, spheres):
    """Displaced icospheres on a ground quad at one density; tri9, counts and
    the half extent."""
    half = max(10.0, 50.0 * math.sqrt(spheres / 150.0))
    parts = [scenes.ground_quad(max(1000.0, 20.0 * half)).reshape(-1, 9)]
    for _ in range(spheres):
        r = rng.uniform(0.5, 3.0)
        cx, cz = rng.uniform(-half, half, 2)
        shape = _shapes(5)[rng.integers(4)]
        parts.append((shape * np.float32(r) + np.array([cx, r, cz], np.float32)).reshape(-1, 9))
    return np.concatenate(parts), np.array([len(p) for p in parts], np.uint32), half


def _camera(rng, half):
    az = 2.0 * math.pi * rng.random()
    d = 1.5 * half
    return np.array([d * math.sin(az), 1.4 * half, -d * math.cos(az), 0, 0, 0, 0, 1, 0, 60.0], np.float32)


def _hits(scene, camera, width, height):
    """The camera's primary hits; the few pixels that miss take the last hit
    before them, so that every seed has as many receivers."""
    rec, hit = scene.primary_hits(camera, width, height)
    at = np.maximum.accumulate(np.where(hit.astype(bool), np.arange(len(hit)), np.argmax(hit)))
    return np.ascontiguousarray(rec[at])


def _image(points):
    w = max(8, int(round(math.sqrt(points * 16.0 / 9.0))))
    return w, max(8, int(round(points / w)))


class State:
    pass


def _outputs(cones, partial=False):
    o = {"full": torch.zeros(cones, dtype=torch.int64, device="cuda"),
         "any": torch.zeros(cones, dtype=torch.int64, device="cuda"),
         "irradiance": torch.zeros(cones, device="cuda"), "fraction": torch.zeros(cones, device="cuda")}
    if partial:
        o["partial"] = torch.zeros(cones, 64, device="cuda")
    return o


def _ptrs(outs):
    return {k: v.data_ptr() for k, v in outs.items()}


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    rng = np.random.default_rng([seed, 17])
    k = _kernel()
    s = State()
    s.kernel, s.case, s.kind = k, case, case["kind"]
    if s.kind == "room":
        s.meshes, s.rect, s.rec = _room(case, rng)
        s.lights = light_gpu(Light.rect(s.rect))[None, :]
        if case["entry"] == "irradiance":
            s.rec6 = np.ascontiguousarray(s.rec[:, [0, 1, 2, 4, 5, 6]])
            return s
        s.scene = k.scene(s.meshes)
    elif s.kind == "field":
        tri9, counts, half = _field(rng, case["spheres"])
        s.scene = k.scene_from_tri9(tri9, counts)
        s.lights = np.stack([_light(rng, half) for _ in range(case["lights"])])
        s.rec = _hits(s.scene, _camera(rng, half), case["width"], case["height"])
    elif s.kind == "batch":
        return _prepare_batch(s, rng)
    elif s.kind == "served":
        return _prepare_served(s, rng)
    else:
        return _prepare_instanced(s, rng)
    if case["entry"] == "host":
        return s
    s.d_rec, s.d_lig = _device(s.rec), _device(s.lights)
    if case["entry"] == "sky":
        s.sky = torch.zeros(len(s.rec), device="cuda")
    else:
        s.outs = _outputs(len(s.rec) * len(s.lights), case.get("partial", False))
    return s


def _prepare_batch(s, rng):
    case = s.case
    s.batch, s.keep, jobs = Batch(s.kernel), [], []
    lo, hi = math.log(case["least_points"]), math.log(case["most_points"])
    for j in range(case["jobs"]):
        # Sizes spread evenly over their logarithms in a fixed order, so that
        # every seed's batch is as much work.
        t = ((j * 7) % case["jobs"] + 0.5) / case["jobs"]
        u = ((j * 11) % case["jobs"] + 0.5) / case["jobs"]
        spheres = max(1, int(round(case["most_spheres"] ** u)))
        tri9, counts, half = _field(rng, spheres)
        scene = s.kernel.scene_from_tri9(tri9, counts)
        lights = np.stack([_light(rng, half) for _ in range(1 + (j * 5) % case["most_lights"])])
        rec = _hits(scene, _camera(rng, half), *_image(math.exp(lo + (hi - lo) * t)))
        jobs.append((scene, _device(rec), len(rec), _device(lights), len(lights)))
    # One set of output arrays, each job's cones at its place in them.
    s.outs, at = _outputs(sum(p * l for _, _, p, _, l in jobs)), 0
    for scene, d_rec, p, d_lig, l in jobs:
        s.batch.add(scene, d_rec.data_ptr(), p, d_lig.data_ptr(), l,
                    {m: v[at:at + p * l].data_ptr() for m, v in s.outs.items()})
        s.keep.append((scene, d_rec, d_lig))
        at += p * l
    return s


def _prepare_served(s, rng):
    case = s.case
    s.server = Server(s.kernel, hbm_budget=3 << 30)
    s.requests = []
    s.scenes = []
    for spheres in (max(1, case["spheres"] // 4), case["spheres"]):
        tri9, counts, half = _field(rng, spheres)
        scene = s.kernel.scene_from_tri9(tri9, counts)
        s.scenes.append((scene, half, s.server.add_scene(scene)))
    lo, hi = math.log(case["least_points"]), math.log(case["most_points"])
    for j in range(case["requests"]):
        scene, half, i = s.scenes[j % 2]
        t = ((j * 5) % case["requests"] + 0.5) / case["requests"]
        rec = _hits(scene, _camera(rng, half), *_image(math.exp(lo + (hi - lo) * t)))
        lights = np.stack([_light(rng, half) for _ in range(1 + (j * 7) % case["most_lights"])])
        shape = (len(lights), len(rec))
        pin = lambda dt: torch.zeros(shape, dtype=dt).pin_memory().numpy()  # noqa: E731
        outs = {"full": pin(torch.int64).view(np.uint64), "any": pin(torch.int64).view(np.uint64),
                "irradiance": pin(torch.float32), "fraction": pin(torch.float32)}
        s.requests.append((i, torch.from_numpy(rec).pin_memory().numpy(), lights, outs))
    return s


def _prepare_instanced(s, rng):
    case = s.case
    n = case["objects"]
    half = 2000.0 * math.sqrt(n / 1e6)
    geometries = list(_boulders()) + [scenes.ground_quad(1.0)]
    inst = np.zeros(n + 1, _lib.INSTANCE_DTYPE)

    def place(out, count):
        yaw = rng.uniform(0.0, 2.0 * math.pi, count)
        c, sn = np.cos(yaw).astype(np.float32), np.sin(yaw).astype(np.float32)
        rot = np.zeros((count, 9), np.float32)
        rot[:, 0], rot[:, 2], rot[:, 4], rot[:, 6], rot[:, 8] = c, sn, 1.0, -sn, c
        out["rotation"] = rot
        xz = rng.uniform(-half, half, (count, 2)).astype(np.float32)
        out["translation"] = np.stack([xz[:, 0], out["scale"], xz[:, 1]], 1)

    inst["geometry"][:n] = rng.integers(0, len(geometries) - 1, n)
    inst["scale"][:n] = rng.uniform(0.5, 4.0, n)
    place(inst[:n], n)
    inst[n] = (len(geometries) - 1, np.eye(3, dtype=np.float32).reshape(9), max(half * 1.05, 400.0), (0.0, 0.0, 0.0))
    movers = np.sort(rng.choice(n, case["moved"], replace=False)).astype(np.uint32) if case["moved"] else None
    s.scene = s.kernel.scene_instanced(geometries, inst, movers)
    spread = 40.0
    az = 2.0 * math.pi * rng.random()
    # Steep enough that every pixel meets the ground.
    camera = np.array([60.0 * math.sin(az), 95.0, -60.0 * math.cos(az), 0, 0, 0, 0, 1, 0, 60.0], np.float32)
    s.lights = np.stack([_light(rng, spread) for _ in range(case["lights"])])
    s.rec = _hits(s.scene, camera, case["width"], case["height"])
    s.d_rec, s.d_lig = _device(s.rec), _device(s.lights)
    cones = len(s.rec) * len(s.lights)
    s.outs = _outputs(cones)
    if movers is not None:
        # The view's results before the move, then the movers' new places: in
        # view, so that a frame has work, and each frame sends them again.
        torch.cuda.synchronize()
        s.kernel.visibility_device(s.scene, s.d_rec.data_ptr(), len(s.rec), s.d_lig.data_ptr(), len(s.lights),
                                   _ptrs(s.outs))
        s.placements = inst[movers].copy()
        xz = rng.uniform(-60.0, 60.0, (len(movers), 2)).astype(np.float32)
        near = rng.random(len(movers)) < 0.05
        s.placements["translation"][near, 0] = xz[near, 0]
        s.placements["translation"][near, 2] = xz[near, 1]
        s.stale = torch.zeros(cones, dtype=torch.uint8, device="cuda")
        boxes = s.scene.move(s.placements)
        s.kernel.stale_cones(s.scene, s.d_rec.data_ptr(), len(s.rec), s.lights, boxes, s.stale.data_ptr())
        s.kernel.visibility_update(s.scene, s.d_rec.data_ptr(), len(s.rec), s.d_lig.data_ptr(), len(s.lights),
                                   s.stale.data_ptr(), _ptrs(s.outs))
    return s


# ---- one pass -------------------------------------------------------------------


def run(s):
    case, k = s.case, s.kernel
    if s.kind == "batch":
        s.batch.submit()
        return s.outs
    if s.kind == "served":
        tickets = [s.server.submit(i, rec, lights, outs) for i, rec, lights, outs in s.requests]
        for t in tickets:
            s.server.wait(t)
        return [{m: (v.view(np.int64) if v.dtype == np.uint64 else v) for m, v in outs.items()}
                for _, _, _, outs in s.requests]
    if s.kind == "instanced" and case["moved"]:
        boxes = s.scene.move(s.placements)
        k.stale_cones(s.scene, s.d_rec.data_ptr(), len(s.rec), s.lights, boxes, s.stale.data_ptr())
        k.visibility_update(s.scene, s.d_rec.data_ptr(), len(s.rec), s.d_lig.data_ptr(), len(s.lights),
                            s.stale.data_ptr(), _ptrs(s.outs))
        return s.outs
    entry = case.get("entry", "device")
    if entry == "host":
        v = k.visibility(s.scene, s.rec, s.lights)
        return {"full": v.full.view(np.int64), "any": v.any.view(np.int64), "irradiance": v.irradiance,
                "fraction": v.fraction}
    if entry == "irradiance":
        return {"irradiance": k.irradiance(s.rec6, s.rect, s.meshes)[0]}
    k.prefilter = case.get("prefilter", 0.0)
    if entry == "sky":
        k.sky_visibility_device(s.scene, s.d_rec.data_ptr(), len(s.rec), s.sky.data_ptr())
        out = {"irradiance": s.sky}
    else:
        call = k.visibility_static if entry == "static" else k.visibility_device
        call(s.scene, s.d_rec.data_ptr(), len(s.rec), s.d_lig.data_ptr(), len(s.lights), _ptrs(s.outs),
             flags=_lib.CC_BACK_FACING if entry == "back" else 0)
        out = s.outs
    k.prefilter = 0.0
    return out


# ---- work and tolerance -----------------------------------------------------------


def work(case):
    """Receivers, lights, triangles and results, each once (a camera case:
    every pixel taken as a hit; a moving frame: every cone)."""
    tri, per = 36, 24 + (256 if case.get("partial") else 0)
    if case["kind"] == "room":
        p, l, t = case["grid"] ** 2, 1, 2 + 12 * case["boxes"]
        if case["entry"] == "sky":
            return {"bytes": p * (32 + 4) + t * tri}
        return {"bytes": p * (32 + (4 if case["entry"] == "irradiance" else 24)) + t * tri}
    if case["kind"] == "field":
        p, t = case["width"] * case["height"], 20480 * case["spheres"]
        if case["entry"] == "sky":
            return {"bytes": p * (32 + 4) + t * tri}
        return {"bytes": p * (32 + case["lights"] * per) + t * tri}
    if case["kind"] == "batch":
        lo, hi = math.log(case["least_points"]), math.log(case["most_points"])
        b, n = 0, case["jobs"]
        for j in range(n):
            t, u = ((j * 7) % n + 0.5) / n, ((j * 11) % n + 0.5) / n
            b += math.exp(lo + (hi - lo) * t) * (32 + (1 + (j * 5) % case["most_lights"]) * per)
            b += max(1, round(case["most_spheres"] ** u)) * 20480 * tri
        return {"bytes": b}
    if case["kind"] == "served":
        lo, hi = math.log(case["least_points"]), math.log(case["most_points"])
        n = case["requests"]
        b = 1.25 * case["spheres"] * 20480 * tri
        for j in range(n):
            b += math.exp(lo + (hi - lo) * (((j * 5) % n + 0.5) / n)) * (32 + (1 + (j * 7) % case["most_lights"]) * per)
        return {"bytes": b}
    p = case["width"] * case["height"]
    return {"bytes": p * (32 + case["lights"] * per) + 4 * 10240 * tri + case["objects"] * 64}


def tolerance(case):
    """A bin's coverage is a sum over a mesh's triangles, and mask words say
    which bins pass a threshold on it. Measured with the oracle, sums in walk
    order against order-free sums: on the fields light and fraction move by rel
    5e-8 (max 1e-5; at scale rel 2e-5 and single cones by 0.015, where a bin's
    snap ends a walk) and 0.2-1 % of the words differ; in the rooms one word in
    16,000. The rooms' light and fraction in 32 against 64 bits: rel 6e-6, max
    1.4e-4 (near the light's horizon)."""
    if case["kind"] == "room":
        return {"rel": 2.5e-5, "max": 6e-4, "differ": 2.5e-4}
    return {"rel": 6e-5, "max": 0.06, "differ": 0.01}


# ---- 64 bits ----------------------------------------------------------------------

NEAR, GRID = 1e-4, 8


def _clip(poly, count, dist):
    """Convex polygons (n, m, 3) of `count` vertices clipped to dist >= 0, with
    dist (n, m) each vertex's signed distance."""
    n, m, _ = poly.shape
    dev = poly.device
    idx = torch.arange(m, device=dev)[None, :].expand(n, m)
    live = idx < count[:, None]
    nxt = torch.where(idx + 1 >= count[:, None], torch.zeros_like(idx), idx + 1)
    b = torch.gather(poly, 1, nxt[:, :, None].expand(n, m, 3))
    db = torch.gather(dist, 1, nxt)
    ins, cross = live & (dist >= 0), live & ((dist >= 0) != (db >= 0))
    den = torch.where(cross, dist - db, torch.ones_like(dist))
    pt = poly + (b - poly) * (dist / den)[:, :, None]
    both = torch.stack([ins, cross], 2).reshape(n, 2 * m)
    pts = torch.stack([poly, pt], 2).reshape(n, 2 * m, 3)
    rank = torch.cumsum(both.long(), 1) - 1
    out = torch.zeros(n, m + 2, 3, dtype=poly.dtype, device=dev)
    r, c = torch.nonzero(both, as_tuple=True)
    out[r, rank[r, c]] = pts[r, c]
    return out, both.sum(1)


def _areas(q, count):
    """Signed area of polygons (n, m, 2) in [0, 8]^2 within each of the 8 x 8
    bins (n, 64), bin row * 8 + col."""
    n, m, _ = q.shape
    total = torch.zeros(n, 64, dtype=q.dtype, device=q.device)
    cols = torch.arange(GRID, device=q.device, dtype=q.dtype)

    def ramp(t):  # the integral of clamp(., 0, 1) up to t
        return torch.where(t <= 0, torch.zeros_like(t), torch.where(t >= 1, t - 0.5, 0.5 * t * t))

    for i in range(m):
        j = torch.where(i + 1 >= count, torch.zeros_like(count), torch.full_like(count, min(i + 1, m - 1)))
        live = i < count
        a, b = q[:, i], q[torch.arange(n, device=q.device), j]
        dy = b[:, 1] - a[:, 1]
        ok = live & (dy.abs() > 0)
        slope = torch.where(ok, (b[:, 0] - a[:, 0]) / torch.where(ok, dy, torch.ones_like(dy)), torch.zeros_like(dy))
        lo, hi = torch.minimum(a[:, 1], b[:, 1]), torch.maximum(a[:, 1], b[:, 1])
        sign = torch.where(ok, torch.sign(dy), torch.zeros_like(dy))
        y0 = torch.maximum(lo[:, None], cols[None, :])
        y1 = torch.minimum(hi[:, None], cols[None, :] + 1)
        h = (y1 - y0).clamp(min=0) * sign[:, None]
        x0 = a[:, 0:1] + slope[:, None] * (y0 - a[:, 1:2])
        x1 = a[:, 0:1] + slope[:, None] * (y1 - a[:, 1:2])
        t0, t1 = x0[:, :, None] - cols, x1[:, :, None] - cols  # (n, rows, cols)
        d = t1 - t0
        flat = d.abs() < 1e-9
        mean = torch.where(flat, (0.5 * (t0 + t1)).clamp(0, 1), (ramp(t1) - ramp(t0)) / torch.where(flat, torch.ones_like(d), d))
        total += (h[:, :, None] * mean).reshape(n, 64)
    return total


def _coverage(apex, frame, window, far, tris, combine):
    """Per cone the coverage of its 64 bins by every mesh: `tris` a list of
    (k, 3, 3); frame (n, 3, 3) rows right, up, forward; window (n, 4) u0 v0 u1
    v1; far (n) the far plane's distance along forward from the apex."""
    n = apex.shape[0]
    cov = torch.zeros(n, 64, dtype=apex.dtype, device=apex.device)
    su, sv = GRID / (window[:, 2] - window[:, 0]), GRID / (window[:, 3] - window[:, 1])
    for mesh in tris:
        acc = torch.zeros_like(cov)
        for t in mesh:
            nrm = torch.linalg.cross(t[1] - t[0], t[2] - t[0])
            front = ((apex - t[0]) @ nrm) > 0
            local = torch.einsum("nij,nkj->nki", frame, t[None] - apex[:, None])  # (n, 3, 3)
            x, y, z = local[..., 0], local[..., 1], local[..., 2]
            u0, v0, u1, v1 = (window[:, k:k + 1] for k in range(4))
            off = (z < NEAR).all(1) | (z > far[:, None]).all(1) | (x < u0 * z).all(1) | (x > u1 * z).all(1)
            ids = torch.nonzero(front & ~(off | (y < v0 * z).all(1) | (y > v1 * z).all(1)))[:, 0]
            if not len(ids):
                continue
            p, cnt = local[ids], torch.full((len(ids),), 3, dtype=torch.long, device=apex.device)
            w = window[ids]
            p, cnt = _clip(p, cnt, p[..., 2] - NEAR)
            p, cnt = _clip(p, cnt, far[ids, None] - p[..., 2])
            for plane in (lambda p: p[..., 0] - w[:, 0:1] * p[..., 2], lambda p: w[:, 2:3] * p[..., 2] - p[..., 0],
                          lambda p: p[..., 1] - w[:, 1:2] * p[..., 2], lambda p: w[:, 3:4] * p[..., 2] - p[..., 1]):
                p, cnt = _clip(p, cnt, plane(p))
            z = torch.where(p[..., 2] > 0, p[..., 2], torch.ones_like(p[..., 2]))
            q = torch.stack([(p[..., 0] / z - w[:, 0:1]) * su[ids, None], (p[..., 1] / z - w[:, 1:2]) * sv[ids, None]], 2)
            cnt = torch.where(cnt < 3, torch.zeros_like(cnt), cnt)
            acc.index_add_(0, ids, _areas(q.clamp(0, GRID), cnt))
        c = acc.abs()
        c = torch.where(c >= 1 - 1e-5, torch.ones_like(c), torch.where(c > 1e-6, c, torch.zeros_like(c)))
        cov = torch.maximum(cov, c) if combine == "max" else 1 - (1 - cov) * (1 - c)
    return cov


def _lambert(normal, quad):
    """The Lambert integral of quads of directions (..., 4, 3) clipped to the
    horizon of `normal` (..., 3)."""
    shape = quad.shape[:-2]
    p = quad.reshape(-1, 4, 3)
    nm = normal.expand(*shape, 3).reshape(-1, 3)
    cnt = torch.full((len(p),), 4, dtype=torch.long, device=p.device)
    p, cnt = _clip(p, cnt, (p * nm[:, None]).sum(-1))
    total = torch.zeros(len(p), dtype=p.dtype, device=p.device)
    rows = torch.arange(len(p), device=p.device)
    for i in range(p.shape[1]):
        j = torch.where(i + 1 >= cnt, torch.zeros_like(cnt), torch.full_like(cnt, min(i + 1, p.shape[1] - 1)))
        a, b = p[:, i], p[rows, j]
        live = (i < cnt) & (cnt >= 3)
        a = a / a.norm(dim=1, keepdim=True).clamp(min=1e-30)
        b = b / b.norm(dim=1, keepdim=True).clamp(min=1e-30)
        g = torch.linalg.cross(a, b)
        l = g.norm(dim=1)
        e = torch.atan2(l, (a * b).sum(1)) * (nm * g).sum(1) / l.clamp(min=1e-30)
        total += torch.where(live & (l > 1e-15), e, torch.zeros_like(e))
    return (0.5 * total).abs().reshape(shape)


def _bins(frame, window):
    """Directions of each bin's four corners, (n, 64, 4, 3)."""
    k = torch.arange(64, device=frame.device, dtype=frame.dtype)
    col, row = k % GRID, torch.div(k, GRID, rounding_mode="floor")
    s = torch.stack([col, col + 1, col + 1, col], 1) / GRID
    t = torch.stack([row, row, row + 1, row + 1], 1) / GRID
    u = window[:, 0, None, None] + s * (window[:, 2] - window[:, 0])[:, None, None]
    v = window[:, 1, None, None] + t * (window[:, 3] - window[:, 1])[:, None, None]
    right, up, fwd = (frame[:, i, None, None, :] for i in range(3))
    return fwd + right * u[..., None] + up * v[..., None]


def exact(case, seed):
    """Rooms only (a rect light or the sky over boxes), every triangle against
    every cone in 64 bits; a field's triangles would take too long."""
    if case["kind"] != "room" or case["grid"] > 256 or case["boxes"] > 64:
        return None
    rng = np.random.default_rng([seed, 17])
    meshes, rect, rec = _room(case, rng)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    to = lambda a: torch.as_tensor(np.asarray(a, np.float32).astype(np.float64), device=dev)  # noqa: E731
    apex, normal = to(rec[:, 0:3]), to(rec[:, 4:7])
    tris = [to(m) for m in meshes]
    n = len(rec)
    if case["entry"] == "sky":
        total = torch.zeros(n, dtype=torch.float64, device=dev)
        for f in range(6):
            axis, sign = f // 2, -1.0 if f % 2 else 1.0
            fwd, right = np.zeros(3), np.zeros(3)
            fwd[axis], right[(axis + 1) % 3] = sign, 1.0
            frame = torch.as_tensor(np.stack([right, np.cross(fwd, right), fwd]), device=dev).expand(n, 3, 3)
            window = torch.tensor([-1.0, -1.0, 1.0, 1.0], dtype=torch.float64, device=dev).expand(n, 4)
            far = torch.full((n,), 1e7, dtype=torch.float64, device=dev)
            above = (torch.einsum("nki,ni->nk", _bins(frame, window)[:, [0, 7, 56, 63], [0, 1, 3, 2]], normal) > 0).any(1)
            cov = _coverage(apex, frame, window, far, tris, "independent")
            w = torch.cat([_lambert(normal[i:i + 8192, None], _bins(frame[i:i + 8192], window[i:i + 8192]))
                           for i in range(0, n, 8192)])
            total += torch.where(above, (w * (1 - cov)).sum(1), torch.zeros_like(total))
        return {"irradiance": total}
    corner, eu, ev = to(rect.corner), to(rect.edge_u), to(rect.edge_v)
    fwd = torch.linalg.cross(eu, ev)
    fwd = fwd / fwd.norm()
    lit = ((apex - corner) @ fwd) > 0  # one-sided: receivers in front
    sgn = torch.where((corner - apex) @ fwd < 0, -1.0, 1.0)[:, None].to(torch.float64)
    forward = fwd[None] * sgn
    right = (eu / eu.norm()).expand(n, 3)
    up = torch.linalg.cross(forward, right)
    frame = torch.stack([right, up, forward], 1)
    dist = ((corner - apex) * forward).sum(1)
    corners = torch.stack([corner, corner + eu, corner + eu + ev, corner + ev])
    rel = torch.einsum("nij,nkj->nki", frame, corners[None] - apex[:, None]) / dist[:, None, None]
    window = torch.cat([rel[..., :2].amin(1), rel[..., :2].amax(1)], 1)
    cov = _coverage(apex, frame, window, dist * (1 - 1e-5), tris, "max")
    w = torch.cat([_lambert(normal[i:i + 8192, None], _bins(frame[i:i + 8192], window[i:i + 8192]))
                   for i in range(0, n, 8192)])
    lit = lit & ((corner + 0.5 * (eu + ev) - apex) * normal).sum(1).gt(0)
    irr = torch.where(lit, (w * (1 - cov)).sum(1), torch.zeros(n, dtype=torch.float64, device=dev))
    if case["entry"] == "irradiance":
        return {"irradiance": irr}
    total = w.sum(1)
    frac = torch.where(total > 0, (irr / total.clamp(min=1e-30)).clamp(0, 1), torch.ones_like(irr))
    out = {"full": None, "any": None, "irradiance": irr, "fraction": frac}
    if case["entry"] == "host":
        out["irradiance"], out["fraction"] = irr[None, :], frac[None, :]
    return out
