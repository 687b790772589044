"""The library's host code over a runtime that has no GPU (tests/fake): no
kernel may be launched while an input's copy from pageable host memory may
still be on its way, as such a copy can return early and the context's streams
do not wait for the legacy stream it runs in."""
import subprocess
import sys
from pathlib import Path

import pytest

from continuum_b200 import build as cbuild

TESTS = Path(__file__).resolve().parent
ROOT = TESTS.parent

PRELUDE = """
import ctypes, sys
from pathlib import Path
import numpy as np
from continuum_b200 import _lib
_lib.LIB_PATH = Path(sys.argv[1])
from continuum_b200 import Batch, MaskConeKernel, Server, scenes
fake = ctypes.CDLL(sys.argv[1])
fake.fake_unordered.restype = ctypes.c_char_p
fake.fake_live_bytes.restype = ctypes.c_ulong
fake.fake_launches.restype = ctypes.c_long
fake.fake_launches.argtypes = [ctypes.c_char_p]
w = scenes.box_field(grid=16)
rec, lights = np.ascontiguousarray(w.receivers), np.ascontiguousarray(w.lights)
P, L = len(rec), len(lights)
def outputs(n=P * L):  # kernels do nothing here: host arrays serve as device buffers
    return {k: np.zeros(2 * n, np.uint32) for k in ("full", "any", "irradiance", "fraction")}
def pointers(o):
    return {k: v.ctypes.data for k, v in o.items()}
kernel = MaskConeKernel(0)
"""


@pytest.fixture(scope="session")
def fake_library(tmp_path_factory):
    """The library's own objects linked with the runtime without a GPU."""
    objects = [cbuild.PKG / "_build" / (s + ".o") for s in cbuild.SOURCES]
    if not cbuild.up_to_date() or not all(o.exists() for o in objects):
        cbuild.build(force=True)
    include = Path(cbuild.nvcc()).resolve().parent.parent / "include"
    out = tmp_path_factory.mktemp("fake") / "libcontinuum_fake.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", str(include), "-o", str(out),
                    str(TESTS / "fake" / "cuda_runtime_fake.cpp"), *map(str, objects), "-Wl,-Bsymbolic",
                    "-Wl,--no-undefined", "-lpthread"], check=True)
    return out


def run(library, code: str) -> str:
    out = subprocess.run([sys.executable, "-c", PRELUDE + code, str(library)], cwd=ROOT, capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr[-3000:]
    return out.stdout


CALLS = {
    "scene": """
scene = kernel.scene(w.meshes)
kernel.visibility_device(scene, rec.ctypes.data, P, lights.ctypes.data, L, pointers(outputs()))
""",
    "large scene": """
scene = kernel.scene([scenes.displaced_icosphere((0, 0, 0), 1.0, seed=1, subdivisions=6)])
kernel.visibility_device(scene, rec.ctypes.data, P, lights.ctypes.data, L, pointers(outputs()))
""",
    "drop-in": """
from continuum_b200.kernel import RectLight
light = RectLight((-1.0, 6.0, -1.0), (2.0, 0.0, 0.0), (0.0, 0.0, 2.0), True)
r6 = np.ascontiguousarray(np.concatenate([rec[:, 0:3], rec[:, 4:7]], axis=1))
kernel.irradiance(r6, light, w.meshes)
kernel.irradiance(r6, light, w.meshes)
kernel.coverage(r6, light, w.meshes)
""",
    "sky": """
scene = kernel.scene(w.meshes)
kernel.sky_visibility_device(scene, rec.ctypes.data, P, outputs()["full"].ctypes.data)
""",
    "prefiltered": """
scene = kernel.scene(w.meshes)
kernel.prefilter = 1.0
kernel.visibility_device(scene, rec.ctypes.data, P, lights.ctypes.data, L, pointers(outputs()))
""",
    "back-facing": """
scene = kernel.scene(w.meshes)
kernel.visibility_device(scene, rec.ctypes.data, P, lights.ctypes.data, L, pointers(outputs()), flags=_lib.CC_BACK_FACING)
""",
    "moved and cleared": """
world = scenes.instanced_world(seed=3, n_instances=300, n_boulders=3, half=40.0, n_lights=2, width=32, height=18,
                               segments=24, rings=13)
scene = kernel.scene_instanced(world.geometries, world.instances, movable=[5, 9])
go = lambda: kernel.visibility_device(scene, rec.ctypes.data, P, lights.ctypes.data, L, pointers(outputs()))
go()
scene.move([world.instances[5], world.instances[9]])
go()
scene.set_clear(np.zeros(len(world.instances), np.float32))
go()
kernel.prefilter = 1.0
go()
scene.set_clear(np.full(len(world.instances), 0.25, np.float32))
go()
""",
    "batch": """
scene = kernel.scene(w.meshes)
b = Batch(kernel)
keep = [outputs() for _ in range(3)]
for k, o in enumerate(keep):
    b.add(scene, rec.ctypes.data, P, lights.ctypes.data, L, pointers(o), prefilter=float(k == 2))
b.submit(Batch.options(flags=0))
b.wait()
b.close()
""",
    "server": """
scene = kernel.scene(w.meshes)
srv = Server(kernel, hbm_budget=64 << 20)
sid = srv.add_scene(scene)
o = {"full": np.zeros((L, P), np.uint64), "any": np.zeros((L, P), np.uint64),
     "irradiance": np.zeros((L, P), np.float32), "fraction": np.zeros((L, P), np.float32)}
srv.wait(srv.submit(sid, rec, lights, o))
srv.close()
""",
}


@pytest.mark.parametrize("call", CALLS)
def test_no_kernel_runs_beside_a_copy_of_its_inputs(fake_library, call):
    out = run(fake_library, CALLS[call] + "\nprint('LAUNCHES', fake.fake_launches(b'_kernel'))"
                                          "\nprint('UNORDERED', fake.fake_unordered().decode())\n")
    assert int(out.split("LAUNCHES", 1)[1].split()[0]) > 0
    assert out.split("UNORDERED", 1)[1].strip() == ""


def test_a_device_gets_its_tables_once(fake_library):
    """The tables that every context's kernels read are not written again when
    another context is created, as those kernels may be running."""
    out = run(fake_library, """
made = fake.fake_launches(b"sky_table")
other = MaskConeKernel(0)
print(made, fake.fake_launches(b"sky_table"), fake.fake_unordered().decode())
""")
    made, after = map(int, out.split())
    assert made == after == 2  # one copy in each unit that walks sky cones


def test_a_large_drop_in_call_keeps_no_inputs(fake_library):
    """cc_irradiance borrows the context's buffers, and gives back what a large
    call made them grow by; and a closed context and batch keep nothing."""
    out = run(fake_library, """
from continuum_b200.kernel import RectLight
light = RectLight((-1.0, 6.0, -1.0), (2.0, 0.0, 0.0), (0.0, 0.0, 2.0), True)
n = 1 << 20
r6 = np.zeros((n, 6), np.float32)
r8 = np.zeros((n, 8), np.float32)
scene = kernel.scene(w.meshes)
o = {"irradiance": np.zeros(n, np.float32)}
kernel.visibility_device(scene, r8.ctypes.data, n, lights.ctypes.data, 1, pointers(o))  # the walk's own scratch
scene.close()
kernel.irradiance(r6[:64], light, w.meshes)
before = fake.fake_live_bytes()
kernel.irradiance(r6, light, w.meshes)
print(before, fake.fake_live_bytes())
""")
    before, after = map(int, out.split())
    assert after - before <= 2 * (4 << 20)  # two buffers of at most 4 MB


def test_closed_contexts_and_batches_keep_nothing(fake_library):
    out = run(fake_library, """
empty = fake.fake_live_bytes()
k = MaskConeKernel(0)
scene = k.scene(w.meshes)
k.visibility(scene, rec, lights, outputs=("full", "any", "partial", "irradiance", "fraction", "work"))
k.sky_visibility(scene, rec, outputs=("full", "fraction"))
b = Batch(k)
keep = [outputs() for _ in range(3)]
stale = np.ones(P * L, np.uint8)
b.add(scene, rec.ctypes.data, P, lights.ctypes.data, L, pointers(keep[0]))
b.add(scene, rec.ctypes.data, P, lights.ctypes.data, L, pointers(keep[1]), prefilter=1.0)
b.add_update(scene, rec.ctypes.data, P, lights.ctypes.data, L, stale.ctypes.data, pointers(keep[2]))
b.submit(Batch.options(flags=0))
b.wait()
b.close()
scene.close()
k.close()
print(empty, fake.fake_live_bytes())
""")
    empty, after = map(int, out.split())
    assert after == empty
