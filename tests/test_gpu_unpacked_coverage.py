"""Coverage materials (whose rays draw random numbers) on trees that do not fit the packed BVH form, as a tile on both
sides of the sizes at which the tail kernel takes over, and
in engine waves beside opaque scenes of either form.  Against the plain kernel, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import pathtracer as pt
import test_gpu_packed_bvh as trees
from pathtracer import abi
from pathtracer.engine import Engine
from worlds import non_opaque_world

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def worlds():
    field = pt.World.procedural(seed=3, grid_x=24, grid_z=16, boxes=40, spheres=2, sphere_subdivision=2,
                                emissive_triangles=8, skybox_width=32, skybox_height=16)
    return {"coverage": (w := non_opaque_world(), w.take_updates()), "field": (field, field.take_updates())}


def accumulation(u, size, spp, bounces, kernel):
    t = pt.PathTracer(u, size)
    t.set_kernel(kernel)
    t.set_max_bounces(bounces)
    assert t.trace(spp) == spp
    out = t.read_tile(abi.PT_TILE_ACCUMULATION)
    t.close()
    return out


# up to 2^17 paths (finished from round 0), 2^18 (round 1), 2^21 (by hits), more (never)
@pytest.mark.parametrize("form", ["leaves of 15", "unreachable nodes"])
@pytest.mark.parametrize("size,spp", [((61, 37), 3), ((129, 128), 9), ((300, 217), 8), ((513, 256), 16)])
def test_tiles_equal_plain(worlds, form, size, spp):
    u, _keep = trees.updates_with(worlds, "coverage", form)
    plain = accumulation(u, size, spp, 7, abi.PT_KERNEL_PLAIN)
    assert plain[..., :3].max() > 0
    assert plain.tobytes() == accumulation(u, size, spp, 7, abi.PT_KERNEL_WAVEFRONT).tobytes()


@pytest.mark.parametrize("size,spp", [((48, 40), 3), ((300, 217), 8), ((520, 258), 16)])
def test_waves_beside_opaque_scenes_equal_plain(worlds, size, spp):
    eng = Engine(wave_paths=1 << 22)
    jobs, keep = [], []
    for name, form in (("coverage", "leaves of 15"), ("field", "as built"), ("field", "leaves of 15"), ("coverage", "as built")):
        u, k = trees.updates_with(worlds, name, form)
        keep.append(k)
        cam = abi.Camera.from_buffer_copy(u.camera.contents)
        jobs.append((u, eng.submit(eng.add_scene(u), cam, *size, spp, 6)))
    eng.wait_idle(timeout_ms=60000)
    for u, job in jobs:
        plain = accumulation(u, size, spp, 6, abi.PT_KERNEL_PLAIN)
        assert eng.read(job, *size, abi.PT_TILE_ACCUMULATION).tobytes() == plain.tobytes()
    eng.close()
